"""A field that spreads into an exactly zero background: its front decays by a factor per cell, so B_x and
psi pass through the subnormal numbers on a long grid (from step 134 on here).  The FP64 form has to follow
the oracle.  Every field is of order one or less and a step is allowed 1e-12: 2e-10 after 200."""
import os
import sys

import numpy as np
import pytest

from mhdturbulence_gb300 import Solver, ic

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu
NX, NY, NZ, GAM, STEPS = 512, 4, 4, 5.0 / 3.0, 200
BC = (1,) * 6


@pytest.mark.parametrize("riemann", ["hlld", "hllc"])
def test_front_into_a_zero_field(riemann):
    p = {k: np.zeros((NZ, NY, NX)) for k in ("rho", "vx", "vy", "vz", "p", "bx", "by", "bz", "psi", "X")}
    p["rho"][...] = p["p"][...] = 1.0
    p["bx"][..., 240:272] = 0.1
    U0 = ic.prim_to_cons(p, GAM)
    orc = O.Oracle(NX, NY, NZ, *ic.grid(NX, NY, NZ, ic.CUBE_DOMAIN), gam=GAM, bc=BC, spacing_quirk=False,
                   riemann={"hlld": 0, "hllc": 2}[riemann])
    Uo, Po = U0.copy(), ic.empty_field(NX, NY, NZ, 12)
    orc.update_prim(Uo, Po)
    orc.run(Uo, Po, STEPS)
    tiny = np.abs(ic.interior(Uo)[:, :, 5:9:3])
    assert ((tiny > 0.0) & (tiny < 2.0 ** -1022)).any()  # the front has got there
    with Solver(NX, NY, NZ, domain=ic.CUBE_DOMAIN, bc=BC, gam=GAM, precision="fp64", riemann=riemann) as s:
        s.upload_cons(U0)
        s.step(STEPS)
        s.sync()
        U = s.download_cons()
    assert np.abs(ic.interior(U) - ic.interior(Uo)).max() <= 2e-10
