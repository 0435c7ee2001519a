"""Whichever kernel a grid of the FP64 forms starts on, the state is the same bit for bit; the run-time solver's
kernel, which an HLLD member of a mixed ensemble runs on, gives it bit for bit in the separately rounded form and
within 1e-12 of each field's largest magnitude in the other, whose compiler contracts its products separately.
The states keep all parts of the face flux busy: strong jumps, walls with a normal velocity, faces on both sides of
the pairs' range and outside it."""
import numpy as np
import pytest

from mhdturbulence_gb300 import Ensemble, Solver, ic

pytestmark = pytest.mark.gpu
N, GAM = (37, 21, 19), 5.0 / 3.0


def _state(kind):
    p = ic.random_smooth_prim(*N, seed=8)
    r = np.random.default_rng(9)
    shape = p["rho"].shape
    if kind == "jumps":
        p["rho"] = p["rho"] * r.uniform(0.5, 2.0, shape)
        p["p"] = p["p"] * r.uniform(0.5, 2.0, shape)
        for k in ("vx", "vy", "vz", "bx", "by", "bz"):
            p[k] = p[k] + r.uniform(-0.3, 0.3, shape)
    elif kind == "range":  # densities on both sides of 2^-20
        for k, f in (("rho", 2.0 ** -20), ("p", 2.0 ** -20), ("bx", 2.0 ** -10), ("by", 2.0 ** -10), ("bz", 2.0 ** -10)):
            p[k] = f * p[k]
    elif kind == "cgs":
        for k, f in (("rho", 1e-24), ("p", 1e-12), ("vx", 1e6), ("vy", 1e6), ("vz", 1e6), ("bx", 1e-6), ("by", 1e-6), ("bz", 1e-6),
                     ("psi", 1.0)):
            p[k] = f * p[k]
    return ic.prim_to_cons(p, GAM)


@pytest.mark.parametrize("precision", ["fp64", "fp64_exact"])
@pytest.mark.parametrize("kind", ["smooth", "jumps", "range", "cgs"])
def test_all_kernels_agree(kind, precision):
    U0 = _state(kind)
    kw = {"domain": ic.CUBE_DOMAIN, "bc": (1, 1, 2, 2, 3, 2)}
    outs = {}

    def run(step, s):
        s.upload_cons(U0)
        step(3)
        return s.download_cons()

    with Solver(*N, precision=precision, gam=GAM, **kw) as s:
        for v in range(len(s.variants())):
            s.select_variant(v)
            s.reset_clock()
            outs[s.variant_name()] = run(s.step, s)
    spec = {"nx": N[0], "ny": N[1], "nz": N[2], **kw}
    with Ensemble([spec, {**spec, "riemann": "hlle"}], precision=precision, gam=GAM) as e:
        e.members[1].upload_cons(U0)
        gen = run(e.step, e.members[0])
    first = next(iter(outs.values()))
    assert np.isfinite(first).all()
    assert {k: np.array_equal(v, first) for k, v in outs.items()} == dict.fromkeys(outs, True)
    if precision == "fp64_exact":
        assert np.array_equal(gen, first)
    a, b = ic.interior(gen), ic.interior(first)
    for m in range(10):
        assert np.abs(a[:, :, m] - b[:, :, m]).max() <= 1e-12 * np.abs(b[:, :, m]).max(), m
