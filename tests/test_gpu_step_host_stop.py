"""mhdgb_step_host and the stop condition: steps after it are skipped, and U_out is the state at the stop
whichever way the arrays travel."""
import numpy as np
import pytest

from mhdturbulence_gb300 import Solver

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

N = (37, 13, 11)


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.numpy()[...] = a
    return t


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp64_exact"])
@pytest.mark.parametrize("nsteps,stop", [(1, 0), (3, 0), (3, 1), (3, 2), (3, 3), (1, 1), (19, 5)])
def test_output_is_the_state_at_the_stop(nsteps, stop, precision):
    outs = []
    for kind in ("staged", "separate", "inplace"):
        with Solver(*N, precision=precision) as s:
            s.init_kh(seed=6)
            U0 = s.download_cons()
            s.step(2)  # the clock stands at 2
            s.sync()
            s.set_stop(max_steps=2 + stop)
            src = U0.copy() if kind == "staged" else _pinned(U0).numpy()
            dst = src if kind == "inplace" else np.full_like(U0, np.nan) if kind == "staged" else _pinned(np.full_like(U0, np.nan)).numpy()
            s.step_host(src, dst, nsteps)
            r = s.sync()
            assert r.done == 1 and r.step == 2 + stop
            assert np.array_equal(dst, s.download_cons())
            outs.append(dst.copy())
    assert np.isfinite(outs[0]).all()
    if stop == 0:
        assert np.array_equal(outs[0], U0)
    assert np.array_equal(outs[1], outs[0]) and np.array_equal(outs[2], outs[0])
