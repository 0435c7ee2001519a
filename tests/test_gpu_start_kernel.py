"""The kernel a small grid starts on: another table entry than the large grids' where its queue is simulated
to finish earlier, with the same state bit for bit."""
import numpy as np
import pytest

from mhdturbulence_gb300 import Solver, ic

pytestmark = pytest.mark.gpu

PREFERRED = {"fp64": "two-phase 16x8/256", "mixed": "fused-slope 16x8/256 x2", "fp64_exact": "two-phase 32x4/128"}


@pytest.mark.parametrize("precision", ["fp64", "fp64_exact"])
@pytest.mark.parametrize("shape", [(3, 3, 3), (8, 8, 8), (9, 7, 5), (16, 16, 16), (24, 40, 20), (17, 33, 9), (130, 12, 30),
                                   (65, 8, 31)])
def test_a_small_grid_starts_on_a_kernel_with_the_same_results(precision, shape):
    U0 = ic.prim_to_cons(ic.kh_prim(*shape, seed=4), 5.0 / 3.0)
    outs = []
    for name in (None, PREFERRED[precision]):
        with Solver(*shape, precision=precision) as s:
            if name:
                s.select_variant([s.variant_name(v) for v in range(len(s.variants()))].index(name))
            s.upload_cons(U0)
            s.step(3)
            r = s.sync()
            outs.append((r.dt, s.download_cons()))
    assert outs[0][0] == outs[1][0] and np.array_equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("precision,shape,name", [
    ("fp64", (24, 40, 20), "two-phase 8x8/256"),        # two planes of a 16x8 tile per SM, or two of an 8x8 one
    ("fp64", (64, 64, 64), "two-phase 16x8/256"),
    ("fp64_exact", (100, 62, 90), "two-phase 16x8/256"),
    ("fp64_exact", (24, 40, 20), "two-phase 8x8/256"),
    ("fp64_exact", (225, 150, 100), "two-phase 32x4/128"),  # 150^3 cells: the preferred entry
    ("mixed", (24, 40, 20), "fused-slope 16x8/256 x2"),
])
def test_the_starting_kernel_by_size(precision, shape, name):
    with Solver(*shape, precision=precision) as s:
        assert s.variant_name() == name
        s.set_riemann("hlle")
        assert s.variant_name().endswith("run-time solver")
        s.set_riemann("hlld")
        assert s.variant_name() == name
