"""The FP64 form's face flux in FP32 pairs, built for the CPU from its own header, where its arithmetic can
go wrong: subnormal operands, and sums that cancel."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from mhdturbulence_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))
DP = C.POINTER(C.c_double)
NPRIM, NCONS = 12, 10
DEN, VX, VY, VZ, ENE, PRE, CS, BX, BY, BZ, PSI, X = range(NPRIM)
GAM, CH = 5.0 / 3.0, 3.0


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = tmp_path_factory.mktemp("face") / "face_split_host.so"
    subprocess.run([build.nvcc(), "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC,-ffp-contract=off", "-I" + build.CSRC,
                    "-x", "c++", os.path.join(HERE, "face_split_host.cpp"), "-o", str(so)], check=True)
    return C.CDLL(str(so))


def _ptr(a):
    return a.ctypes.data_as(DP)


def faces(host, left, right, riemann="hlld"):
    """Fluxes (n, 10) and which faces the split takes, of states (n, 12)."""
    left, right = (np.ascontiguousarray(a, dtype=np.float64) for a in (left, right))
    F, ok = np.empty((len(left), NCONS)), np.empty(len(left), dtype=np.int32)
    host.faces(len(left), _ptr(left), _ptr(right), C.c_double(CH), int(riemann == "hllc"), _ptr(F),
               ok.ctypes.data_as(C.POINTER(C.c_int)))
    return F, ok != 0


def states(n, **f):
    """n states from their fields: density 1, pressure 1 and the rest 0 unless given."""
    P = np.zeros((n, NPRIM))
    P[:, DEN] = P[:, PRE] = 1.0
    for k, v in f.items():
        P[:, {"rho": DEN, "vx": VX, "vy": VY, "vz": VZ, "p": PRE, "bx": BX, "by": BY, "bz": BZ, "psi": PSI, "X": X}[k]] = v
    P[:, ENE] = P[:, PRE] / ((GAM - 1.0) * P[:, DEN])
    P[:, CS] = np.sqrt(GAM * P[:, PRE] / P[:, DEN])
    return P


def test_halving_is_exact_at_every_exponent(host):
    rng = np.random.default_rng(1)
    bits = rng.integers(0, 1 << 52, 1 << 16, dtype=np.uint64) | rng.integers(0, 4096, 1 << 16, dtype=np.uint64) << np.uint64(52)
    edge = np.array([m | e << 52 for e in (0, 1, 2, 3, 2045, 2046) for m in (0, 1, 2, 3, 4, 5, 2 ** 32 - 1, 2 ** 32, 2 ** 32 + 1,
                                                                              2 ** 52 - 1, 2 ** 52 - 2, 2 ** 52 - 3)] +
                    [2047 << 52, 2047 << 52 | 1 << 51], dtype=np.uint64)
    x = np.concatenate([bits, edge, edge | np.uint64(1 << 63)]).view(np.float64)
    y = np.empty_like(x)
    host.halve(len(x), _ptr(x), _ptr(y))
    with np.errstate(all="ignore"):
        ref = 0.5 * x
    nan = np.isnan(ref)
    assert np.array_equal(y[~nan].view(np.uint64), ref[~nan].view(np.uint64)) and np.isnan(y[nan]).all()


@pytest.mark.parametrize("riemann", ["hlld", "hllc"])
@pytest.mark.parametrize("field", ["bx", "psi"])
def test_subnormal_normal_field_and_psi(host, field, riemann):
    """One side or both hold a value at or below the smallest normal number: the GLM pair is what FP64
    products give (0.5 (a + b) - (c_h / 2) (b - a) and its counterpart, each within an ulp)."""
    tiny = [0.0] + [s * v for v in (1e-300, 4.5e-308, 2.3e-308, 2e-308, 1e-308, 1e-310, 1e-320, 5e-324) for s in (1.0, -1.0)]
    a, b = (v.ravel() for v in np.meshgrid(tiny, tiny))
    F, ok = faces(host, states(len(a), **{field: a}), states(len(b), **{field: b}), riemann)
    assert ok.all() and np.isfinite(F).all()
    lo, hi = 0.5 * (a + b), b - a
    if field == "bx":
        want = {5: -0.5 * CH * hi, 8: lo * (CH * CH)}
    else:
        want = {5: lo, 8: -0.5 * CH * hi}
    for m, w in want.items():
        assert (np.abs(F[:, m] - w) <= 2.0 * np.spacing(np.abs(w))).all()
