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


def reference(left, right, riemann="hlld"):
    """The flux (n, 10) of mhd.cpp:97-417 (with its energy flux term B^2 B_n, mhd.cpp:1049) in extended precision, and for each component the magnitudes of the terms it is the
    sum of: the upwind side's physical flux, and wave speed times jump for each wave inside the fan, a speed or
    a jump that is itself a difference of larger terms (jumps of velocity and pressure; S_M and |B_n| / sqrt(rho*))
    counted by those."""
    L, R = (np.asarray(a, dtype=np.longdouble).T for a in (left, right))

    def side(P):
        rho, vx, vy, vz, e, p, cs, bx, by, bz, psi, x = P
        b2 = bx * bx + by * by + bz * bz
        E = rho * e + rho * (vx * vx + vy * vy + vz * vz) / 2 + b2 / 2
        pt = p + b2 / 2
        U = [rho, rho * vx, rho * vy, rho * vz, E, by, bz, rho * x]
        F = [[rho * vx], [rho * vx * vx, pt, -bx * bx], [rho * vy * vx, -by * bx], [rho * vz * vx, -bz * bx],
             [E * vx, pt * vx, -b2 * bx], [by * vx, -vy * bx], [bz * vx, -vz * bx], [rho * x * vx]]
        a = cs * cs + b2 / rho
        cf = np.sqrt((a + np.sqrt((cs * cs - bx * bx / rho) ** 2 + (by * by + bz * bz) / rho *
                                  (2 * cs * cs + 2 * bx * bx / rho + (by * by + bz * bz) / rho))) / 2)
        return U, F, cf, pt

    (Ul, Fl, cl, pl), (Ur, Fr, cr, pr) = side(L), side(R)
    c = np.maximum(cl, cr)
    vl, vr = L[VX], R[VX]
    sl, sr = np.minimum(vl, vr) - c, np.maximum(vl, vr) + c
    al, ar = L[DEN] * (sl - vl), R[DEN] * (sr - vr)
    dpt = R[PRE] - L[PRE] + sum((R[q] - L[q]) * (R[q] + L[q]) for q in (BX, BY, BZ)) / 2  # (pr - pl would round)
    sm = (ar * vr - al * vl - dpt) / (ar - al)
    ps = (ar * pl - al * pr + al * ar * (vr - vl)) / (ar - al)
    bx = (L[BX] + R[BX]) / 2

    def star(P, U, s, a, pt):
        rho = a / (s - sm)
        if riemann == "hllc":
            k = rho / P[DEN]
            return [rho, rho * sm, rho * P[VY], rho * P[VZ], ((s - P[VX]) * U[4] - pt * P[VX] + ps * sm) / (s - sm), k * U[5],
                    k * U[6], k * U[7]], None
        T = a * (s - sm) - bx * bx
        t1, t2 = bx * (sm - P[VX]) / T, (a * (s - P[VX]) - bx * bx) / T
        vy, vz, by, bz = P[VY] - P[BY] * t1, P[VZ] - P[BZ] * t1, P[BY] * t2, P[BZ] * t2
        vb = sm * bx + vy * by + vz * bz
        E = ((s - P[VX]) * U[4] - pt * P[VX] + ps * sm + bx * (P[VX] * bx + P[VY] * P[BY] + P[VZ] * P[BZ] - vb)) / (s - sm)
        return [rho, rho * sm, rho * vy, rho * vz, E, by, bz, rho * P[X]], (vy, vz, vb)

    (Sl, tl), (Sr, tr) = star(L, Ul, sl, al, pl), star(R, Ur, sr, ar, pr)
    up = ~(sm < 0)
    terms = [[np.where(up, p, q) for p, q in zip(f, g)] for f, g in zip(Fl, Fr)]
    size = [[abs(x) for x in t] for t in terms]
    # S_M relative to a side: (rho_o (v_r - v_l) -+ (pt_r - pt_l) / w) / (rho_l + rho_r)
    w = c - np.minimum(vr - vl, 0)
    # (the mean of B_n is one FP64 sum; those of B_t are sums of pairs)
    psize = abs(R[PRE] - L[PRE]) + (abs((R[BX] - L[BX]) * (R[BX] + L[BX])) +
                                    sum(abs(R[q] - L[q]) * (abs(R[q]) + abs(L[q])) for q in (BY, BZ))) / 2
    d = abs(sm - np.where(up, vl, vr))
    dsize = (np.where(up, R[DEN], L[DEN]) * abs(vr - vl) + psize / w) / (L[DEN] + R[DEN])
    grow = np.where(d > 0, dsize / np.where(d > 0, d, 1), 1)
    s = np.where(up, np.minimum(sl, 0), np.maximum(sr, 0))
    jump = [np.where(up, a - b, e - f) for a, b, e, f in zip(Sl, Ul, Sr, Ur)]
    jump[0] = np.where(up, L[DEN] * (sm - vl) / (sl - sm), R[DEN] * (sm - vr) / (sr - sm))  # (rho* - rho would round)
    jump[7] = jump[0] * np.where(up, L[X], R[X])
    for m in range(8):
        terms[m].append(s * jump[m])
        size[m].append(abs(terms[m][-1]) * grow)
    if riemann == "hlld":
        ql, qr, h = np.sqrt(Sl[0]), np.sqrt(Sr[0]), np.where(bx < 0, -1, 1)
        vy, vz = ((ql * a + qr * b + h * (q - p)) / (ql + qr) for a, b, p, q in
                  ((tl[0], tr[0], Sl[5], Sr[5]), (tl[1], tr[1], Sl[6], Sr[6])))
        by, bz = ((ql * q + qr * p + h * ql * qr * (b - a)) / (ql + qr) for a, b, p, q in
                  ((tl[0], tr[0], Sl[5], Sr[5]), (tl[1], tr[1], Sl[6], Sr[6])))
        vb = sm * bx + vy * by + vz * bz
        q, i = np.where(up, ql, qr), np.where(up, 1, -1)
        S = [np.where(up, a, b) for a, b in zip(Sl, Sr)]
        s2 = np.where(up, np.minimum(sm - abs(bx) / ql, 0), np.maximum(sm + abs(bx) / qr, 0)) * (bx != 0)
        dd = {2: S[0] * vy - S[2], 3: S[0] * vz - S[3], 4: -i * h * q * (np.where(up, tl[2], tr[2]) - vb), 5: by - S[5],
              6: bz - S[6]}
        qo = np.where(up, qr, ql)
        D = [(qo * (abs(tl[a] - L[v]) + abs(tr[a] - R[v]) + abs(R[v] - L[v])) +
              abs(Sl[b] - L[f]) + abs(Sr[b] - R[f]) + abs(R[f] - L[f])) / (ql + qr)
             for a, v, b, f in ((0, VY, 5, BY), (1, VZ, 6, BZ))]
        s2size = (s2 != 0) * (abs(sm) + abs(bx) / q)
        dsizes = {2: S[0] * D[0], 3: S[0] * D[1], 5: q * D[0], 6: q * D[1],
                  4: q * (D[0] * (abs(S[5]) + q * abs(vy)) + D[1] * (abs(S[6]) + q * abs(vz)))}
        for m, e in dd.items():
            terms[m].append(s2 * e)
            size[m].append(s2size * dsizes[m])
    glm = [[(L[PSI] + R[PSI]) / 2, -CH * (R[BX] - L[BX]) / 2], [CH * CH * bx, -CH * (R[PSI] - L[PSI]) / 2]]
    glms = [[(abs(L[PSI]) + abs(R[PSI])) / 2, abs(glm[0][1])], [CH * CH * (abs(L[BX]) + abs(R[BX])) / 2, abs(glm[1][1])]]
    terms, size = (x[:5] + [g[0]] + x[5:7] + [g[1], x[7]] for x, g in ((terms, glm), (size, glms)))
    return np.stack([sum(t) for t in terms], axis=1), np.stack([sum(t) for t in size], axis=1)


# A pair carries 48 bits, and the chains behind a correction lose a few of them: 2^-43 of the flux's terms is
# the accuracy that the form states for itself.
def assert_accurate(host, left, right, riemann, taken):
    F, ok = faces(host, left, right, riemann)
    assert ok.mean() >= taken
    ref, scale = reference(left, right, riemann)
    err = np.abs(F - ref) / np.where(scale > 0, scale, 1)
    assert err[ok].max() <= 2.0 ** -43, (err[ok].max(axis=0), 2.0 ** -43)


def _random(rng, n, **width):
    """Background fields of order one, and a jump of the given width in each."""
    mid = dict(rho=rng.uniform(0.5, 1.5, n), vx=rng.uniform(-0.8, 0.8, n), vy=rng.uniform(-0.8, 0.8, n), vz=rng.uniform(-0.8, 0.8, n),
               p=rng.uniform(0.3, 1.5, n), bx=rng.uniform(-1, 1, n), by=rng.uniform(-1, 1, n), bz=rng.uniform(-1, 1, n),
               psi=rng.uniform(-0.01, 0.01, n), X=rng.uniform(0, 1, n))
    out = []
    for _ in range(2):
        out.append(states(n, **{k: v + width.get(k, width["all"]) * rng.uniform(-0.5, 0.5, n) for k, v in mid.items()}))
    return out


@pytest.mark.parametrize("riemann", ["hlld", "hllc"])
@pytest.mark.parametrize("jump", [1e-12, 1e-6, 1e-2, 0.1])
def test_accuracy_over_jumps(host, jump, riemann):
    left, right = _random(np.random.default_rng(2), 20000, all=jump, psi=0.01 * jump)
    assert_accurate(host, left, right, riemann, 0.5)


def test_nearly_stationary_alfven_wave(host):
    """S_M -+ |B_n| / sqrt(rho*) swept through zero: the rotation's flux is switched by the sign of a
    difference that cancels."""
    rng = np.random.default_rng(3)
    n = 20000
    rho, b, bt, th = rng.uniform(0.5, 1.5, n), rng.uniform(0.2, 1, n), rng.uniform(0.2, 1, n), rng.uniform(0, 2 * np.pi, n)
    v = rng.choice([-1.0, 1.0], n) * b / np.sqrt(rho) * (1 + 10.0 ** rng.uniform(-16, -2, n) * rng.choice([-1.0, 1.0], n))
    common = dict(rho=rho, vx=v, p=rng.uniform(0.3, 1.5, n), bx=b * rng.choice([-1.0, 1.0], n), X=0.5)
    left, right = (states(n, by=bt * np.cos(a), bz=bt * np.sin(a), **common) for a in (th, th + rng.uniform(-0.02, 0.02, n)))
    assert_accurate(host, left, right, "hlld", 0.9)


def test_normal_fields_that_cancel(host):
    """B_n of the two sides nearly opposite: the sign and size of their mean come from what is left."""
    rng = np.random.default_rng(4)
    n = 20000
    b, by, bz = rng.uniform(0.2, 1, n), rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    left, right = (states(n, rho=rng.uniform(0.9, 1.1, n), vx=rng.uniform(-1e-9, 1e-9, n), vy=rng.uniform(-0.01, 0.01, n),
                          vz=rng.uniform(-0.01, 0.01, n), p=1.0, bx=x, by=by + rng.uniform(-0.01, 0.01, n), bz=bz)
                   for x in (b, -b * (1 + 10.0 ** rng.uniform(-16, -6, n) * rng.choice([-1.0, 1.0], n))))
    assert_accurate(host, left, right, "hlld", 0.9)


def _mirrored(P):
    M = P.copy()
    M[:, [VX, BX]] *= -1.0
    return M


@pytest.mark.parametrize("riemann", ["hlld", "hllc"])
@pytest.mark.parametrize("ratio", [1.0, 10.0, 1e3, 1e6])
def test_mirror_images_and_density_ratios(host, ratio, riemann):
    """Swapping the sides and mirroring the normal axis mirrors the flux bit for bit, whichever side is
    the denser, and the flux keeps its accuracy on both."""
    rng = np.random.default_rng(5)
    left, right = _random(rng, 20000, all=0.1, bx=0.0, psi=0.001)
    for P, k in ((left, 1.0), (right, ratio)):
        P[:, DEN] *= k
        P[:, ENE] /= k
        P[:, CS] = np.sqrt(GAM * P[:, PRE] / P[:, DEN])
    for a, b in ((left, right), (right, left)):
        F, ok = faces(host, a, b, riemann)
        G, ok2 = faces(host, _mirrored(b), _mirrored(a), riemann)
        moving = F[:, 0] != 0  # (at S_M = 0 both take the left side)
        sign = np.array([-1, 1, -1, -1, -1, 1, -1, -1, -1, -1.0])
        assert np.array_equal(ok, ok2) and ok.any()
        both = ok & moving
        assert np.array_equal(F[both], (G * sign)[both])
        assert_accurate(host, a, b, riemann, 0.2)


@pytest.mark.parametrize("kind", ["rotation", "sheet"])
def test_strong_jumps_are_left_to_the_general_flux(host, kind):
    """Jumps that the outer waves do not carry, where FP64 rounds at 2^-53 of rho w^2 (and so on): a pair's
    2^-46 of the jump is accepted up to a jump of 2^-5, with two bits for the number of operations."""
    rng = np.random.default_rng(6)
    n = 20000
    rho, b, bt, p = rng.uniform(0.5, 1.5, n), rng.uniform(0.2, 1, n), rng.uniform(0.2, 1, n), rng.uniform(0.3, 1.5, n)
    if kind == "rotation":  # nearly stationary, any angle
        v = b / np.sqrt(rho) * (1 + 1e-8 * rng.uniform(-1, 1, n))
        th = rng.uniform(0, 2 * np.pi, (2, n)) * 10.0 ** rng.uniform(-3, 0, n)
        left, right = (states(n, rho=rho, vx=v, p=p, bx=b, by=bt * np.cos(a), bz=bt * np.sin(a), X=0.5) for a in th)
    else:  # a static sheet, balanced to rounding
        b2 = bt * (1 - 10.0 ** rng.uniform(-3, 0, n))
        left, right = (states(n, rho=rho, p=p + (bt * bt - f * f) / 2, by=f, vy=0.1, X=0.5) for f in (bt, b2))
    F, ok = faces(host, left, right)
    ref, _ = reference(left, right)
    assert 0.2 < ok.mean() < 0.9
    w = np.abs(left[:, VX]) + np.sqrt(np.maximum(*((GAM * P[:, PRE] + (P[:, BX:PSI] ** 2).sum(axis=1)) / P[:, DEN]
                                                   for P in (left, right))))
    unit = {0: rho * w, 1: rho * w ** 2, 2: rho * w ** 2, 3: rho * w ** 2, 4: rho * w ** 3, 6: np.sqrt(rho) * w ** 2,
            7: np.sqrt(rho) * w ** 2, 9: rho * w}
    for m, u in unit.items():
        assert (np.abs(F[:, m] - ref[:, m])[ok] <= 2.0 ** -49 * u[ok]).all(), m
