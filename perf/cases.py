"""The work a user of the solver has it do, as cases that can be timed and checked.

A case is one call sequence of a user's program on one grid (or one ensemble of grids):

  host      Solver.step_host: the state lives in the program's page-locked memory, every call
            advances it by `steps` steps and writes the new state back (a coupled program with one
            step per call; a run with many steps between two looks at the state)
  resident  upload_cons, step(steps), sync, download_cons: a job that keeps the state on the device
  stage     upload_cons and one pass through the reference-shaped stage functions (stage_step)
  ensemble  the resident job over uneven Kelvin-Helmholtz grids advanced together

Every pass starts from the same input state, so passes can be repeated without end.  The states are
those of the benchmark and the studies: the Kelvin-Helmholtz layer (periodic x and z, reflecting y),
decaying turbulence in a periodic box, and a smooth state with every field non-trivial behind mixed
boundaries.
"""
import math

import numpy as np
import torch

NGH = 2
KH_DOMAIN = ((-0.5, 0.5), (-1.0, 1.0), (-0.5, 0.5))
CUBE_DOMAIN = ((-0.5, 0.5), (-0.5, 0.5), (-0.5, 0.5))
PERIODIC, REFLECTION, OUTFLOW = 1, 2, 3
DOMAINS = {"kh": KH_DOMAIN, "turb": CUBE_DOMAIN, "smooth": CUBE_DOMAIN}
BOUNDARIES = {
    "kh": (PERIODIC, PERIODIC, REFLECTION, REFLECTION, PERIODIC, PERIODIC),
    "turb": (PERIODIC,) * 6,
    "smooth": (OUTFLOW, REFLECTION, PERIODIC, PERIODIC, REFLECTION, OUTFLOW),
}
GAM = 5.0 / 3.0
ENSEMBLE_SIZES = (32, 48, 64, 96, 128)  # extents of the benchmark's ensemble members


def _case(name, mode, precision, nx, ny, nz, steps, state="kh", riemann="hlld", cfl=0.05, members=1):
    return {"name": name, "mode": mode, "precision": precision, "nx": nx, "ny": ny, "nz": nz, "steps": steps,
            "state": state, "riemann": riemann, "cfl": cfl, "members": members}


def listed():
    return [
        # a small grid of the tests stepped once per call by a program that keeps the state: latency
        _case("host_fp64_24x40x20", "host", "fp64", 24, 40, 20, 1, "smooth"),
        # a small study: many steps of a small grid between two looks at it, launches and tails count
        _case("resident_mixed_32x48x24", "resident", "mixed", 32, 48, 24, 64),
        # the reference's benchmark problem, one step per call on the program's own array
        _case("host_fp64_150", "host", "fp64", 150, 150, 150, 1),
        # the same in the mixed form
        _case("host_mixed_150", "host", "mixed", 150, 150, 150, 1),
        # the benchmark run itself: steps on the device in the two forms
        _case("resident_fp64_150", "resident", "fp64", 150, 150, 150, 4),
        _case("resident_mixed_150", "resident", "mixed", 150, 150, 150, 32),
        # decaying turbulence 256^3, the largest grid of the studies in both forms
        _case("host_fp64_turb_256", "host", "fp64", 256, 256, 256, 1, "turb"),
        _case("resident_mixed_turb_256", "resident", "mixed", 256, 256, 256, 8, "turb"),
        # odd extents, mixed boundaries and the alternative Riemann solvers
        _case("resident_fp64_hllc_97x61x75", "resident", "fp64", 97, 61, 75, 4, "smooth", "hllc"),
        # separately rounded arithmetic (the reference's, bit for bit) in the fused step
        _case("resident_exact_100x62x90", "resident", "fp64_exact", 100, 62, 90, 2),
        # a reference-shaped main loop: one function per stage
        _case("stage_fp64_64x96x48", "stage", "fp64", 64, 96, 48, 1),
        # a parameter study: uneven Kelvin-Helmholtz grids advanced together
        _case("ensemble_mixed_12", "ensemble", "mixed", 0, 0, 0, 16, members=12),
    ]


# Rough time of one cell and step in nanoseconds, to keep a drawn case below the largest listed one.
_COST = {"fp64": 2.7, "fp64_exact": 6.0, "mixed": 0.15, "stage": 8.0}


def draw(rng):
    mode = rng.choice(("host", "host", "resident", "resident", "resident", "stage", "ensemble"))
    precision = "fp64" if mode == "stage" else rng.choice(("fp64", "fp64", "mixed", "mixed", "fp64_exact"))
    if mode == "ensemble":
        precision = rng.choice(("fp64", "mixed"))
        return {"mode": mode, "precision": precision, "nx": 0, "ny": 0, "nz": 0,
                "steps": rng.choice((1, 2)) if precision == "fp64" else rng.choice((4, 16, 32)), "state": "kh",
                "riemann": "hlld", "cfl": 0.05, "members": rng.randint(3, 10)}
    state = rng.choice(("kh", "kh", "smooth", "turb"))
    riemann = rng.choice(("hlld",) * 5 + ("hlle", "hllc"))
    steps = 1 if mode == "stage" else rng.choice((1, 2, 3, 5) if precision != "mixed" else (1, 4, 17, 40))
    cost = _COST["stage" if mode == "stage" else precision]
    while True:
        nx, ny, nz = (round(math.exp(rng.uniform(math.log(6), math.log(256)))) for _ in range(3))
        cells = nx * ny * nz
        if cells >= 2000 and cells * (steps * cost + 0.5) < 40e6:
            break
    return {"mode": mode, "precision": precision, "nx": nx, "ny": ny, "nz": nz, "steps": steps, "state": state,
            "riemann": riemann, "cfl": rng.choice((0.05, 0.05, 0.05, 0.3)) if state != "smooth" else 0.05,
            "members": 1}


def _members(case):
    """The grids of a case: dicts of extents and Kelvin-Helmholtz parameters."""
    if case["mode"] != "ensemble":
        return [{"nx": case["nx"], "ny": case["ny"], "nz": case["nz"], "mach": 0.5 / math.sqrt(GAM), "bx": 0.1}]
    r = np.random.default_rng(2026 + case["members"])
    out = []
    for _ in range(case["members"]):
        nx, ny, nz = (int(r.choice(ENSEMBLE_SIZES)) for _ in range(3))
        out.append({"nx": nx, "ny": ny, "nz": nz, "mach": float(r.uniform(0.3, 1.5)), "bx": float(r.uniform(0.0, 0.3))})
    return out


# ---- initial states -------------------------------------------------------------------------------

def _faces(n, lo, hi):
    dx = (hi - lo) / float(n)
    return dx * (torch.arange(n + 2 * NGH + 1, dtype=torch.float64, device="cuda") - (NGH + 1)) + lo


def _mesh(n, domain):
    c = []
    for m, (lo, hi) in zip(n, domain):
        xa = _faces(m, lo, hi)
        c.append((0.5 * (xa[1:] + xa[:-1]))[NGH:NGH + m])
    z, y, x = torch.meshgrid(c[2], c[1], c[0], indexing="ij")
    return x, y, z


def _spectral(shape, gen):
    """Real random-phase field with 3-D power ~ k^-2 on 1 <= |k| <= 8, unit rms."""
    nz, ny, nx = shape
    f = [torch.fft.fftfreq(nz, 1.0 / nz), torch.fft.fftfreq(ny, 1.0 / ny), torch.fft.rfftfreq(nx, 1.0 / nx)]
    kz, ky, kx = torch.meshgrid(*(a.to("cuda", torch.float64) for a in f), indexing="ij")
    k = torch.sqrt(kx * kx + ky * ky + kz * kz)
    amp = torch.where((k >= 1.0) & (k <= 8.0), 1.0 / k.clamp_min(1e-30), torch.zeros_like(k))
    phase = 2.0 * math.pi * torch.rand(k.shape, dtype=torch.float64, device="cuda", generator=gen)
    g = torch.fft.irfftn(torch.polar(amp, phase), s=shape)
    return g / torch.sqrt(torch.mean(g * g)), (kx, ky, kz)


def _prims(case, m, seed):
    """rho, vx, vy, vz, p, bx, by, bz, psi, X of the interior, each (nz, ny, nx)."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n = (m["nx"], m["ny"], m["nz"])
    shape = (n[2], n[1], n[0])
    if case["state"] == "turb":
        g, (kx, ky, kz) = _spectral(shape, gen)
        rho = torch.exp(0.3 * g)
        rho = rho / rho.mean()
        v = [_spectral(shape, gen)[0] for _ in range(3)]
        s = 0.5 / torch.sqrt(torch.mean(v[0] ** 2 + v[1] ** 2 + v[2] ** 2))
        a = [torch.fft.rfftn(_spectral(shape, gen)[0]) for _ in range(3)]
        curl = (ky * a[2] - kz * a[1], kz * a[0] - kx * a[2], kx * a[1] - ky * a[0])
        b = [torch.fft.irfftn(2j * math.pi * c, s=shape) for c in curl]
        t = 0.4 / torch.sqrt(torch.mean(b[0] ** 2 + b[1] ** 2 + b[2] ** 2))
        o = torch.ones_like(rho)
        return rho, s * v[0], s * v[1], s * v[2], o, 0.2 * o + t * b[0], t * b[1], t * b[2], 0.0 * o, \
            0.5 + 0.5 * torch.tanh(4.0 * g)
    x, y, z = _mesh(n, DOMAINS[case["state"]])
    o = torch.ones_like(x)
    tp = 2.0 * math.pi
    if case["state"] == "smooth":
        r = tp * torch.rand(16, dtype=torch.float64, device="cuda", generator=gen)
        return (1.0 + 0.3 * torch.sin(tp * x + r[0]) * torch.cos(tp * y + r[1]) + 0.1 * torch.sin(tp * z + r[2]),
                0.4 * torch.sin(tp * y + r[5]) + 0.1 * torch.cos(tp * z + r[6]),
                0.4 * torch.sin(tp * z + r[7]) * torch.cos(tp * x + r[8]),
                0.4 * torch.cos(tp * x + r[9]) - 0.05,
                0.8 + 0.2 * torch.cos(tp * (x + y) + r[3]) * torch.sin(tp * z + r[4]),
                0.2 + 0.3 * torch.sin(tp * z + r[10]), 0.3 * torch.cos(tp * x + r[11]),
                -0.1 + 0.3 * torch.sin(tp * y + r[12]), 0.01 * torch.sin(tp * (x + z) + r[13]),
                0.5 + 0.4 * torch.sin(tp * y + r[14]) * torch.cos(tp * z + r[15]))
    noise = 1.0e-4 * (2.0 * torch.rand(shape, dtype=torch.float64, device="cuda", generator=gen) - 1.0)
    th = torch.tanh(y / 0.05)
    return (o, m["mach"] * math.sqrt(GAM) * th, 1.0e-2 * torch.sin(tp * x) * torch.exp(-(y / 0.2) ** 2) + noise,
            0.0 * o, o, m["bx"] * o, 0.0 * o, 0.0 * o, 0.0 * o, 0.5 * (1.0 + th))


def _cons(case, m, seed):
    """The conserved state in the solver's host layout (ktot, jtot, 10, itot), as a device tensor."""
    rho, vx, vy, vz, p, bx, by, bz, psi, X = _prims(case, m, seed)
    U = torch.zeros(m["nz"] + 5, m["ny"] + 5, 10, m["nx"] + 5, dtype=torch.float64, device="cuda")
    E = p / (GAM - 1.0) + 0.5 * rho * (vx * vx + vy * vy + vz * vz) + 0.5 * (bx * bx + by * by + bz * bz)
    for q, f in enumerate((rho, rho * vx, rho * vy, rho * vz, E, bx, by, bz, psi, rho * X)):
        U[2:-3, 2:-3, q, 2:-3] = f
    return U


# ---- the measured passes --------------------------------------------------------------------------

def _pinned(t):
    h = torch.empty(t.shape, dtype=torch.float64, pin_memory=True)
    h.copy_(t)
    return h


def prepare(case, seed):
    from mhdturbulence_gb300 import Ensemble, Solver
    ms = _members(case)
    kw = {"domain": DOMAINS[case["state"]], "bc": BOUNDARIES[case["state"]]}
    U = [_pinned(_cons(case, m, 1000 * seed + i)) for i, m in enumerate(ms)]
    out = [torch.zeros(u.shape, dtype=torch.float64, pin_memory=True) for u in U]
    if case["mode"] == "ensemble":
        e = Ensemble([{**kw, **m} for m in ms], precision=case["precision"], gam=GAM, cfl=case["cfl"])
        return {"case": case, "solver": e, "members": e.members, "U": U, "out": out}
    s = Solver(case["nx"], case["ny"], case["nz"], gam=GAM, cfl=case["cfl"], precision=case["precision"],
               riemann=case["riemann"], **kw)
    return {"case": case, "solver": s, "members": [s], "U": U, "out": out}


def _fetch(member, out):
    """The member's state into page-locked memory, through the C entry point (the Python method
    allocates a new pageable array for each call)."""
    import ctypes
    from mhdturbulence_gb300 import MhdgbError
    from mhdturbulence_gb300._lib import lib
    rc = lib().mhdgb_download_cons(member._h, ctypes.cast(out.data_ptr(), ctypes.POINTER(ctypes.c_double)))
    if rc:
        raise MhdgbError(rc, "download_cons")
    return out


def run(state):
    case, s = state["case"], state["solver"]
    if case["mode"] == "host":
        dt, ch = s.step_host(state["U"][0].numpy(), state["out"][0].numpy(), case["steps"])
        return {"U": state["out"], "dt": [dt], "chg": [ch]}
    for m, u in zip(state["members"], state["U"]):
        m.upload_cons(u.numpy())
    if case["mode"] == "stage":
        dt, ch = s.stage_step()
        return {"U": [_fetch(s, state["out"][0])], "dt": [dt], "chg": [ch]}
    s.step(case["steps"])
    reps = s.sync()
    reps = reps if isinstance(reps, list) else [reps]
    return {"U": [_fetch(m, o) for m, o in zip(state["members"], state["out"])], "dt": [r.dt for r in reps],
            "chg": [r.chg for r in reps]}


def work(case):
    """A step reads and writes the ten conserved fields (160 bytes a cell) and takes 2127 floating-point
    operations a cell in the reference's arithmetic (932 additions, 1063 products, 105 divisions, 26
    roots).  A pass brings the state in from the host and back out besides."""
    cells = sum(m["nx"] * m["ny"] * m["nz"] for m in _members(case))
    return {"bytes": 160.0 * cells * (case["steps"] + 1), "flops": 2127.0 * cells * case["steps"]}


# ---- the same steps in plain torch, 64 bits -------------------------------------------------------
# Fields are (nz+4, ny+4, nx+4) tensors.  Primitives: rho, v (3), e, p, c_s, B (3), psi, X; conserved:
# rho, m (3), E, B (3), psi, rho X.

def _recover(U):
    rho = U[0]
    ri = 1.0 / rho
    v = [U[q] * ri for q in (1, 2, 3)]
    ek = 0.5 * (U[1] * U[1] + U[2] * U[2] + U[3] * U[3]) * ri
    em = 0.5 * (U[5] * U[5] + U[6] * U[6] + U[7] * U[7])
    e = (U[4] - ek - em) / rho
    return torch.stack([rho, *v, e, e * rho * (GAM - 1.0), torch.sqrt(e * GAM * (GAM - 1.0)), U[5], U[6], U[7], U[8],
                        U[9] * ri])


def _fill(P, bc):
    """Ghost layers, two deep, of all three axes (edges and corners are never read)."""
    for a in range(3):
        ax = 3 - a
        n = P.shape[ax] - 4
        at = lambda i: P.select(ax, i)  # noqa: E731
        vals = {}
        for g in range(2):
            for side in range(2):
                kind = bc[2 * a + side]
                to = 1 - g if side == 0 else n + 2 + g  # g = 0 next to the interior
                if kind == PERIODIC:
                    f = at(n + 1 - g if side == 0 else 2 + g).clone()
                elif kind == REFLECTION:
                    f = at(2 + g if side == 0 else n + 1 - g).clone()
                    f[1 + a] = -f[1 + a]
                else:
                    f = at(2 if side == 0 else n + 1).clone()
                vals[to] = f
        for to, f in vals.items():
            at(to).copy_(f)


def _speeds(P, spacing, cfl):
    i = (slice(None),) + (slice(2, -2),) * 3
    rho, cs = P[0][i[1:]], P[6][i[1:]]
    v, b = [P[1 + d][i[1:]] for d in range(3)], [P[7 + d][i[1:]] for d in range(3)]
    css = cs * cs
    ctot = torch.sqrt(css + (b[0] ** 2 + b[1] ** 2 + b[2] ** 2) / rho)
    dt, ch = None, None
    for d in range(3):
        t = (spacing[d] / (v[d].abs() + ctot)).min()
        dt = t if dt is None else torch.minimum(dt, t)
        cts = css + (b[0] ** 2 + b[1] ** 2 + b[2] ** 2) / rho
        c = (v[d].abs() + torch.sqrt(0.5 * (cts + torch.sqrt(cts * cts - 4.0 * css * b[d] ** 2 / rho)))).max()
        ch = c if ch is None else torch.maximum(ch, c)
    return cfl * dt, ch


def _side(S):
    """Conserved vector, flux vector, fast speed and total pressure of one rotated face state."""
    rho, vx, vy, vz, e, p, cs, bx, by, bz, psi, X = S
    b2 = bx * bx + by * by + bz * bz
    E = rho * e + 0.5 * rho * (vx * vx + vy * vy + vz * vz) + 0.5 * b2
    pt = p + 0.5 * b2
    C = [rho, rho * vx, rho * vy, rho * vz, E, bx, by, bz, psi, rho * X]
    Fl = [rho * vx, rho * vx * vx - bx * bx + pt, rho * vy * vx - by * bx, rho * vz * vx - bz * bx,
          (E + pt) * vx - b2 * bx, 0.0 * bx, by * vx - vy * bx, bz * vx - vz * bx, 0.0 * bx, rho * X * vx]
    cts = cs * cs + b2 / rho
    cf = torch.sqrt(0.5 * (cts + torch.sqrt(cts * cts - 4.0 * cs * cs * bx * bx / rho)))
    return C, Fl, cf, pt


def _hlle(L, R, cl, cr, vl, vr):
    c = torch.maximum(cl, cr)
    sl, sr = (torch.minimum(vl, vr) - c).clamp(max=0.0), (torch.maximum(vl, vr) + c).clamp(min=0.0)
    return [(sr * L[1][q] - sl * R[1][q] + sl * sr * (R[0][q] - L[0][q])) / (sr - sl) for q in range(10)]


def _hllc(L, R, cl, cr, pl, pr, SL, SR):
    c = torch.maximum(cl, cr)
    vl, vr = SL[1], SR[1]
    sl, sr = torch.minimum(vl, vr) - c, torch.maximum(vl, vr) + c
    al, ar = SL[0] * (sl - vl), SR[0] * (sr - vr)
    d = 1.0 / (ar - al)
    sm = (ar * vr - al * vl - pr + pl) * d
    ps = (ar * pl - al * pr + al * ar * (vr - vl)) * d
    left = ~torch.signbit(sm)

    def side(S, C, Fl, a, s, pt, clip):
        i = 1.0 / (s - sm)
        ro = a * i
        k = ro / S[0]
        st = [ro, ro * sm, ro * S[2], ro * S[3], ((s - S[1]) * C[4] - pt * S[1] + ps * sm) * i, None, k * C[6], k * C[7],
              None, k * C[9]]
        return [Fl[q] if st[q] is None else Fl[q] + clip * (st[q] - C[q]) for q in range(10)]

    a = side(SL, L[0], L[1], al, sl, pl, sl.clamp(max=0.0))
    b = side(SR, R[0], R[1], ar, sr, pr, sr.clamp(min=0.0))
    return [torch.where(left, x, y) for x, y in zip(a, b)]


def _hlld(L, R, cl, cr, pl, pr, SL, SR):
    eps = 1.0e-30
    c = torch.maximum(cl, cr)
    vl, vr = SL[1], SR[1]
    sl, sr = torch.minimum(vl, vr) - c, torch.maximum(vl, vr) + c
    sdl, sdr = (sl - vl).clamp(max=-1e-20), (sr - vr).clamp(min=1e-20)
    al, ar = SL[0] * sdl, SR[0] * sdr
    d = 1.0 / (ar - al)
    sm = (ar * vr - al * vl - pr + pl) * d
    ps = (ar * pl - al * pr + al * ar * (vr - vl)) * d
    bx = 0.5 * (SL[7] + SR[7])
    bq = bx * bx

    def star(S, C, sd, a, sdm, pt):
        T = a * sdm - bq
        ok = T.abs() >= eps
        it = 1.0 / torch.where(ok, T, torch.ones_like(T))
        t1, t2 = bx * (sd - sdm) * it, (a * sd - bq) * it
        pick = lambda x, y: torch.where(ok, x, y)  # noqa: E731
        ro, vx = pick(a / sdm, S[0]), pick(sm, S[1])
        vy, vz = pick(S[2] - S[8] * t1, S[2]), pick(S[3] - S[9] * t1, S[3])
        by, bz = pick(S[8] * t2, S[8]), pick(S[9] * t2, S[9])
        vb = vx * bx + vy * by + vz * bz
        E = pick((sd * C[4] - pt * S[1] + ps * sm + bx * (S[1] * bx + S[2] * S[8] + S[3] * S[9] - vb)) / sdm, C[4])
        return ro, vx, vy, vz, by, bz, E, vb

    l = star(SL, L[0], sdl, al, (sl - sm).clamp(max=-1e-20), pl)
    r = star(SR, R[0], sdr, ar, (sr - sm).clamp(min=1e-20), pr)
    ql, qr = torch.sqrt(l[0]), torch.sqrt(r[0])
    on = bx.abs() >= eps
    sg = torch.copysign(torch.ones_like(bx), bx)
    inv = 1.0 / (ql + qr)
    vy = inv * (ql * l[2] + qr * r[2] + sg * (r[4] - l[4]))
    vz = inv * (ql * l[3] + qr * r[3] + sg * (r[5] - l[5]))
    by = inv * (ql * r[4] + qr * l[4] + sg * ql * qr * (r[2] - l[2]))
    bz = inv * (ql * r[5] + qr * l[5] + sg * ql * qr * (r[3] - l[3]))
    vb = sm * bx + vy * by + vz * bz

    def flux(S, C, Fl, st, q, s, ss, sign):
        E2 = st[6] + sign * sg * q * (vb - st[7])
        star_ = [st[0], st[0] * st[1], st[0] * st[2], st[0] * st[3], st[6], None, st[4], st[5], None, st[0] * S[11]]
        dbl = [st[0], st[0] * st[1], st[0] * vy, st[0] * vz, E2, None, by, bz, None, st[0] * S[11]]
        out = []
        for k in range(10):
            if star_[k] is None:
                out.append(torch.zeros_like(s))
            else:
                out.append(Fl[k] + s * (star_[k] - C[k]) + torch.where(on, ss * (dbl[k] - star_[k]), torch.zeros_like(s)))
        return out

    zero = torch.zeros_like(sm)
    a = flux(SL, L[0], L[1], l, ql, sl.clamp(max=0.0), torch.where(on, sm - bx.abs() / ql, zero).clamp(max=0.0), 1.0)
    b = flux(SR, R[0], R[1], r, qr, sr.clamp(min=0.0), torch.where(on, sm + bx.abs() / qr, zero).clamp(min=0.0), -1.0)
    left = ~torch.signbit(sm)
    return [torch.where(left, x, y) for x, y in zip(a, b)]


def _flux(P, d, chg, riemann):
    """Fluxes through the faces of axis d (interior transverse extent), in unrotated order."""
    ax = 3 - d
    idx = [slice(None)] + [slice(2, -2)] * 3
    idx[ax] = slice(None)
    Q = P[tuple(idx)]
    n = Q.shape[ax] - 4
    D = Q.narrow(ax, 1, n + 3) - Q.narrow(ax, 0, n + 3)
    pr = D.narrow(ax, 1, n + 2) * D.narrow(ax, 0, n + 2)
    sm = D.narrow(ax, 1, n + 2) + D.narrow(ax, 0, n + 2)
    sl = torch.where(pr > 0.0, 2.0 * pr / torch.where(pr > 0.0, sm, torch.ones_like(sm)), torch.zeros_like(pr))
    rot = [0, 1 + d, 1 + (d + 1) % 3, 1 + (d + 2) % 3, 4, 5, 6, 7 + d, 7 + (d + 1) % 3, 7 + (d + 2) % 3, 10, 11]
    Cl, Cr = Q.narrow(ax, 1, n + 1), Q.narrow(ax, 2, n + 1)
    sL, sR = sl.narrow(ax, 0, n + 1), sl.narrow(ax, 1, n + 1)
    SL, SR = [Cl[q] + 0.5 * sL[q] for q in rot], [Cr[q] - 0.5 * sR[q] for q in rot]
    L, R = _side(SL), _side(SR)
    if riemann == "hlle":
        f = _hlle(L, R, L[2], R[2], SL[1], SR[1])
    else:
        f = (_hllc if riemann == "hllc" else _hlld)(L, R, L[2], R[2], L[3], R[3], SL, SR)
    f[5] = 0.5 * (SL[10] + SR[10]) - 0.5 * chg * (SR[7] - SL[7])
    f[8] = (0.5 * (SL[7] + SR[7]) - 0.5 / chg * (SR[10] - SL[10])) * chg * chg
    out = [None] * 10
    for q, to in enumerate((0, 1 + d, 1 + (d + 1) % 3, 1 + (d + 2) % 3, 4, 5 + d, 5 + (d + 1) % 3, 5 + (d + 2) % 3, 8, 9)):
        out[to] = f[q]
    return torch.stack(out)


def _advance(U, n, domain, bc, cfl, steps, riemann):
    """U (10, nz, ny, nx) after `steps` steps, with the last step's dt and c_h."""
    spacing = []
    for a, (m, (lo, hi)) in enumerate(zip(n, domain)):
        xa = _faces(m, lo, hi)
        shape = [1, 1, 1]
        shape[2 - a] = m
        spacing.append((xa[1:] - xa[:-1])[NGH:NGH + m].reshape(shape))
    small = torch.minimum(torch.minimum(spacing[0], spacing[1]), spacing[2])
    P = torch.zeros(12, n[2] + 4, n[1] + 4, n[0] + 4, dtype=torch.float64, device="cuda")
    dt = chg = None
    for _ in range(steps):
        P[:, 2:-2, 2:-2, 2:-2] = _recover(U)
        _fill(P, bc)
        dt, chg = _speeds(P, spacing, cfl)
        div = torch.zeros_like(U)
        for d in range(3):
            F = _flux(P, d, chg, riemann)
            m = F.shape[3 - d] - 1
            div += (F.narrow(3 - d, 1, m) - F.narrow(3 - d, 0, m)) * (1.0 / spacing[d])
        U = U - dt * div
        U[8] = U[8] * (1.0 - dt * (0.1 * chg / small))
    return U, dt, chg


def exact(case, seed):
    out = {"U": [], "dt": [], "chg": []}
    for i, m in enumerate(_members(case)):
        n = (m["nx"], m["ny"], m["nz"])
        U = _cons(case, m, 1000 * seed + i)
        V, dt, chg = _advance(U[2:-3, 2:-3, :, 2:-3].permute(2, 0, 1, 3).contiguous(), n, DOMAINS[case["state"]],
                              BOUNDARIES[case["state"]], case["cfl"], case["steps"], case["riemann"])
        U[2:-3, 2:-3, :, 2:-3] = V.permute(1, 2, 0, 3)
        out["U"].append(U)
        out["dt"].append(float(dt))
        out["chg"].append(float(chg))
    return out
