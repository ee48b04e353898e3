"""The solver's performance cases: what programs that use it have it do, through its public calls.

Four kinds of work, each with the sizes and data of this repository's configurations and tests:

* solve    -- u from source samples of the constant-k problem (Plan.solve_source), 2D and 3D, orders
              2, 4 and 6, one field or a batch: the benchmark configurations, the README problem, the
              sizes the request loop serves, and the grid sizes the published tables use (50, 100,
              125, 197, 500: n + 1 is no power of two there);
* general  -- assembled right-hand sides on a plan made from stencil rows (Plan.solve);
* pipeline -- the program's main sequence on a variable-k problem: rhs() on the device, then solver()
              (Plan.assemble_rhs, Plan.solve); the 2D problem has complex k(y) = y^2 + iy, the 3D one
              is the published k(z) = 10 - 9 sin 10z;
* multi    -- one batch over several wavenumbers of one shape (solve_source_multi), as the request
              loop runs requests that share a shape.

A plan is kept from call to call, as every such program does; throughput cases tune it first, as the
benchmark does (the result is cached per shape), single solves take a new plan as it comes.
"""
import math
import random

import numpy as np
import torch

import hackathon_b200 as hh

LEGACY_STREAM = 1  # cudaStreamLegacy: the stream that torch's default stream is


def _solve(name, dim, n, order, k, batch, tune):
    return {"name": name, "kind": "solve", "dim": dim, "n": n, "order": order, "k": k, "k_im": 0.0, "batch": batch,
            "tune": tune}


def listed():
    return [
        # one README-sized solve (N = 100, order 6, k = 10): latency of a single small call
        _solve("readme_2d_100", 2, 100, 6, 10.0, 1, False),
        # one request of the served mix at an ordinary size
        _solve("single_2d_255", 2, 255, 4, 20.0, 1, False),
        # the benchmark's headline batch, at its two orders
        _solve("batch_2d_1023_o6", 2, 1023, 6, 50.0, 64, True),
        _solve("batch_2d_1023_o4", 2, 1023, 4, 200.0, 64, True),
        # the large 2D configuration
        _solve("batch_2d_2047", 2, 2047, 6, 100.0, 16, True),
        # a batch at a size a user types in (the published tables' N = 500, in 2D)
        _solve("batch_2d_500", 2, 500, 6, 30.0, 16, True),
        # the smallest served 3D shape
        _solve("small_3d_31", 3, 31, 4, 10.0, 8, False),
        # the 3D configuration
        _solve("batch_3d_255", 3, 255, 6, 30.0, 4, True),
        # 3D at an ordinary typed-in size
        _solve("batch_3d_100", 3, 100, 6, 20.0, 4, True),
        # the published 3D problem at 125^3 (6th-order accuracy table): rhs() then solver()
        {"name": "pipeline_3d_125", "kind": "pipeline", "dim": 3, "n": 125},
        # the reference program's 2D problem, complex variable k: rhs() then solver()
        {"name": "pipeline_2d_511", "kind": "pipeline", "dim": 2, "n": 511},
        # requests at eight wavenumbers that the request loop merges into one batch
        {"name": "multi_2d_255", "kind": "multi", "n": 255, "order": 4, "plans": 8, "per": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["solve", "solve", "solve", "solve", "general", "pipeline", "multi"])
    if kind == "solve":
        dim = rng.choice([2, 2, 3])
        pow2 = rng.random() < 0.4  # n + 1 a power of two, or any size
        if dim == 2:
            n = rng.choice([63, 127, 255, 511, 1023, 2047]) if pow2 else _log_int(rng, 40, 700)
            most = 64 * 1023 ** 2 / n ** 2 if pow2 else min(64.0, 16 * 500.0 ** 3 / n ** 3)
        else:
            n = rng.choice([31, 63, 127]) if pow2 else _log_int(rng, 20, 120)
            most = 4 * 255 ** 3 / n ** 3 if pow2 else min(32.0, 4 * 100.0 ** 4 / n ** 4)
        batch = _log_int(rng, 1, max(1, min(64, int(most))))
        return {"kind": "solve", "dim": dim, "n": n, "order": rng.choice([2, 4, 6, 6]), "k": round(rng.uniform(1.0, 0.4 * n), 3),
                "k_im": round(rng.uniform(1.0, 5.0), 3) if rng.random() < 0.2 else 0.0, "batch": batch,
                "tune": batch >= 4 and rng.random() < 0.5}
    if kind == "general":
        n = rng.choice([127, 255, 511, _log_int(rng, 40, 500)])
        return {"kind": "general", "n": n, "batch": _log_int(rng, 1, max(1, min(16, int(16 * 300.0 ** 3 / n ** 3))))}
    if kind == "pipeline":
        dim = rng.choice([2, 3])
        return {"kind": "pipeline", "dim": dim, "n": _log_int(rng, 63, 640) if dim == 2 else _log_int(rng, 24, 128)}
    return {"kind": "multi", "n": rng.choice([63, 127, 255, 511, _log_int(rng, 50, 300)]), "order": rng.choice([2, 4, 6]),
            "plans": rng.randint(2, 12), "per": rng.randint(1, 4)}


def _points(case):
    if case["kind"] == "solve":
        return case["n"] ** case["dim"] * case["batch"]
    if case["kind"] == "general":
        return case["n"] ** 2 * case["batch"]
    if case["kind"] == "pipeline":
        return case["n"] ** case["dim"]
    return case["n"] ** 2 * case["plans"] * case["per"]


def work(case):
    """Source in, solution out (the pipelines: the source on the extended grid in, rhs and solution
    out), 16 bytes a value; the transforms as complex FFTs of length n + 1, about 40 operations a
    point for the line solve and 40 for an assembly."""
    pts, dim = _points(case), case.get("dim", 2)
    fft = 5.0 * math.log2(case["n"] + 1) + 10.0
    flops = pts * (2 * (dim - 1) * fft + 40.0)
    if case["kind"] == "pipeline":
        return {"bytes": 16.0 * ((case["n"] + 2) ** dim + 2 * pts), "flops": flops + 40.0 * pts}
    return {"bytes": 32.0 * pts, "flops": flops}


# ------------------------------------------------------------------------------- inputs --------

def _sources(dim, n, batch, seed, device):
    """Sine-mode sources with a little noise at every point, as the benchmark configurations have."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    modes, pmax = 16, max(2, min(200, n // 2))
    x = torch.arange(1, n + 1, dtype=torch.float64, device=device) / (n + 1)
    out = torch.empty((batch,) + (n,) * dim, dtype=torch.complex128, device=device)
    noise = torch.Generator(device=device).manual_seed(seed + 1)
    for b in range(batch):
        amp = torch.view_as_complex(torch.randn((modes, 2), dtype=torch.float64, generator=g)).to(device)
        s = [torch.sin(math.pi * torch.randint(1, pmax + 1, (modes, 1), generator=g).to(device) * x).to(torch.complex128)
             for _ in range(dim)]
        if dim == 2:
            out[b] = (s[1] * amp[:, None]).T @ s[0]
        else:
            yx = (s[1][:, :, None] * s[0][:, None, :]).reshape(modes, n * n)
            out[b] = ((s[2] * amp[:, None]).T @ yx).reshape(n, n, n)
        out[b] += 0.02 * torch.view_as_complex(
            torch.randn((n,) * dim + (2,), dtype=torch.float64, device=device, generator=noise))
    return out


def _multi_k(case, seed):
    r = random.Random(seed)
    return [r.uniform(1.0, 0.4 * case["n"]) for _ in range(case["plans"])]


def _pade(v, diag):
    """tridiag(1, diag, 1)^-1 along the first axis, Thomas."""
    n = v.shape[0]
    u = np.empty(n)
    u[0] = diag
    for j in range(1, n):
        u[j] = diag - 1.0 / u[j - 1]
    v = v.copy()
    for j in range(1, n):
        v[j] -= v[j - 1] / u[j - 1]
    v[n - 1] /= u[n - 1]
    for j in range(n - 2, -1, -1):
        v[j] = (v[j] - v[j + 1]) / u[j]
    return v


def _problem_2d(n, seed):
    """The 2D program's problem, k(y) = y^2 + iy on [0.5, pi - 0.5]^2, scaled, with a little noise on
    the interior source."""
    rng = np.random.default_rng(seed)
    amp = rng.uniform(0.5, 2.0)
    x0, x1 = 0.5, math.pi - 0.5
    h = (x1 - x0) / (n + 1)
    g = x0 + h * np.arange(n + 2)
    k = g * g + 1j * g

    def k2y(y):
        return 4.0 * y ** 3 + 6.0j * y * y - 2.0 * y

    def k2yy(y):
        return 12.0 * y * y + 12.0j * y - 2.0

    def kk(y):
        return (y * y + 1j * y) ** 2

    def f(x, y):
        return (kk(y) - 2.0) * np.sin(x) * np.sin(y)

    def fy(x, y):
        return (kk(y) - 2.0) * np.sin(x) * np.cos(y) + k2y(y) * np.sin(x) * np.sin(y)

    def fxx(x, y):
        return (2.0 - kk(y)) * np.sin(x) * np.sin(y)

    def fyy(x, y):
        return (2.0 - kk(y) + k2yy(y)) * np.sin(x) * np.sin(y) + 2.0 * k2y(y) * np.sin(x) * np.cos(y)

    fe = amp * f(g[None, :], g[:, None])
    fe[1:-1, 1:-1] += 1e-3 * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
    c = lambda a: np.ascontiguousarray(a, dtype=np.complex128)  # noqa: E731
    d = dict(f_ext=c(fe),
             fxx_xb=c(amp * np.concatenate([fxx(x0, g), fxx(x1, g)])), fxx_yb=c(amp * np.concatenate([fxx(g, x0), fxx(g, x1)])),
             fyy_xb=c(amp * np.concatenate([fyy(x0, g), fyy(x1, g)])), fyy_yb=c(amp * np.concatenate([fyy(g, x0), fyy(g, x1)])),
             fy_yb=c(amp * np.concatenate([fy(g[1:-1], x0), fy(g[1:-1], x1)])),
             u_xb=amp * np.concatenate([math.sin(x0) * np.sin(g), math.sin(x1) * np.sin(g)]),
             u_yb=amp * np.concatenate([np.sin(g) * math.sin(x0), np.sin(g) * math.sin(x1)]))
    k2 = k * k
    h2, h3, h4 = h ** 2, h ** 3, h ** 4
    ky, kyy, kp, km, kc = k2y(g[1:-1]), k2yy(g[1:-1]), k2[2:], k2[:-2], k2[1:-1]
    coef = dict(ap=2 / 3 + h2 * kp / 90 + h3 * ky * (h2 * kp / 6 + 2 / 3) / 20, bp=1 / 6 + h2 * kp / 90 + h3 * ky / 120,
                a=-10 / 3 + 41 * h2 * kc / 45 - h4 * kc * kc / 20 + h4 * kyy / 20, b=2 / 3 + h2 * kc / 90,
                am=2 / 3 + h2 * km / 90 - h3 * ky * (h2 * km / 6 + 2 / 3) / 20, bm=1 / 6 + h2 * km / 90 - h3 * ky / 120)
    return h, c(k), c([k2y(x0), k2y(x1)]), coef, d


def _problem_3d(n, seed):
    """The published 3D problem (A = 10, B = 9, C = 10, gamma = 9 on [0, pi]^3), scaled, with a little
    noise on the interior source."""
    rng = np.random.default_rng(seed)
    amp = rng.uniform(0.5, 2.0)
    A, B, Cc, gamma, x1 = 10.0, 9.0, 10.0, 9.0, math.pi
    h = x1 / (n + 1)
    beta = math.sqrt(A * A + B * B - gamma * gamma)
    z = h * np.arange(n + 2)
    k = A - B * np.sin(Cc * z)
    ue = amp * np.exp(-k / Cc)[:, None, None] * np.sin(beta * z)[None, :, None] * np.sin(gamma * z)[None, None, :]
    f = -h * h * B * (2.0 * A + Cc) * np.sin(Cc * z)[:, None, None] * ue
    fxx = np.concatenate([(-gamma ** 2 * f[:, :, 0]).ravel(), (-gamma ** 2 * f[:, :, n + 1]).ravel()])
    fyy = np.concatenate([(-beta ** 2 * f[:, 0, :]).ravel(), (-beta ** 2 * f[:, n + 1, :]).ravel()])

    def zterm(zz):
        s, co = math.sin(Cc * zz), math.cos(Cc * zz)
        return B * Cc * s * s + s * (Cc * Cc - B * B * co * co) - 2.0 * B * Cc * co * co

    fzz = h * h * B * (2.0 * A + Cc) * np.concatenate([(ue[0] * zterm(0.0)).ravel(), (ue[n + 1] * zterm(x1)).ravel()])
    f = f.astype(np.complex128)
    f[1:-1, 1:-1, 1:-1] += 1e-3 * h * h * (rng.standard_normal((n, n, n)) + 1j * rng.standard_normal((n, n, n)))
    kz_bc = np.array([2 * B * Cc * math.cos(Cc * t) * (A - B * math.sin(Cc * t)) for t in (0.0, x1)])
    kzz_bc = np.array([2 * B * Cc * Cc * (B * math.sin(Cc * t) ** 2 - A * math.sin(Cc * t) - B * math.cos(Cc * t) ** 2)
                       for t in (0.0, x1)])
    k2 = k * k
    kp, kpp = 3.0 * (k2[2:] - k2[:-2]) / h, 12.0 * (k2[2:] - 2.0 * k2[1:-1] + k2[:-2]) / h / h
    kp[0] += kz_bc[0]
    kp[-1] += kz_bc[1]
    kpp[0] += kzz_bc[0]
    kpp[-1] += kzz_bc[1]
    kp, kpp = _pade(kp, 4.0), _pade(kpp, 10.0)
    h2, h3, h4 = h ** 2, h ** 3, h ** 4
    kc, ku, kd = k2[1:-1], k2[2:], k2[:-2]
    one = np.ones(n)
    coef = dict(a=1 / 10 + h2 * kc / 90, b=7 / 15 - h2 * kc / 90, c=7 / 15 - h2 * kc / 90,
                d=-64 / 15 + 14 * h2 * kc / 15 - h4 * kc * kc / 20 + h4 * kpp / 20, ap=one / 30, am=one / 30,
                bp=1 / 10 + h2 * ku / 90 + kp * h3 / 120, cp=1 / 10 + h2 * ku / 90 + kp * h3 / 120,
                dp=7 / 15 - h2 * ku / 90 + kp * h3 / 20 * (1 / 3 + ku * h2 / 6),
                bm=1 / 10 + h2 * kd / 90 - kp * h3 / 120, cm=1 / 10 + h2 * kd / 90 - kp * h3 / 120,
                dm=7 / 15 - h2 * kd / 90 - kp * h3 / 20 * (1 / 3 + kd * h2 / 6))
    c = lambda a: np.ascontiguousarray(a, dtype=np.complex128)  # noqa: E731
    d = dict(f_ext=c(f), fxx_b=c(fxx), fyy_b=c(fyy), fzz_b=c(fzz), ue_ext=c(ue))
    return h, c(k2), c(kz_bc), coef, kp, d


def _general_rhs(case, seed, device):
    g = torch.Generator(device=device).manual_seed(seed)
    return torch.view_as_complex(torch.randn((case["batch"], case["n"], case["n"], 2), dtype=torch.float64, device=device,
                                             generator=g))


# -------------------------------------------------------------------------------- running ------

def prepare(case, seed):
    ctx = hh.Context(0, LEGACY_STREAM)
    kind, n = case["kind"], case["n"]
    st = {"case": case, "ctx": ctx}
    if kind == "solve":
        st["f"] = _sources(case["dim"], n, case["batch"], seed, "cuda")
        st["u"] = torch.empty_like(st["f"])
        st["plan"] = hh.Plan.helmholtz(ctx, case["dim"], n, case["order"], complex(case["k"], case["k_im"]))
        if case["tune"]:
            st["plan"].tune(case["batch"])
    elif kind == "multi":
        total = case["plans"] * case["per"]
        st["f"] = _sources(2, n, total, seed, "cuda")
        st["u"] = torch.empty_like(st["f"])
        st["plans"] = [hh.Plan.helmholtz(ctx, 2, n, case["order"], k) for k in _multi_k(case, seed)]
    elif kind == "general":
        _, _, _, coef, _ = _problem_2d(n, seed)
        st["plan"] = hh.Plan.from_coefficients_2d(ctx, n, n, coef)
        st["f"] = _general_rhs(case, seed, "cuda")
        st["u"] = torch.empty_like(st["f"])
    elif case["dim"] == 2:
        h, k, k2y_bc, coef, d = _problem_2d(n, seed)
        st["plan"] = hh.Plan.from_coefficients_2d(ctx, n, n, coef)
        st["data"] = {nm: torch.from_numpy(a).cuda() for nm, a in d.items()}
        st["host"] = dict(k_ext=k, k2y_bc=k2y_bc)
        st["h"] = (h, h)
        st["rhs"] = torch.empty((n, n), dtype=torch.complex128, device="cuda")
        st["u"] = torch.empty_like(st["rhs"])
    else:
        h, k2, kz_bc, coef, _, d = _problem_3d(n, seed)
        st["plan"] = hh.Plan.from_coefficients_3d(ctx, n, n, n, coef)
        st["data"] = {nm: torch.from_numpy(a).cuda() for nm, a in d.items()}
        st["host"] = dict(k2_ext=k2, kz_bc=kz_bc)
        st["h"] = (h, h, h)
        st["rhs"] = torch.empty((n, n, n), dtype=torch.complex128, device="cuda")
        st["u"] = torch.empty_like(st["rhs"])
    return st


def run(st):
    case = st["case"]
    if case["kind"] == "solve":
        st["plan"].solve_source(st["f"], st["u"], case["batch"])
    elif case["kind"] == "multi":
        hh.solve_source_multi(st["plans"], [case["per"]] * case["plans"], st["f"], st["u"])
    elif case["kind"] == "general":
        st["plan"].solve(st["f"], st["u"], case["batch"])
    else:
        st["plan"].assemble_rhs(st["rhs"], 6, st["h"], **st["data"], **st["host"])
        st["plan"].solve(st["rhs"], st["u"], 1)
        return {"rhs": st["rhs"], "u": st["u"]}
    return {"u": st["u"]}


# ---------------------------------------------------------------- the same, in plain 64 bits ----

def _dst(x, dim):
    """Orthonormal DST-I along `dim`, through the FFT of the odd extension."""
    x = x.movedim(dim, -1)
    n = x.shape[-1]
    z = torch.zeros(x.shape[:-1] + (1,), dtype=x.dtype, device=x.device)
    y = torch.fft.fft(torch.cat([z, x, z, -x.flip(-1)], -1))[..., 1:n + 1]
    return (y * (0.5j * math.sqrt(2.0 / (n + 1)))).movedim(-1, dim)


def _spectral(f, n, dim, order, k):
    """The compact scheme solved mode by mode along every axis (f: one field)."""
    h2 = 1.0 / (n + 1) ** 2
    k2 = k * k
    i = torch.arange(1, n + 1, dtype=torch.float64, device=f.device)
    lam = (2.0 * torch.cos(math.pi * i / (n + 1))).to(torch.complex128)
    # second difference by the half-angle form: lam - 2 = -4 sin^2
    d2 = (-4.0 * torch.sin(0.5 * math.pi * i / (n + 1)) ** 2).to(torch.complex128)
    mu = 12.0 * d2 / (12.0 + d2)
    ax = lambda v, a: v.reshape([-1 if b == a else 1 for b in range(dim)])  # noqa: E731
    L, D, M = ([ax(v, a) for a in range(dim)] for v in (lam, d2, mu))
    s = lambda vs: sum(vs[1:], vs[0])  # noqa: E731
    pairs = [(a, b) for a in range(dim) for b in range(a)]  # axes are z, y, x
    if order == 2:
        op, rhs = s(D) + k2 * h2, h2
    elif order == 4:
        rhs = h2 * (1.0 + s(D) / 12.0)
        op = s(D) + s([D[a] * D[b] for a, b in pairs]) / 6.0 + k2 * h2 * (1.0 + s(D) / 12.0)
    else:
        rhs = h2 * (1.0 - k2 * h2 / 20.0 + s(M) / 12.0 + s([D[a] * M[a] for a in range(dim)]) / 360.0
                    + s([D[b] * M[a] for a, b in pairs]) / 90.0)
        if dim == 2:
            a6, b6, c6 = -10 / 3 + 41 * h2 * k2 / 45 - h2 * h2 * k2 * k2 / 20, 2 / 3 + h2 * k2 / 90, 1 / 6 + h2 * k2 / 90
            op = a6 + b6 * s(L) + c6 * L[0] * L[1]
        else:
            d6 = -64 / 15 + 14 * h2 * k2 / 15 - h2 * h2 * k2 * k2 / 20
            op = d6 + (7 / 15 - h2 * k2 / 90) * s(L) + (1 / 10 + h2 * k2 / 90) * s([L[a] * L[b] for a, b in pairs]) \
                + L[0] * L[1] * L[2] / 30
    for a in range(dim):
        f = _dst(f, a)
    f = f * rhs / op
    for a in range(dim):
        f = _dst(f, a)
    return f


def _rows_2d(coef, n):
    lam = 2.0 * np.cos(math.pi * np.arange(1, n + 1) / (n + 1))
    row = lambda b, a: coef[b][:, None] * lam[None, :] + coef[a][:, None]  # noqa: E731
    return row("bm", "am"), row("b", "a"), row("bp", "ap")


def _rows_3d(coef, n):
    lam = 2.0 * np.cos(math.pi * np.arange(1, n + 1) / (n + 1))
    ly, lx = np.repeat(lam, n), np.tile(lam, n)

    def row(a, b, c, d):
        return (coef[a][:, None] * (lx * ly) + coef[b][:, None] * lx + coef[c][:, None] * ly + coef[d][:, None])

    return row("am", "bm", "cm", "dm"), row("a", "b", "c", "d"), row("ap", "bp", "cp", "dp")


def _thomas(sub, dia, sup, f):
    """Lines along the first axis; f [rows, lines] or [rows, lines, batch]."""
    w = (lambda v: v[..., None]) if f.ndim == 3 else (lambda v: v)
    n = f.shape[0]
    u, y = dia.astype(np.complex128), f.astype(np.complex128)
    for r in range(1, n):
        m = sub[r] / u[r - 1]
        u[r] -= m * sup[r - 1]
        y[r] -= w(m) * y[r - 1]
    y[n - 1] /= w(u[n - 1])
    for r in range(n - 2, -1, -1):
        y[r] = (y[r] - w(sup[r]) * y[r + 1]) / w(u[r])
    return y


def _np_dst(x, dim):
    return _dst(torch.from_numpy(np.ascontiguousarray(x, dtype=np.complex128)), dim).numpy()


def _rhs_2d(n, h, k, k2y_bc, coef, d):
    """The sixth-order right-hand side with its Dirichlet terms."""
    fe, m = d["f_ext"], n + 2
    k2 = k * k
    fy = 3.0 * (fe[2:, 1:-1] - fe[:-2, 1:-1]) / h
    fy[0] -= d["fy_yb"][:n]
    fy[-1] -= d["fy_yb"][n:]
    fy = _pade(fy, 4.0)
    ky = 3.0 * (k2[2:] - k2[:-2]) / h
    ky[0] -= k2y_bc[0]
    ky[-1] -= k2y_bc[1]
    ky = _pade(ky, 4.0)
    ext = {}
    for nm, axis in (("fyy", 0), ("fxx", 1)):
        near = d[nm + ("_yb" if axis == 0 else "_xb")]
        t = fe if axis == 0 else fe.T
        v = 12.0 * (t[2:, 1:-1] - 2.0 * t[1:-1, 1:-1] + t[:-2, 1:-1]) / h / h
        v[0] -= near[1:m - 1]
        v[-1] -= near[m + 1:2 * m - 1]
        v = _pade(v, 10.0)
        e = np.zeros((m, m), dtype=np.complex128)
        e[1:-1, 1:-1] = v if axis == 0 else v.T
        e[0], e[-1] = d[nm + "_yb"][:m], d[nm + "_yb"][m:]
        e[:, 0], e[:, -1] = d[nm + "_xb"][:m], d[nm + "_xb"][m:]
        ext[nm] = e
    fxx, fyy = ext["fxx"], ext["fyy"]
    dx = lambda e: (e[1:-1, :-2] - 2.0 * e[1:-1, 1:-1] + e[1:-1, 2:]) / h / h  # noqa: E731
    dy = lambda e: (e[:-2, 1:-1] - 2.0 * e[1:-1, 1:-1] + e[2:, 1:-1]) / h / h  # noqa: E731
    c = lambda e: e[1:-1, 1:-1]  # noqa: E731
    h2, h4 = h * h, h ** 4
    rhs = h2 * ((1.0 - k2[1:-1, None] * h2 / 20.0) * c(fe) + h2 * (c(fxx) + c(fyy)) / 12.0 + h4 * (dx(fxx) + dy(fyy)) / 360.0
                + h4 * dy(fxx) / 90.0 + h4 * ky[:, None] * fy / 60.0)
    # the Dirichlet ring: the stencil's terms that reach it (corners belong to the edge y = const)
    ring = np.zeros((m, m))
    ring[:, 0], ring[:, -1] = d["u_xb"][:m], d["u_xb"][m:]
    ring[0], ring[-1] = d["u_yb"][:m], d["u_yb"][m:]
    for j0, near, mid in ((0, "bm", "am"), (1, "b", None), (2, "bp", "ap")):
        part = ring[j0:j0 + n]
        rhs -= coef[near][:, None] * (part[:, :-2] + part[:, 2:])
        if mid:
            rhs -= coef[mid][:, None] * part[:, 1:-1]
    return rhs


def _rhs_3d(n, h, k2, coef, kp, d):
    f, m = d["f_ext"], n + 2
    faces = {"fxx": (2, d["fxx_b"].reshape(2, m, m)), "fyy": (1, d["fyy_b"].reshape(2, m, m)),
             "fzz": (0, d["fzz_b"].reshape(2, m, m))}
    ext = {}
    for nm, (axis, b) in faces.items():
        t = np.moveaxis(f, axis, 0)
        v = 12.0 * (t[:-2, 1:-1, 1:-1] - 2.0 * t[1:-1, 1:-1, 1:-1] + t[2:, 1:-1, 1:-1]) / h / h
        v[0] -= b[0][1:-1, 1:-1]
        v[-1] -= b[1][1:-1, 1:-1]
        e = np.zeros((m, m, m), dtype=np.complex128)
        te = np.moveaxis(e, axis, 0)
        te[1:-1, 1:-1, 1:-1] = _pade(v, 10.0)
        te[0], te[-1] = b[0], b[1]
        ext[nm] = e

    def d2(e, axis):
        t = np.moveaxis(e, axis, 0)
        o = [slice(1, -1)] * 2
        return np.moveaxis((t[(slice(0, -2), *o)] - 2.0 * t[(slice(1, -1), *o)] + t[(slice(2, None), *o)]) / h / h, 0, axis)

    c = lambda e: e[1:-1, 1:-1, 1:-1]  # noqa: E731
    fxx, fyy, fzz = ext["fxx"], ext["fyy"], ext["fzz"]
    z = lambda v: v[:, None, None]  # noqa: E731
    rhs = (1.0 - z(k2[1:-1]) * h * h / 20.0) * c(f) + h * h / 12.0 * (c(fxx) + c(fyy) + c(fzz)) \
        + h ** 4 / 360.0 * (d2(fxx, 2) + d2(fyy, 1) + d2(fzz, 0)) + h ** 4 / 90.0 * (d2(fxx, 1) + d2(fxx, 0) + d2(fyy, 0)) \
        + z(kp) * h ** 3 / 120.0 * (f[2:, 1:-1, 1:-1] - f[:-2, 1:-1, 1:-1])
    for l, le, s in ((0, 0, "m"), (n - 1, n + 1, "p")):
        u = d["ue_ext"][le]
        rhs[l] -= coef["a" + s][l] * (u[:-2, :-2] + u[:-2, 2:] + u[2:, :-2] + u[2:, 2:]) \
            + coef["b" + s][l] * (u[1:-1, :-2] + u[1:-1, 2:]) + coef["c" + s][l] * (u[:-2, 1:-1] + u[2:, 1:-1]) \
            + coef["d" + s][l] * u[1:-1, 1:-1]
    return rhs


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind in ("solve", "multi"):
        dim = case.get("dim", 2)
        total = case["batch"] if kind == "solve" else case["plans"] * case["per"]
        f = _sources(dim, n, total, seed, "cuda")
        ks = [complex(case["k"], case["k_im"])] * total if kind == "solve" else \
            [k for k in _multi_k(case, seed) for _ in range(case["per"])]
        for b in range(total):
            f[b] = _spectral(f[b], n, dim, case["order"], ks[b])
        return {"u": f}
    if kind == "general":
        _, _, _, coef, _ = _problem_2d(n, seed)
        f = np.moveaxis(_np_dst(_general_rhs(case, seed, "cuda").cpu().numpy(), 2), 0, 2)
        u = _np_dst(np.moveaxis(_thomas(*_rows_2d(coef, n), f), 2, 0), 2)
        return {"u": torch.from_numpy(np.ascontiguousarray(u))}
    if case["dim"] == 2:
        h, k, k2y_bc, coef, d = _problem_2d(n, seed)
        rhs = _rhs_2d(n, h, k, k2y_bc, coef, d)
        u = _np_dst(_thomas(*_rows_2d(coef, n), _np_dst(rhs, 1)), 1)
    else:
        h, k2, _, coef, kp, d = _problem_3d(n, seed)
        rhs = _rhs_3d(n, h, k2, coef, kp, d)
        t = _np_dst(_np_dst(rhs, 2), 1).reshape(n, n * n)
        u = _np_dst(_np_dst(_thomas(*_rows_3d(coef, n), t).reshape(n, n, n), 1), 2)
    return {"rhs": torch.from_numpy(np.ascontiguousarray(rhs)), "u": torch.from_numpy(np.ascontiguousarray(u))}
