"""The work that users of the method-of-lines framework have it do, as timed cases.

Each case is one call (or one solve) through the public Python API: spectral Crank-Nicolson
diffusion on 2D grids and 3D boxes of powers of two and of other sizes, nonperiodic sine and
cosine solves, adaptive IMEX-Strang Gray-Scott alone and batched, ETDRK4, Newton-Krylov BDF2,
adaptive explicit Runge-Kutta, batched tubular reactors and the fixed-step Gray-Scott methods.
``exact`` gives the same results in 64 bits from plain torch.
"""

import math

import torch

import moljax_gb300 as M
from moljax_gb300.core import reactor

DU, DV = 2e-5, 1e-5          # Gray-Scott diffusivities of the benchmark configurations
L_BOX = 2.5                  # and their box
ATOL, RTOL = 1e-7, 1e-5
DTYPES = {"f32": torch.float32, "f64": torch.float64}


def listed():
    return [
        # FFT-CN on the published 128^2 double-precision grid: 100 small steps, latency counts
        {"name": "cn2d_128_f64", "kind": "cn2d", "ny": 128, "nx": 128, "dtype": "f64", "steps": 100},
        # the same stepper in single precision on a grid whose sides are no powers of two
        {"name": "cn2d_450x600_f32", "kind": "cn2d", "ny": 450, "nx": 600, "dtype": "f32", "steps": 10},
        # 3D FFT-CN, the published 128^3 and 100^3 double-precision boxes, 10 steps each
        {"name": "cn3d_128_f64", "kind": "cn3d", "nz": 128, "ny": 128, "nx": 128, "dtype": "f64", "steps": 10},
        {"name": "cn3d_100_f64", "kind": "cn3d", "nz": 100, "ny": 100, "nx": 100, "dtype": "f64", "steps": 10},
        # one implicit diffusion solve between walls on a few lines: the smallest call
        {"name": "walls_100x64_f64", "kind": "walls", "n": 100, "rows": 64, "bc": "dirichlet", "dtype": "f64"},
        # the headline workload: adaptive IMEX-Strang Gray-Scott at 1024^2 in mixed precision,
        # from its noisy start through the first stretch of the solve
        {"name": "imex_1024_mixed", "kind": "imex", "n": 1024, "precision": "mixed", "t_end": 20.0},
        # uneven Gray-Scott solves in flight together, as a server batches them
        {"name": "batch_8_uneven", "kind": "batch", "count": 8, "t_end": 20.0},
        # ETDRK4 Gray-Scott at 4096^2 in single precision, fields far larger than L2
        {"name": "etdrk4_4096_f32", "kind": "etdrk4", "n": 4096, "dtype": "f32", "steps": 10},
        # implicit nonlinear diffusion: BDF2 by Newton-Krylov at 512^2
        {"name": "nk_bdf2_512", "kind": "nk", "n": 512, "steps": 5},
        # adaptive RK4 advection-diffusion of two species on a ragged grid with walls
        {"name": "rk4_1500x2000_f32", "kind": "rk4", "ny": 1500, "nx": 2000, "dtype": "f32", "bc": "neumann",
         "attempts": 10},
        # tubular reactor requests of uneven lengths (n log-uniform in 64..4096) in one launch
        {"name": "reactor_48_f32", "kind": "reactor", "count": 48, "dtype": "f32"},
        # the fixed-step Strang method of the 256^2 double-precision Gray-Scott comparison
        {"name": "strang_256_f64", "kind": "strang", "n": 256, "dtype": "f64", "steps": 100},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cn2d", "cn2d", "cn3d", "cn3d", "walls", "imex", "batch", "etdrk4", "nk", "rk4", "reactor",
                       "strang"])
    dtype = rng.choice(["f32", "f64"])
    if kind == "cn2d":
        if rng.random() < 0.4:
            ny, nx = 2 ** rng.randint(5, 11), 2 ** rng.randint(5, 11)
        else:
            ny, nx = _log_int(rng, 24, 1600), _log_int(rng, 24, 1600)
        return {"kind": kind, "ny": ny, "nx": nx, "dtype": dtype, "steps": min(100, max(1, 3_000_000 // (ny * nx)))}
    if kind == "cn3d":
        top = 256 if dtype == "f32" else 128
        if rng.random() < 0.4:
            nz, ny, nx = (2 ** rng.randint(4, int(math.log2(top))) for _ in range(3))
        else:
            nz, ny, nx = (_log_int(rng, 16, top) for _ in range(3))
        return {"kind": kind, "nz": nz, "ny": ny, "nx": nx, "dtype": dtype,
                "steps": min(10, max(1, 16_000_000 // (nz * ny * nx)))}
    if kind == "walls":
        return {"kind": kind, "n": _log_int(rng, 16, 1000), "rows": _log_int(rng, 16, 4096),
                "bc": rng.choice(["dirichlet", "neumann"]), "dtype": dtype}
    if kind == "imex":
        precision = rng.choice(["mixed", "mixed", "fp32", "fp64"])
        return {"kind": kind, "n": 2 ** rng.randint(6, 9 if precision == "fp64" else 10), "precision": precision,
                "t_end": round(rng.uniform(4.0, 12.0 if precision == "fp64" else 20.0), 2)}
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 2, 10), "t_end": round(rng.uniform(5.0, 20.0), 2)}
    if kind == "etdrk4":
        n = 2 ** rng.randint(7, 12 if dtype == "f32" else 9)
        return {"kind": kind, "n": n, "dtype": dtype, "steps": rng.randint(4, 10)}
    if kind == "nk":
        return {"kind": kind, "n": 2 ** rng.randint(5, 9), "steps": rng.randint(2, 5)}
    if kind == "rk4":
        top = 2500 if dtype == "f32" else 600
        return {"kind": kind, "ny": _log_int(rng, 64, top), "nx": _log_int(rng, 64, top), "dtype": dtype,
                "bc": rng.choice(["periodic", "dirichlet", "neumann"]), "attempts": rng.randint(4, 10)}
    if kind == "reactor":
        return {"kind": kind, "count": _log_int(rng, 4, 64 if dtype == "f32" else 24), "dtype": dtype}
    return {"kind": kind, "n": 2 ** rng.randint(6, 9 if dtype == "f32" else 8), "dtype": dtype,
            "steps": rng.randint(20, 100)}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _smooth(shape, seed, dtype):
    """A few random low modes plus 5 % noise on a periodic box."""
    g = _gen(seed)
    u = 0.05 * torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)
    grids = torch.meshgrid(*[torch.arange(n, device="cuda", dtype=torch.float64) / n for n in shape], indexing="ij")
    for _ in range(4):
        k = torch.randint(1, 4, (len(shape),), generator=g, device="cuda")
        ph = 2 * math.pi * torch.rand(len(shape), generator=g, device="cuda", dtype=torch.float64)
        term = torch.ones((), device="cuda", dtype=torch.float64)
        for d in range(len(shape)):
            term = term * torch.sin(2 * math.pi * k[d] * grids[d] + ph[d])
        u = u + term
    return u.to(dtype).contiguous()


def _gray_scott_state(n, seed, dtype):
    """Padded (u, v): 1 and 0, a central square of (0.5, 0.25), 1 % uniform noise."""
    g = _gen(seed)
    x = (torch.arange(n + 2, device="cuda", dtype=torch.float64) - 0.5) / n - 0.5
    sq = (x.abs()[:, None] < 0.1) & (x.abs()[None, :] < 0.1)
    out = {}
    for name, base, core in (("u", 1.0, 0.5), ("v", 0.0, 0.25)):
        f = torch.where(sq, torch.full_like(sq, core, dtype=torch.float64),
                        torch.full_like(sq, base, dtype=torch.float64))
        f = f + 0.01 * (2 * torch.rand(f.shape, generator=g, device="cuda", dtype=torch.float64) - 1)
        out[name] = f.to(dtype).contiguous()
    return out


def _gaussians(n, seed):
    g = _gen(seed)
    x = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n
    u = torch.zeros((n, n), device="cuda", dtype=torch.float64)
    for _ in range(8):
        a, w, cx, cy = torch.rand(4, generator=g, device="cuda", dtype=torch.float64)
        w = 0.02 + 0.08 * w
        u += a * torch.exp(-((x[None, :] - cx) ** 2 + (x[:, None] - cy) ** 2) / (2 * w * w))
    return u


def _uniform(seed, count, lo, hi):
    g = torch.Generator().manual_seed(int(seed))
    return [lo + (hi - lo) * float(t) for t in torch.rand(count, generator=g, dtype=torch.float64)]


def _batch_parameters(case, seed):
    sizes = [(64, 128, 256, 512)[i % 4] for i in range(case["count"])]
    return list(zip(sizes, _uniform(seed, len(sizes), 0.02, 0.06), _uniform(seed + 1, len(sizes), 0.05, 0.07)))


def _reactor_parameters(case, seed):
    """(n, Pe, Da, dt, steps): lengths spread over 64..4096, Pe in [10, 200], Da in [0.5, 5]."""
    c = case["count"]
    jitter, pe, da = _uniform(c, c, 0.0, 1.0), _uniform(seed, c, 10.0, 200.0), _uniform(seed + 1, c, 0.5, 5.0)
    out = []
    for i in range(c):
        n = int(round(64 * 64.0 ** ((i + 0.8 * jitter[i] + 0.2) / c)))
        out.append((n, pe[i], da[i]) + tuple(reactor.served_dt(n)))
    return out


def _rk4_setup(case):
    grid = M.Grid2D(case["nx"], case["ny"], 0.0, 1.0, 0.0, 1.0)
    dt = 0.2 * min(grid.min_dx / 0.8, grid.min_dx2 / 4e-4)
    return grid, dt


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "cn2d":
        s["u"] = _smooth((case["ny"], case["nx"]), seed, DTYPES[case["dtype"]])
    elif kind == "cn3d":
        s["u"] = _smooth((case["nz"], case["ny"], case["nx"]), seed, DTYPES[case["dtype"]])
    elif kind == "walls":
        dt = DTYPES[case["dtype"]]
        s["f"] = torch.randn((case["rows"], case["n"]), generator=_gen(seed), device="cuda",
                             dtype=torch.float64).to(dt)
        symbol = {"dirichlet": M.laplacian_symbol_dirichlet, "neumann": M.laplacian_symbol_neumann}[case["bc"]]
        s["lam"] = symbol(case["n"], 1.0 / (case["n"] + 1), dt, "cuda")
    elif kind == "imex":
        dt = torch.float64 if case["precision"] == "fp64" else torch.float32
        grid = M.Grid2D(case["n"], case["n"], 0.0, L_BOX, 0.0, L_BOX)
        s["model"], s["cache"], s["diff"] = M.create_gray_scott_periodic_fft(grid, DU, DV, 0.035, 0.065, dt, "cuda")
        s["y0"] = _gray_scott_state(case["n"], seed, dt)
        s["pid"] = M.PIDParams(atol=ATOL, rtol=RTOL)
    elif kind == "batch":
        s["problems"] = []
        for i, (n, F, k) in enumerate(_batch_parameters(case, seed)):
            grid = M.Grid2D(n, n, 0.0, L_BOX, 0.0, L_BOX)
            s["problems"].append(M.GrayScottProblem(grid, DU, DV, F, k, _gray_scott_state(n, seed + i, torch.float32),
                                                    0.0, case["t_end"], 1.0, pid=M.PIDParams(atol=ATOL, rtol=RTOL),
                                                    max_steps=20000, save_every=100))
    elif kind == "etdrk4":
        dt = DTYPES[case["dtype"]]
        grid = M.Grid2D(case["n"], case["n"], 0.0, L_BOX, 0.0, L_BOX)
        s["model"] = M.create_gray_scott_model(grid, DU, DV, 0.035, 0.065, dtype=dt)
        s["y0"] = _gray_scott_state(case["n"], seed, dt)
    elif kind == "nk":
        s["u"] = _gaussians(case["n"], seed)
        s["nk"] = M.NKParams(gmres_restart=30)
    elif kind == "rk4":
        grid, _ = _rk4_setup(case)
        bc = {"periodic": M.BCType.PERIODIC, "dirichlet": M.BCType.DIRICHLET, "neumann": M.BCType.NEUMANN}[case["bc"]]
        s["model"] = M.create_advection_diffusion_model(grid, ("c1", "c2"), 1e-4, 0.5, -0.3, bc,
                                                        dtype=DTYPES[case["dtype"]])
        s["y0"] = {}
        for i, name in enumerate(("c1", "c2")):
            f = torch.zeros((case["ny"] + 2, case["nx"] + 2), device="cuda", dtype=DTYPES[case["dtype"]])
            f[1:-1, 1:-1] = _smooth((case["ny"], case["nx"]), 2 * seed + i, f.dtype)
            s["y0"][name] = f
        s["pid"] = M.PIDParams(atol=ATOL, rtol=RTOL)
    elif kind == "reactor":
        s["cases"] = [reactor.ReactorCase(n, Pe, Da, dt, steps, reactor.DANCKWERTS_CN, 0.0)
                      for n, Pe, Da, dt, steps in _reactor_parameters(case, seed)]
    elif kind == "strang":
        y = _gray_scott_state(case["n"], seed, DTYPES[case["dtype"]])
        s["u"], s["v"] = (y[k][1:-1, 1:-1].contiguous() for k in ("u", "v"))
    else:
        raise ValueError(kind)
    return s


# ------------------------------------------------------------------ the calls
def _adaptive_outputs(r, names):
    # the state and what the driver says of the run; the log of step sizes stays behind, whose
    # last digits follow the single-precision error estimate of each attempt
    return {"y": {n: r.y_final[n] for n in names}, "t": float(r.t_final), "accepted": int(r.n_accepted),
            "rejected": int(r.n_rejected), "status": int(r.status)}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "cn2d":
        return M.fft_cn_step(s["u"], 0.1, 1.0 / case["nx"], 1e-3, case["steps"], dy=1.0 / case["ny"])
    if kind == "cn3d":
        return M.fft_cn_step_3d(s["u"], 0.1, 1.0 / case["nx"], 1e-3, case["steps"], dy=1.0 / case["ny"],
                                dz=1.0 / case["nz"])
    if kind == "walls":
        solve = {"dirichlet": M.solve_helmholtz_dirichlet, "neumann": M.solve_helmholtz_neumann}[case["bc"]]
        return solve(s["f"], s["lam"], 1e-3, 0.1)
    if kind == "imex":
        r = M.adaptive_integrate_imex(s["model"], s["y0"], 0.0, case["t_end"], 1.0, s["cache"], s["diff"],
                                      max_steps=20000, pid_params=s["pid"], save_every=100, save_y_history=False,
                                      precision=case["precision"])
        return _adaptive_outputs(r, ("u", "v"))
    if kind == "batch":
        return [_adaptive_outputs(r, ("u", "v")) for _, r in M.adaptive_integrate_imex_batch(s["problems"])]
    if kind == "etdrk4":
        return M.etdrk4_gray_scott(s["model"], s["y0"], 1.0, case["steps"])
    if kind == "nk":
        dx = 1.0 / case["n"]
        u, _ = M.integrate_implicit_vardiff(s["u"], dx, 100 * dx * dx, case["steps"], "bdf2", nk_params=s["nk"],
                                            be_guess="previous")
        return u
    if kind == "rk4":
        _, dt = _rk4_setup(case)
        r = M.adaptive_integrate(s["model"], s["y0"], 0.0, case["attempts"] * dt, dt, M.IntegratorType.RK4,
                                 max_steps=1000, pid_params=s["pid"], save_y_history=False)
        return _adaptive_outputs(r, ("c1", "c2"))
    if kind == "reactor":
        return reactor.solve_batch(s["cases"], DTYPES[case["dtype"]])
    return M.gray_scott_strang_exp(s["u"], s["v"], DU, DV, 0.035, 0.065, 0.5, case["steps"], 1.0 / case["n"])


# ------------------------------------------------------------------ what a pass cannot do without
def _pair_flops(points):
    """A real forward and inverse transform of so many points."""
    return 5.0 * points * math.log2(max(points, 2))


def work(case):
    """Each input and output once; operations: the transforms, stencils and pointwise work of
    every step (an adaptive Gray-Scott pass by about 200 attempts while the noise of its start
    fades, then 0.45 of time each)."""
    kind = case["kind"]
    size = {"f32": 4, "f64": 8}.get(case.get("dtype"), 4)
    if kind in ("cn2d", "cn3d"):
        n = case.get("nz", 1) * case["ny"] * case["nx"]
        return {"bytes": 2 * size * n, "flops": case["steps"] * (_pair_flops(n) + 4 * n)}
    if kind == "walls":
        n = case["n"] * case["rows"]
        return {"bytes": size * (2 * n + case["n"]), "flops": n * (10 * math.log2(max(case["n"], 2)) + 4)}
    if kind == "imex":
        size = 8 if case["precision"] == "fp64" else 4
        n = case["n"] ** 2
        attempts = 200 + case["t_end"] / 0.45
        return {"bytes": 4 * size * n, "flops": attempts * 2 * n * (6 * 5.0 * math.log2(n) + 60)}
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for n, _, _ in _batch_parameters(case, 0):
            w = work({"kind": "imex", "n": n, "precision": "mixed", "t_end": case["t_end"]})
            total = {k: total[k] + w[k] for k in total}
        return total
    if kind == "etdrk4":
        n = case["n"] ** 2
        return {"bytes": 4 * size * n, "flops": case["steps"] * 2 * n * (4 * 5.0 * math.log2(n) + 60)}
    if kind == "nk":
        n = case["n"] ** 2  # about three Newton and eleven Krylov iterations a step
        return {"bytes": 16 * n, "flops": case["steps"] * n * (6 * 60 + 11 * (10 * math.log2(n) + 80))}
    if kind == "rk4":
        n = case["ny"] * case["nx"]
        return {"bytes": 4 * size * n, "flops": case["attempts"] * 2 * n * 12 * 25}
    if kind == "reactor":
        p = _reactor_parameters(case, 0)
        return {"bytes": size * sum(q[0] for q in p), "flops": sum(14.0 * q[0] * q[4] for q in p)}
    n = case["n"] ** 2
    return {"bytes": 4 * size * n, "flops": case["steps"] * 2 * (_pair_flops(n) + 20 * n)}


# ------------------------------------------------------------------ the same in 64 bits
def _k(n, d):
    return 2 * math.pi * torch.fft.fftfreq(n, d=d, device="cuda", dtype=torch.float64)


def _fd(n, d):
    m = torch.arange(n, device="cuda", dtype=torch.float64)
    return (2 * torch.cos(2 * math.pi * m / n) - 2) / (d * d)


def _half(lam):
    return lam[..., : lam.shape[-1] // 2 + 1]


def _real_pair(u, m):
    """real(ifftn(m fftn(u))) with m given on the half spectrum."""
    dims = tuple(range(u.dim() - m.dim(), u.dim()))
    return torch.fft.irfftn(m * torch.fft.rfftn(u, dim=dims), s=[u.shape[d] for d in dims], dim=dims)


def _pad(u, bc="periodic"):
    u = torch.cat([u[..., -1:], u, u[..., :1]], -1) if bc == "periodic" else torch.cat(
        [u[..., :1], u, u[..., -1:]], -1) if bc == "neumann" else torch.cat([-u[..., :1], u, -u[..., -1:]], -1)
    v = u.transpose(-1, -2)
    v = torch.cat([v[..., -1:], v, v[..., :1]], -1) if bc == "periodic" else torch.cat(
        [v[..., :1], v, v[..., -1:]], -1) if bc == "neumann" else torch.cat([-v[..., :1], v, -v[..., -1:]], -1)
    return v.transpose(-1, -2).contiguous()


def _adaptive(step, y, t_end, dt0, dt_cfl, order):
    """Step doubling with the PI controller: (y, t, accepted, rejected)."""
    safety, kI, kP = 0.9, 0.7 / order, 0.4 / order
    t, dt, prev, acc, rej = 0.0, min(dt0, dt_cfl), 1.0, 0, 0
    while t < t_end:
        h = min(dt, t_end - t)
        half = step(step(y, 0.5 * h), 0.5 * h)
        err = half - step(y, h)
        e = max(float(((err / (ATOL + RTOL * half.abs())) ** 2).mean().sqrt()), 1e-10)
        if e <= 1.0:
            fac = (1.0 / e) ** kI * (max(prev, 1e-10) / e) ** kP
            fac = min(max(safety * fac, 0.2), 5.0)
        else:
            fac = min(max(safety * (1.0 / e) ** kI, 0.2), 1.0)
        new = min(max(min(min(max(h * fac, 1e-12), 1.0), dt_cfl), 1e-12), 1.0)
        if e <= 1.0:
            t, y, dt, prev, acc = t + h, half, new, e, acc + 1
        else:
            dt, rej = max(0.5 * new, 1e-12), rej + 1
    return y, t, acc, rej


def _gs_rates(y, F, k):
    uvv = y[0] * y[1] * y[1]
    return torch.stack([-uvv + F * (1 - y[0]), uvv - (F + k) * y[1]])


def _exact_imex(y0, n, F, k, t_end):
    y = torch.stack([y0[c][1:-1, 1:-1].double() for c in ("u", "v")])
    lam = _half(_fd(n, L_BOX / n)[:, None] + _fd(n, L_BOX / n)[None, :])
    D = torch.tensor([DU, DV], device="cuda", dtype=torch.float64)[:, None, None]

    def diffuse(x, h):
        m = 1.0 / (1.0 - h * D * lam)
        return torch.fft.irfft2(m * torch.fft.rfft2(x), s=(n, n))

    def step(x, h):
        x = diffuse(x, 0.5 * h)
        r = _gs_rates(x, F, k)
        x = x + 0.5 * h * (r + _gs_rates(x + h * r, F, k))
        return diffuse(x, 0.5 * h)

    dt_cfl = min(max(0.9 * min(1.0, 0.5 / (F + k)), 1e-12), 1.0)
    y, t, acc, rej = _adaptive(step, y, t_end, 1.0, dt_cfl, 2)
    y = _pad(y)
    return {"y": {"u": y[0], "v": y[1]}, "t": t, "accepted": None, "rejected": None, "status": None}


def _exact_etdrk4(case, seed):
    n, dt, F, k = case["n"], 1.0, 0.035, 0.065
    y0 = _gray_scott_state(n, seed, DTYPES[case["dtype"]])
    lam = _half(_fd(n, L_BOX / n)[:, None] + _fd(n, L_BOX / n)[None, :])
    tabs = []
    for D in (DU, DV):
        z = dt * D * lam
        Q, f1, f2, f3 = (torch.zeros_like(z) for _ in range(4))
        for j in range(32):
            a = math.pi * (j + 0.5) / 32
            w = z + complex(math.cos(a), math.sin(a))
            ew, w3 = torch.exp(w), w ** 3
            Q += ((torch.exp(0.5 * w) - 1) / w).real
            f1 += ((-4 - w + ew * (4 - 3 * w + w * w)) / w3).real
            f2 += ((2 + w + ew * (w - 2)) / w3).real
            f3 += ((-4 - 3 * w - w * w + ew * (4 - w)) / w3).real
        c = dt / 32
        tabs.append((torch.exp(z), torch.exp(0.5 * z), c * Q, c * f1, 2 * c * f2, c * f3))
    E, E2, Q, f1, f2, f3 = (torch.stack([tabs[0][i], tabs[1][i]]) for i in range(6))
    y = torch.stack([y0[c][1:-1, 1:-1].double() for c in ("u", "v")])

    def N(h):
        return torch.fft.rfft2(_gs_rates(torch.fft.irfft2(h, s=(n, n)), F, k))

    h = torch.fft.rfft2(y)
    for _ in range(case["steps"]):
        n0 = N(h)
        a = E2 * h + Q * n0
        na = N(a)
        nb = N(E2 * h + Q * na)
        nc = N(E2 * a + Q * (2 * nb - n0))
        h = E * h + f1 * n0 + f2 * (na + nb) + f3 * nc
    y = _pad(torch.fft.irfft2(h, s=(n, n)))
    return {"u": y[0], "v": y[1]}


def _exact_nk(case, seed):
    n = case["n"]
    dx = 1.0 / n
    dt = 100 * dx * dx
    lam = _half(_fd(2 * n, dx)[:, None] + _fd(2 * n, dx)[None, :])

    def F(u):
        p = _pad(u, "dirichlet")
        D = 1 + p * p
        c, cd = p[1:-1, 1:-1], D[1:-1, 1:-1]
        out = -c ** 3
        for q, qd in ((p[1:-1, 2:], D[1:-1, 2:]), (p[1:-1, :-2], D[1:-1, :-2]), (p[2:, 1:-1], D[2:, 1:-1]),
                      (p[:-2, 1:-1], D[:-2, 1:-1])):
            out = out + 0.5 * (cd + qd) * (q - c) / (dx * dx)
        return out

    def inverse(r, a0, kappa):  # (a0 - kappa Lap)^-1 between walls by the odd extension
        e = torch.cat([torch.cat([r, -r.flip(1)], 1), torch.cat([-r.flip(0), r.flip(0).flip(1)], 1)], 0)
        return _real_pair(e, 1.0 / (a0 - kappa * lam))[:n, :n]

    def gmres(A, b, P):
        r = P(b)
        beta = float(r.norm())
        V, H = [r / beta], torch.zeros(41, 40, dtype=torch.float64)
        for j in range(40):
            w = P(A(V[j]))
            for _ in range(2):
                c = torch.stack([(v * w).sum() for v in V])
                for i, v in enumerate(V):
                    w = w - c[i] * v
                H[: j + 1, j] += c.cpu()
            H[j + 1, j] = float(w.norm())
            e1 = torch.zeros(j + 2, 1, dtype=torch.float64)
            e1[0] = beta
            y = torch.linalg.lstsq(H[: j + 2, : j + 1], e1).solution
            if float((H[: j + 2, : j + 1] @ y - e1).norm()) < 1e-11 * beta or float(H[j + 1, j]) == 0:
                break
            V.append(w / H[j + 1, j])
        return sum(float(y[i]) * V[i] for i in range(y.shape[0]))

    old = u = _gaussians(n, seed)
    for s in range(case["steps"]):
        a0, a1, a2, beta = (1.0, -1.0, 0.0, dt) if s == 0 else (1.5, -2.0, 0.5, dt * 2 / 3)
        cst, kappa = a1 * u + a2 * old, beta * (1 + float((u * u).mean()))
        x = u.clone() if s == 0 else 2 * u - old
        R = lambda z: a0 * z + cst - beta * F(z)  # noqa: E731
        for _ in range(8):
            r = R(x)
            if float(r.norm()) < 1e-13 * float(x.norm()):
                break
            x = x + gmres(lambda v: torch.func.jvp(R, (x,), (v,))[1], -r, lambda v: inverse(v, a0, kappa))
        old, u = u, x
    return u


def _exact_rk4(case, seed):
    s = prepare(case, seed)
    bc, D, vx, vy = case["bc"], 1e-4, 0.5, -0.3
    dx, dy = 1.0 / case["nx"], 1.0 / case["ny"]

    def f(y):
        p = _pad(y, bc)
        c, e, w, n, o = p[:, 1:-1, 1:-1], p[:, 1:-1, 2:], p[:, 1:-1, :-2], p[:, 2:, 1:-1], p[:, :-2, 1:-1]
        return (D * ((e - 2 * c + w) / (dx * dx) + (n - 2 * c + o) / (dy * dy)) - vx * (c - w) / dx
                - vy * (n - c) / dy)

    def step(y, h):
        k1 = f(y)
        k2 = f(y + 0.5 * h * k1)
        k3 = f(y + 0.5 * h * k2)
        return y + h / 6 * (k1 + 2 * k2 + 2 * k3 + f(y + h * k3))

    y = torch.stack([s["y0"][c][1:-1, 1:-1].double() for c in ("c1", "c2")])
    _, dt = _rk4_setup(case)
    d = min(dx, dy)
    dt_cfl = 0.9 * min(1.0, 0.5 * d / (abs(vx) + abs(vy)), 0.25 * d * d / D)
    y, t, acc, rej = _adaptive(step, y, case["attempts"] * dt, dt, dt_cfl, 4)
    y = _pad(y, bc)
    return {"y": {"c1": y[0], "c2": y[1]}, "t": t, "accepted": None, "rejected": None, "status": None}


def _exact_reactor(case, seed):
    out = []
    for n, Pe, Da, dt, steps in _reactor_parameters(case, seed):
        dz = 1.0 / n
        op = torch.zeros((n, n), device="cuda", dtype=torch.float64)
        i = torch.arange(n, device="cuda")
        op[i, i] = -2.0 / (Pe * dz * dz) - 1.0 / dz - Da
        op[i[1:], i[:-1]] = 1.0 / (Pe * dz * dz) + 1.0 / dz
        op[i[:-1], i[1:]] = 1.0 / (Pe * dz * dz)
        op[-1, -2] = 2.0 / (Pe * dz * dz) + 1.0 / dz
        one = torch.eye(n, device="cuda", dtype=torch.float64)
        inv = torch.linalg.inv(one - 0.5 * dt * op)
        step = inv @ (one + 0.5 * dt * op)
        add = inv[:, 0] * (dt / dz)
        c = torch.zeros(n, device="cuda", dtype=torch.float64)
        for _ in range(steps):
            c = torch.addmv(add, step, c)
        out.append(c)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "cn2d":
        ny, nx = case["ny"], case["nx"]
        u = _smooth((ny, nx), seed, DTYPES[case["dtype"]]).double()
        x = 0.5e-3 * 0.1 * _half(-(_k(ny, 1.0 / ny)[:, None] ** 2 + _k(nx, 1.0 / nx)[None, :] ** 2))
        for _ in range(case["steps"]):
            u = _real_pair(u, (1 + x) / (1 - x))
        return u
    if kind == "cn3d":
        nz, ny, nx = case["nz"], case["ny"], case["nx"]
        u = _smooth((nz, ny, nx), seed, DTYPES[case["dtype"]]).double()
        x = 0.5e-3 * 0.1 * _half(-(_k(nz, 1.0 / nz)[:, None, None] ** 2 + _k(ny, 1.0 / ny)[:, None] ** 2
                                   + _k(nx, 1.0 / nx) ** 2))
        for _ in range(case["steps"]):
            u = _real_pair(u, (1 + x) / (1 - x))
        return u
    if kind == "walls":
        s, n = prepare(case, seed), case["n"]
        m = torch.arange(n, device="cuda", dtype=torch.float64)
        d = n + 1.0
        if case["bc"] == "dirichlet":
            q = math.sqrt(2.0 / (n + 1)) * torch.sin(math.pi * (m[:, None] + 1) * (m[None, :] + 1) / (n + 1))
            lam = -4 * d * d * torch.sin(math.pi * (m + 1) / (2 * (n + 1))) ** 2
        else:
            q = math.sqrt(2.0 / n) * torch.cos(math.pi * m[:, None] * (m[None, :] + 0.5) / n)
            q[0] /= math.sqrt(2.0)
            lam = -4 * d * d * torch.sin(math.pi * m / (2 * n)) ** 2
        return ((s["f"].double() @ q.T) / (1 - 1e-4 * lam)) @ q
    if kind == "imex":
        y0 = _gray_scott_state(case["n"], seed, torch.float64 if case["precision"] == "fp64" else torch.float32)
        return _exact_imex(y0, case["n"], 0.035, 0.065, case["t_end"])
    if kind == "batch":
        out = []
        for i, (n, F, k) in enumerate(_batch_parameters(case, seed)):
            r = _exact_imex(_gray_scott_state(n, seed + i, torch.float32), n, F, k, case["t_end"])
            r["y"] = {c: f[1:-1, 1:-1].contiguous() for c, f in r["y"].items()}
            out.append(r)
        return out
    if kind == "etdrk4":
        return _exact_etdrk4(case, seed)
    if kind == "nk":
        return _exact_nk(case, seed)
    if kind == "rk4":
        return _exact_rk4(case, seed)
    if kind == "reactor":
        return _exact_reactor(case, seed)
    n, F, k, dt = case["n"], 0.035, 0.065, 0.5
    y0 = _gray_scott_state(n, seed, DTYPES[case["dtype"]])
    y = torch.stack([y0[c][1:-1, 1:-1].double() for c in ("u", "v")])
    lam = _half(-(_k(n, 1.0 / n)[:, None] ** 2 + _k(n, 1.0 / n)[None, :] ** 2))
    m = torch.exp(dt * lam * torch.tensor([DU, DV], device="cuda", dtype=torch.float64)[:, None, None])
    for _ in range(case["steps"]):
        y = y + 0.5 * dt * _gs_rates(y, F, k)
        y = torch.fft.irfft2(m * torch.fft.rfft2(y), s=(n, n))
        y = y + 0.5 * dt * _gs_rates(y, F, k)
    return y[0], y[1]
