"""Spectral passes on the GPU vs the NumPy FP64 oracle."""

import numpy as np
import pytest
import torch

from oracle import fftcn, mol

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("ny,nx", [(2, 2), (4, 8), (16, 16), (32, 64), (128, 128), (256, 32),
                                   (64, 1024), (512, 512), (4096, 16), (16, 4096)])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_helmholtz_vs_oracle(cuda, ny, nx, dtype):
    from moljax_gb300.core import fft_solvers
    rng = np.random.default_rng(ny * 7 + nx)
    dy, dx = 2.5 / ny, 2.5 / nx
    rhs = rng.standard_normal((3, ny, nx))
    D = [2e-5, 1e-5, 0.3]
    plan = fft_solvers.get_plan(ny, nx, dy, dx, "fd", dtype, cuda)
    out = plan.apply(torch.tensor(rhs, dtype=dtype, device=cuda), D, 0.7, 1).cpu().numpy()
    lam = mol.fd_symbol_2d(ny, nx, dy, dx)
    tol = 1e-13 if dtype == torch.float64 else 3e-6
    for f in range(3):
        ref = mol.solve_helmholtz_2d(rhs[f], lam, 0.7, D[f])
        assert _rel(out[f], ref) < tol


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_roundtrip_identity(cuda, dtype):
    from moljax_gb300.core import fft_solvers
    rng = np.random.default_rng(5)
    x = rng.standard_normal((2, 256, 128))
    plan = fft_solvers.get_plan(256, 128, 0.1, 0.1, "fd", dtype, cuda)
    out = plan.apply(torch.tensor(x, dtype=dtype, device=cuda), [1.0, 1.0], 0.0, 0).cpu().numpy()
    tol = 1e-14 if dtype == torch.float64 else 1e-6
    assert _rel(out, x) < tol


def test_zero_diffusivity_passes_through(cuda):
    # fft_solvers.py:435-443 / tests/test_fft_solver.py:253-279
    from moljax_gb300.core import fft_solvers
    x = torch.randn(2, 32, 32, dtype=torch.float64, device=cuda)
    plan = fft_solvers.get_plan(32, 32, 0.1, 0.1, "fd", torch.float64, cuda)
    out = plan.apply(x, [0.0, 0.5], 0.1, 1)
    assert torch.equal(out[0], x[0])
    assert not torch.equal(out[1], x[1])


def test_fft_cn_config1_fp64(cuda):
    # 128^2 on [0,1)^2, D=0.1, dt=0.01, 100 steps one by one; spectral symbol
    from moljax_gb300.core import fft_solvers
    u0 = fftcn.node_grid_ic(128)
    u = fft_solvers.fft_cn_step(torch.tensor(u0, device=cuda), 0.1, 1 / 128, 0.01, n_steps=100)
    u = u.cpu().numpy()
    ref = fftcn.fft_cn_2d(u0, 0.1, 1 / 128, 0.01, 100)
    assert _rel(u, ref) < 1e-12
    ana = fftcn.analytic_decay(u0, 0.1, 1.0)
    assert _rel(u, ana) < 5e-3  # CN truncation (4.10e-3)


def test_fft_cn_published_table(cuda):
    # benchmarks/results/precision_fp32_fp64.json, FP64 rows, through the GPU path
    import json, os
    from moljax_gb300.core import fft_solvers
    g = json.load(open(os.path.join(os.path.dirname(__file__), "golden", "fftcn_published.json")))
    u0 = fftcn.node_grid_ic(128)
    D, T = g["precision_table"]["D"], g["precision_table"]["t_final"]
    for row in g["precision_table"]["fp64"][:4]:
        n = row["n_steps"]
        u = fft_solvers.fft_cn_step(torch.tensor(u0, device=cuda), D, 1 / 128, row["dt"], n)
        err = np.max(np.abs(u.cpu().numpy() - fftcn.analytic_decay(u0, D, n * row["dt"])))
        assert err == pytest.approx(row["error"], rel=1e-6)


def test_fft_cn_fd_symbol(cuda):
    from moljax_gb300.core import fft_solvers
    u0 = fftcn.node_grid_ic(64)
    u = fft_solvers.fft_cn_step(torch.tensor(u0, device=cuda), 0.1, 1 / 64, 0.01, 10, symbol="fd")
    ref = fftcn.fft_cn_2d(u0, 0.1, 1 / 64, 0.01, 10, kind="fd")
    assert _rel(u.cpu().numpy(), ref) < 1e-12


def test_solver_comparison_1d_published(cuda):
    """benchmarks/results/solver_comparison.json through the native 1D advection-diffusion
    path (N = 1024, D = 0.01, v = 1, t = 10, FP64): FFT-CN (dt 1e-3, 10 000 steps) and the
    exponential Strang IMEX (dt 5e-3, 2 000 steps) reproduce the published max differences
    from SciPy Radau (tests/golden/radau_advdiff1d.npy) and the oracle's final states."""
    import json
    import os
    import moljax_gb300 as M
    gold = os.path.join(os.path.dirname(__file__), "golden")
    g = json.load(open(os.path.join(gold, "solver_comparison_published.json")))
    ref = np.load(os.path.join(gold, "radau_advdiff1d.npy"))
    cfg = g["config"]
    n, D, v, T = cfg["N"], cfg["D"], cfg["v"], cfg["t_final"]
    u0 = fftcn.solver_comparison_ic(n)
    cn, im = g["solvers"][1], g["solvers"][2]
    ut = torch.tensor(u0, device=cuda)
    u = M.fft_cn_advdiff_1d(ut, D, v, 1.0 / n, cn["dt"], cn["steps"]).cpu().numpy()
    assert float(np.max(np.abs(u - ref))) == pytest.approx(cn["error_vs_scipy"], rel=1e-5)
    o = fftcn.fft_cn_1d(u0, D, 1.0 / n, cn["dt"], cn["steps"], "spectral", v=v)
    assert float(np.max(np.abs(u - o))) < 1e-12
    u = M.imex_advdiff_1d(ut, D, v, 1.0 / n, im["dt"], im["steps"]).cpu().numpy()
    assert float(np.max(np.abs(u - ref))) == pytest.approx(im["error_vs_scipy"], rel=1e-5)
    o = fftcn.strang_exp_1d(u0, D, v, 1.0 / n, im["dt"], im["steps"])
    assert float(np.max(np.abs(u - o))) < 1e-12
    # a length that is not a power of two takes the general path with the same results
    m = 768
    w0 = fftcn.solver_comparison_ic(m)
    w = M.fft_cn_advdiff_1d(torch.tensor(w0, device=cuda), D, v, 1.0 / m, 1e-3, 200).cpu().numpy()
    assert float(np.max(np.abs(w - fftcn.fft_cn_1d(w0, D, 1.0 / m, 1e-3, 200, "spectral", v=v)))) < 1e-12
    w = M.imex_advdiff_1d(torch.tensor(w0, device=cuda), D, v, 1.0 / m, 5e-3, 100).cpu().numpy()
    assert float(np.max(np.abs(w - fftcn.strang_exp_1d(w0, D, v, 1.0 / m, 5e-3, 100)))) < 1e-12


@pytest.mark.parametrize("shape", [(2, 2), (2, 16), (4, 8), (16, 2), (64, 64), (128, 256), (1024, 4), (2048, 16), (8, 2048),
                                   (4096, 4), (2, 4096)])
def test_fp64_passes_at_tile_edges(cuda, shape):
    """The FP64 row and column passes at the edges of their tiles (one to 32 sequences, radix 2, 4
    and 8, single sequences of 2048, and 4096 on the FP32-style passes), one step against several
    in a row (fused rows, tabulated multipliers), with a workspace that holds only the spectra, and
    two-output column passes (an IMEX attempt), against NumPy FFTs."""
    import ctypes as C
    from moljax_gb300 import _native as N
    from moljax_gb300.core.fft_solvers import get_plan
    ny, nx = shape
    rng = np.random.default_rng(ny + 3 * nx)
    u = rng.standard_normal((ny, nx))
    dy, dx, D, dt = 1.0 / ny, 1.0 / nx, 0.1, 1e-4
    ky, kx = 2 * np.pi * np.fft.fftfreq(ny, dy), 2 * np.pi * np.fft.fftfreq(nx, dx)
    x = -0.5 * dt * D * (ky[:, None] ** 2 + kx[None, :] ** 2)
    plan = get_plan(ny, nx, dy, dx, "spectral", torch.float64, cuda)
    ut = torch.tensor(u, device=cuda)
    out = torch.empty_like(ut)
    full = N.lib().mjx_spec2d_ws_bytes(ny, nx, 1, plan.code)
    for steps in (1, 3):
        ref = u
        for _ in range(steps):
            ref = np.real(np.fft.ifft2(np.fft.fft2(ref) * (1 + x) / (1 - x)))
        for nbytes in (full, ny * ((nx // 2 + 1 + 3) // 4 * 4) * 16):
            ws = torch.empty(nbytes, dtype=torch.uint8, device=cuda)
            N.check("mjx_fft_cn2d", N.lib().mjx_fft_cn2d(
                N.ptr(plan.buf), C.byref(plan.cgrid), plan.code, D, dt, steps, N.ptr(ut), N.ptr(out), N.ptr(ws),
                ws.numel(), N.stream_ptr(cuda)))
            assert float(np.max(np.abs(out.cpu().numpy() - ref))) < 1e-13 * max(1.0, float(np.max(np.abs(u))))
    assert N.lib().mjx_fft_cn2d(N.ptr(plan.buf), C.byref(plan.cgrid), plan.code, D, dt, 1, N.ptr(ut), N.ptr(out),
                                N.ptr(ws), ws.numel() - 16, N.stream_ptr(cuda)) == 10  # MJX_WORKSPACE


@pytest.mark.parametrize("n,m", [(8, 32), (64, 128), (128, 512), (256, 2048), (1024, 256), (2048, 1024)])
def test_fp32_passes_each_last_radix(cuda, n, m):
    """FP32 row and column transforms of every length class of the pass tables (no second pass, a
    last pass of radix 2, 4, 8 or 16 at sub-length 16 or 256), both ways round,
    against the FP64 oracle.  Tolerance: 1.2e-7 a radix-2 level and direction, 24 levels at
    most, rounded up; a misplaced twiddle gives an error of order one."""
    from moljax_gb300.core import fft_solvers
    rng = np.random.default_rng(n + 5 * m)
    for ny, nx in ((n, m), (m, n)):
        plan = fft_solvers.get_plan(ny, nx, 1.0 / ny, 1.0 / nx, "fd", torch.float32, cuda)
        rhs = rng.standard_normal((2, ny, nx))
        out = plan.apply(torch.tensor(rhs, dtype=torch.float32, device=cuda), [1e-4, 2e-4], 0.5, 1).cpu().numpy()
        lam = mol.fd_symbol_2d(ny, nx, 1.0 / ny, 1.0 / nx)
        for f in range(2):
            assert _rel(out[f], mol.solve_helmholtz_2d(rhs[f], lam, 0.5, [1e-4, 2e-4][f])) < 3e-6
