"""The row-band kernels (csrc/band.cuh) on a B200, where their splits can go wrong: the smallest rows, rows of
one to several bands, bands of uneven length, the fewest rows of a grid (both walls in one band), and every
row length with a transform plan of its own.

A step by the row-band kernels evaluates the per-point and transform arithmetic of the step by separate
kernels (the one that nse2d_step_profiled times): the same fields and the same stored rhs to the bit. The
Poisson solve is compared with the oracle at the 1e-12 of the other solves."""
import ctypes

import numpy as np
import pytest

from test_parity_gpu import laminar_perturbed, relerr

pytestmark = pytest.mark.gpu

GRIDS = [(64, 5), (64, 6), (64, 11), (64, 900), (128, 150), (128, 1333), (256, 151), (256, 300), (512, 9), (512, 597), (1024, 6),
         (1024, 595), (1024, 745), (2048, 5), (2048, 61)]


@pytest.mark.parametrize("Nx,Ny", GRIDS)
def test_band_step_gives_the_plain_step_and_solve_the_oracle(nse, oracle, cuda, Nx, Ny):
    torch = cuda
    cfg = dict(Nx=Nx, Ny=Ny, Lx=2 * np.pi, stretch=1, beta=1.5, Ub=1.0, Reb=2000.0, F0=0.05, nforce=4, lin_drag=1e-3, adapt=1)
    a, b = nse.Solver(**cfg), nse.Solver(**cfg)
    w0 = laminar_perturbed(Nx, Ny, a.metric(0), seed=Nx + Ny, amp=2e-2)
    a.set_omega(w0)
    b.set_omega(w0)
    ms = [ctypes.c_double() for _ in range(3)]
    rhs = np.empty((2, Ny, Nx))
    for _ in range(3):
        a.step_store_rhs(1)
        assert b.lib.nse2d_step_profiled(b.h, *[ctypes.byref(x) for x in ms], None) == 0
        assert a.time() == b.time()
        assert all(np.array_equal(x, y) for x, y in zip(a.fields(), b.fields()))
        for s, out in zip((a, b), rhs):
            assert s.lib.nse2d_get_field(s.h, 4, out.ctypes.data_as(ctypes.c_void_p), None) == 0
        assert np.array_equal(rhs[0], rhs[1])
    assert np.all(np.isfinite(a.fields()[0]))
    m = oracle.metrics(Nx, Ny, 2 * np.pi, 1.0, 1, 1.5)
    w = np.random.default_rng(Nx * Ny).standard_normal((Ny, Nx))
    wd = torch.from_numpy(w).cuda()
    pd = torch.zeros_like(wd)
    a.poisson_solve(wd, pd)
    torch.cuda.synchronize()
    assert relerr(pd.cpu().numpy(), oracle.poisson_solve(w, 2 * np.pi, m, 0.0, 2.0)) < 1e-12
    a.close()
    b.close()


@pytest.mark.parametrize("Nx,Ny", [(64, 5), (64, 37), (128, 150), (256, 66), (256, 301), (512, 9), (512, 301), (512, 650), (1024, 300),
                                   (1024, 514), (2048, 40)])
def test_fp32_band_step_gives_the_plain_step(nse, cuda, Nx, Ny):
    """The FP32-bulk step by bands and in one launch against the one by separate kernels: the same bits; and the same
    steps through nse2d_run."""
    cfg = dict(Nx=Nx, Ny=Ny, Lx=2 * np.pi, stretch=1, beta=1.5, Ub=1.0, Reb=2000.0, F0=0.05, nforce=4, lin_drag=1e-3, adapt=1, precision=32)
    a, b, c = (nse.Solver(**cfg) for _ in range(3))
    w0 = laminar_perturbed(Nx, Ny, a.metric(0), seed=Nx + Ny, amp=2e-2)
    for s in (a, b, c):
        s.set_omega(w0)
    ms = [ctypes.c_double() for _ in range(3)]
    a.step(2, use_graph=True)
    a.step_store_rhs(1)
    for _ in range(3):
        assert b.lib.nse2d_step_profiled(b.h, *[ctypes.byref(x) for x in ms], None) == 0
    assert c.run(max_steps=3) == nse.HALT_BUDGET
    rhs = np.empty((2, Ny, Nx))
    for s in (b, c):
        assert a.time() == s.time()
        assert all(np.array_equal(x, y) for x, y in zip(a.fields(), s.fields()))
        for q, out in zip((a, s), rhs):
            assert q.lib.nse2d_get_field(q.h, 4, out.ctypes.data_as(ctypes.c_void_p), None) == 0
        assert np.array_equal(rhs[0], rhs[1])
    assert np.all(np.isfinite(a.fields()[0]))
    for s in (a, b, c):
        s.close()


@pytest.mark.parametrize("precision", [64, 32])
def test_steps_in_one_launch_follow_the_schedule(nse, cuda, precision):
    """Many steps in one launch, runs to an output time and single steps give the same dt, times and fields as steps
    one at a time (whose dt is trimmed and snapped to the same schedule)."""
    cfg = dict(Nx=128, Ny=70, Lx=2 * np.pi, stretch=1, beta=1.5, Ub=1.0, Reb=2000.0, F0=0.05, nforce=4, lin_drag=1e-3, adapt=1,
               precision=precision)
    a, b = nse.Solver(**cfg), nse.Solver(**cfg)
    w0 = laminar_perturbed(128, 70, a.metric(0), seed=3, amp=2e-2)
    for s in (a, b):
        s.set_omega(w0)
    a.step(7)
    for _ in range(7):
        b.step(1)
    assert a.time() == b.time()
    t, dt = a.time()[:2]
    t_out = t + 12.3 * dt
    assert a.run(next_snap=t_out) & nse.HALT_OUTPUT
    b.set_schedule(t_out, 1e300)
    while b.time()[0] < t_out:
        b.step(1)
    assert a.time() == b.time() and a.time()[0] == t_out
    assert all(np.array_equal(x, y) for x, y in zip(a.fields(), b.fields()))
    a.close()
    b.close()


@pytest.mark.parametrize("Nx,Ny", [(64, 515), (512, 1026), (1024, 515), (1024, 777), (1024, 1026), (2048, 520), (64, 1027)])
def test_solve_of_tall_columns(nse, oracle, cuda, Nx, Ny):
    """The one-CTA tridiagonal solve of 513 to 1024 interior rows (two or four columns a CTA) and the first grid
    beyond it: the Poisson solve against the oracle at the 1e-12 of the other solves, an FP32-bulk step against the
    FP64 one at the 1e-5 of its psi."""
    from test_fp32_gpu import omega0, rel
    torch = cuda
    cfg = dict(Nx=Nx, Ny=Ny, Lx=2 * np.pi, stretch=1, beta=1.5, Ub=1.0, Reb=2000.0, adapt=1)
    a, b = nse.Solver(**cfg), nse.Solver(precision=32, **cfg)
    m = oracle.metrics(Nx, Ny, 2 * np.pi, 1.0, 1, 1.5)
    w = np.random.default_rng(Nx * Ny).standard_normal((Ny, Nx))
    wd = torch.from_numpy(w).cuda()
    pd = torch.zeros_like(wd)
    a.poisson_solve(wd, pd)
    torch.cuda.synchronize()
    assert relerr(pd.cpu().numpy(), oracle.poisson_solve(w, 2 * np.pi, m, 0.0, 2.0)) < 1e-12
    w0 = omega0(Nx, Ny, a.metric(0))
    for s in (a, b):
        s.set_omega(w0)
        s.step(1)
    assert rel(b.fields()[1], a.fields()[1]) < 1e-5
    a.close()
    b.close()


@pytest.mark.parametrize("precision,Nx,Ny,bands", [
    (64, 1024, 594, True), (64, 1024, 595, False), (64, 1024, 4097, False), (64, 512, 890, True), (64, 512, 891, False), (64, 512, 2049, False),
    (64, 128, 1778, True), (64, 128, 1779, False), (64, 64, 4097, False), (32, 1024, 594, True), (32, 1024, 595, False), (32, 512, 2049, False),
    (32, 128, 3554, True), (32, 128, 3555, False), (32, 64, 8193, False)])
def test_bands_while_they_fit_the_device(nse, cuda, precision, Nx, Ny, bands):
    """The step by bands of rows is taken while its bands are resident at once (of rows of up to 256 points: in two
    rounds), on 148 SMs; taller grids take the separate kernels, which are the faster ones there."""
    s = nse.Solver(Nx=Nx, Ny=Ny, Lx=2 * np.pi, stretch=1, beta=1.0, Ub=1.0, Reb=2000.0, adapt=1, precision=precision)
    names = [s.lib.nse2d_step_kernel_name(s.h, k).decode() for k in range(s.launches_per_step())]
    assert ("k_band_inv_stage_fwd" in names) == bands, names
    s.close()


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("Nx,Ny,names", [
    (1024, 700, ("k_rows_fwd", "k_thomas_wide", "k_rows_inv")), (2048, 300, ("k_rows_fwd", "k_thomas_cta", "k_rows_inv")),
    (16, 129, ("k_fft_fwd", "k_thomas_cta", "k_ifft_thom")), (4096, 1500, ("k_fft_fwd", "k_thomas_cluster", "k_ifft_thom"))])
def test_the_names_are_those_of_the_kernels(nse, cuda, precision, Nx, Ny, names):
    """A step by separate kernels names the transforms and the solve that its grid uses, and nse2d_step_profiled counts
    them as transforms and as solve."""
    s = nse.Solver(Nx=Nx, Ny=Ny, Lx=2 * np.pi, stretch=1, beta=1.0, Ub=1.0, Reb=2000.0, adapt=1, precision=precision)
    got = [n for n, _ in s.step_timed(1)]
    want = [n + "32" if precision == 32 and n in ("k_fft_fwd", "k_ifft_thom") else n for n in names]
    assert [n for n in got if not n.startswith(("k_stage", "k_maxuv"))] == want * 3, got
    ms = [ctypes.c_double() for _ in range(3)]
    assert s.lib.nse2d_step_profiled(s.h, *[ctypes.byref(x) for x in ms], None) == 0
    step, fft, tri = (x.value for x in ms)
    assert fft > 0 and tri > 0 and fft + tri < step
    s.close()


@pytest.mark.parametrize("Ny,rows", [(5, True), (594, True), (595, False), (739, False), (742, True), (1778, True), (1779, False), (2073, False),
                                     (2074, True), (2371, True)])
def test_rows_of_2048_points_either_side_of_a_round(nse, oracle, cuda, Ny, rows):
    """Four rows of 2048 points to a CTA, unless their last round over 148 SMs is nearly empty: the transforms named in
    the step, the Poisson solve (which takes one row to a CTA on grids of less than a round too) against the oracle at
    the 1e-12 of the other solves, and an FP32-bulk step against the FP64 one at the 1e-5 of its psi."""
    from test_fp32_gpu import omega0, rel
    torch = cuda
    cfg = dict(Nx=2048, Ny=Ny, Lx=2 * np.pi, stretch=1, beta=1.0, Ub=1.0, Reb=2000.0, adapt=1)
    a, b = nse.Solver(**cfg), nse.Solver(precision=32, **cfg)
    for s in (a, b):
        names = [s.lib.nse2d_step_kernel_name(s.h, k).decode() for k in range(s.launches_per_step())]
        assert ("k_rows_fwd" in names) == rows and ("k_rows_inv" in names) == rows, names
    w = np.random.default_rng(Ny).standard_normal((Ny, 2048))
    wd = torch.from_numpy(w).cuda()
    pd = torch.zeros_like(wd)
    a.poisson_solve(wd, pd)
    torch.cuda.synchronize()
    m = oracle.metrics(2048, Ny, 2 * np.pi, 1.0, 1, 1.0)
    assert relerr(pd.cpu().numpy(), oracle.poisson_solve(w, 2 * np.pi, m, 0.0, 2.0)) < 1e-12
    w0 = omega0(2048, Ny, a.metric(0))
    for s in (a, b):
        s.set_omega(w0)
        s.step(1)
    assert rel(b.fields()[1], a.fields()[1]) < 1e-5
    a.close()
    b.close()
