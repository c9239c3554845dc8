"""The kernel forms of a step on grids where each of them is the one that runs, on a B200.

  - The two-pass and the cluster solve: grids of more than 1026 rows (below, one CTA solves two or four columns whatever
    the plan says). They reassociate the same recurrences: 1e-12 of the largest psi in FP64; in the FP32-bulk step
    1e-6 of psi and 1e-5 of omega, as between its other forms.
  - The two stage kernels: rows of 2048 points and tall grids, which have no bands. The same bits.
  - Programmatic dependent launch: steps that are captured by the caller (by launches on every grid). The same bits.
  - Steps in one launch against the step by separate kernels (nse2d_step_profiled), for the layouts that
    test_band_gpu.py leaves out: one to four rows a CTA, two and four columns a solve, one to eight rows a segment.
"""
import ctypes

import numpy as np
import pytest

from test_parity_gpu import laminar_perturbed, relerr

pytestmark = pytest.mark.gpu

CFG = dict(Lx=2 * np.pi, stretch=1, beta=1.2, Ub=1.0, Reb=2000.0, F0=0.05, nforce=4, lin_drag=1e-3, adapt=1)


def channel(nse, Nx, Ny, precision, seed=3, **plan):
    s = nse.Solver(Nx=Nx, Ny=Ny, precision=precision, **CFG)
    if plan:
        s.set_plan(**plan)
    s.set_omega(laminar_perturbed(Nx, Ny, s.metric(0), seed=seed, amp=2e-2))
    return s


def kernels(s):
    return {s.lib.nse2d_step_kernel_name(s.h, k).decode() for k in range(s.launches_per_step())}


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("Nx,Ny", [(128, 1100), (1024, 1027), (64, 2500)])
def test_solves_of_tall_grids_agree(nse, cuda, Nx, Ny, precision):
    a, b = (channel(nse, Nx, Ny, precision, tridiag_clusters=cl) for cl in (1, 0))
    assert "k_thomas_cluster" in kernels(a)
    assert {"k_thomas_maps", "k_thomas_apply"} <= kernels(b)
    for s in (a, b):
        s.step(3, use_graph=True)
    (wa, pa), (wb, pb) = a.fields(), b.fields()
    if precision == 64:
        assert np.max(np.abs(pa - pb)) <= 1e-12 * np.max(np.abs(pa))
        assert np.max(np.abs(wa[2:-2] - wb[2:-2])) <= 1e-10 * np.max(np.abs(wa))
    else:
        assert relerr(pb, pa) < 1e-6 and relerr(wb[2:-2], wa[2:-2]) < 1e-5
    a.close()
    b.close()


@pytest.mark.parametrize("Nx,Ny,clusters", [(128, 1100, 0), (64, 4099, 0), (64, 4098, 1), (2048, 1100, 0)])
def test_two_pass_solve_matches_the_oracle(nse, oracle, cuda, Nx, Ny, clusters):
    """The Poisson solve by the two passes, which more than 4098 rows always take, at the 1e-12 of the other solves."""
    torch = cuda
    s = nse.Solver(Nx=Nx, Ny=Ny, **dict(CFG, beta=1.0))
    s.set_tridiag_form(bool(clusters))
    assert ("k_thomas_cluster" in kernels(s)) == bool(clusters)
    w = np.random.default_rng(Nx + Ny).standard_normal((Ny, Nx))
    wd = torch.from_numpy(w).cuda()
    pd = torch.zeros_like(wd)
    s.poisson_solve(wd, pd)
    torch.cuda.synchronize()
    m = oracle.metrics(Nx, Ny, 2 * np.pi, 1.0, 1, 1.0)
    assert relerr(pd.cpu().numpy(), oracle.poisson_solve(w, 2 * np.pi, m, 0.0, 2.0)) < 1e-12
    s.close()


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("Nx,Ny", [(256, 1800 * 2), (1024, 700), (2048, 129)])
def test_stage_kernels_give_the_same_bits(nse, cuda, Nx, Ny, precision):
    a, b = (channel(nse, Nx, Ny, precision, stage_tma=st) for st in (1, 0))
    f = "32" if precision == 32 else ""
    assert f"k_stage{f}_tma" in kernels(a) and f"k_stage{f}" in kernels(b)
    for s in (a, b):
        s.step(3, use_graph=True)
    assert a.time() == b.time()
    assert all(np.array_equal(x, y) for x, y in zip(a.fields(), b.fields()))
    a.close()
    b.close()


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("Nx,Ny", [(256, 129), (1024, 300), (512, 700), (1024, 700), (2048, 257)])
def test_programmatic_launches_of_a_captured_step(nse, cuda, Nx, Ny, precision):
    """A caller's graph of two steps, launched twice, with each kernel launched programmatically and in stream order,
    and the same steps by nse2d_step (in one launch where the grid has it)."""
    torch = cuda
    out = []
    for pdl in (1, 0, None):
        s = channel(nse, Nx, Ny, precision, pdl=pdl or 0)
        s.step(1)
        if pdl is None:
            s.step(4)
        else:
            g = torch.cuda.CUDAGraph()
            torch.cuda.synchronize()
            with torch.cuda.graph(g):
                s.step(2, stream=torch.cuda.current_stream())
            for _ in range(2):
                g.replay()
            torch.cuda.synchronize()
            del g
        out.append((s.time(), s.fields()))
        s.close()
    for t, f in out[1:]:
        assert t == out[0][0] and t[2] == 5
        assert all(np.array_equal(x, y) for x, y in zip(f, out[0][1]))


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("Nx,Ny", [(64, 65), (64, 514), (128, 300), (256, 130), (256, 514), (512, 150), (512, 257), (512, 514), (1024, 131),
                                   (1024, 300), (1024, 446), (1024, 513), (1024, 514)])
def test_steps_in_one_launch_give_the_plain_step(nse, cuda, Nx, Ny, precision):
    a, b = (channel(nse, Nx, Ny, precision, seed=Nx + Ny) for _ in range(2))
    a.step(2, use_graph=True)
    a.step_store_rhs(1)
    ms = [ctypes.c_double() for _ in range(3)]
    for _ in range(3):
        assert b.lib.nse2d_step_profiled(b.h, *[ctypes.byref(x) for x in ms], None) == 0
    assert a.time() == b.time()
    assert all(np.array_equal(x, y) for x, y in zip(a.fields(), b.fields()))
    rhs = np.empty((2, Ny, Nx))
    for s, out in zip((a, b), rhs):
        assert s.lib.nse2d_get_field(s.h, 4, out.ctypes.data_as(ctypes.c_void_p), None) == 0
    assert np.array_equal(rhs[0], rhs[1]) and np.all(np.isfinite(rhs))
    a.close()
    b.close()
