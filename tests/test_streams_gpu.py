"""Channels on several streams and threads, and other work beside a channel's steps, on a B200."""
import threading

import numpy as np
import pytest

from test_parity_gpu import laminar_perturbed

pytestmark = pytest.mark.gpu


def channel(nse, Nx, Ny, seed, precision=64):
    s = nse.Solver(Nx=Nx, Ny=Ny, Lx=2 * np.pi, stretch=1, beta=1.5, Ub=1.0, Reb=2000.0, F0=0.05, nforce=4, lin_drag=1e-3, adapt=1,
                   precision=precision)
    s.set_omega(laminar_perturbed(Nx, Ny, s.metric(0), seed=seed, amp=2e-2))
    return s


def test_a_kernel_of_another_stream_does_not_wait_for_all_steps(nse, cuda):
    """4000 steps of 1024x513 are 0.2 s; a small kernel of another stream comes in between."""
    torch = cuda
    s = channel(nse, 1024, 513, 1)
    q1, q2 = torch.cuda.Stream(), torch.cuda.Stream()
    x = torch.zeros(1 << 16, device="cuda")
    s.step(1, use_graph=True, stream=q1)
    x.add_(1)
    torch.cuda.synchronize()
    s.step(4000, use_graph=True, stream=q1)
    with torch.cuda.stream(q2):
        x.add_(1)
    q2.synchronize()
    assert not q1.query()
    q1.synchronize()
    s.close()


@pytest.mark.parametrize("precision", [64, 32])
def test_a_long_call_is_its_steps(nse, cuda, precision):
    """Calls that are cut into several launches, by nse2d_step and by nse2d_run, give the bits of short ones."""
    a, b, c = (channel(nse, 128, 70, 3, precision) for _ in range(3))
    a.step(300)
    for n in (1, 63, 64, 65, 107):
        b.step(n)
    assert c.run(max_steps=300) == nse.HALT_BUDGET
    for s in (b, c):
        assert a.time() == s.time() and a.time()[2] == 300
        assert all(np.array_equal(x, y) for x, y in zip(a.fields(), s.fields()))
    for s in (a, b, c):
        s.close()


@pytest.mark.parametrize("precision", [64, 32])
def test_channels_of_several_threads_are_those_alone(nse, cuda, precision):
    """Four threads, each with a channel and a stream of its own, which run and step at the same time."""
    torch = cuda
    sizes = [(128, 129), (256, 65), (64, 40), (512, 130)]
    alone = [channel(nse, Nx, Ny, k, precision) for k, (Nx, Ny) in enumerate(sizes)]
    for s in alone:
        s.run(max_steps=700)
        s.step(150)
    beside = [channel(nse, Nx, Ny, k, precision) for k, (Nx, Ny) in enumerate(sizes)]
    fail = []

    def work(s):
        try:
            q = torch.cuda.Stream()
            assert s.run(max_steps=700, stream=q) == nse.HALT_BUDGET
            for _ in range(10):
                s.step(15, use_graph=True, stream=q)
            q.synchronize()
        except Exception as e:                               # noqa: BLE001 (reported by the test)
            fail.append(e)
    threads = [threading.Thread(target=work, args=(s,)) for s in beside]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not fail, fail
    for a, b in zip(alone, beside):
        assert a.time() == b.time() and a.nonfinite() == b.nonfinite() == 0
        assert all(np.array_equal(x, y) for x, y in zip(a.fields(), b.fields()))
    for s in alone + beside:
        s.close()
