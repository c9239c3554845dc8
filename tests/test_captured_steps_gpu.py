"""What a captured step holds by value follows what is set after the capture, on a B200: the wall constants of the
FP32-bulk step (of the x-mean profiles that a state is split into) and the settings of the closure model."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CFG = dict(Lx=2 * np.pi, stretch=1, beta=1.5, Ub=1.0, Reb=2000.0, F0=0.05, nforce=4, lin_drag=1e-3, adapt=1)


def start(s, mean):
    """The laminar vorticity with an x-mean part of its own, and a wave."""
    y = s.metric(0)
    x = np.arange(s.Nx) * (2 * np.pi / s.Nx)
    w = (3.0 * y + mean * np.sin(np.pi * (y + 1.0)))[:, None] + 0.05 * np.sin(np.pi * (y + 1.0))[:, None] * np.cos(2 * x)[None]
    s.set_omega(np.ascontiguousarray(w))


def same(a, b):
    return a.time() == b.time() and all(np.array_equal(x, y) for x, y in zip(a.fields(), b.fields()))


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("Nx,Ny", [(2048, 65), (1024, 700), (128, 65), (16, 33)])
def test_a_second_state_steps_as_in_a_new_channel(nse, cuda, Nx, Ny, precision):
    """set_omega with another mean profile after steps: the graphs of nse2d_step and nse2d_run step it as a new channel."""
    a, b = (nse.Solver(Nx=Nx, Ny=Ny, precision=precision, **CFG) for _ in range(2))
    start(a, 0.0)
    a.step(2, use_graph=True)
    a.run(max_steps=2)
    start(a, 0.4)
    start(b, 0.4)
    for s in (a, b):
        s.step(2, use_graph=True)
        s.run(max_steps=2)
    assert same(a, b)
    a.close()
    b.close()


@pytest.mark.parametrize("precision", [64, 32])
def test_an_ensembles_second_states_step_as_in_new_channels(nse, cuda, precision):
    sizes = [(128, 65), (256, 40), (2048, 33)]
    members = [nse.Solver(Nx=Nx, Ny=Ny, precision=precision, **CFG) for Nx, Ny in sizes]
    alone = [nse.Solver(Nx=Nx, Ny=Ny, precision=precision, **CFG) for Nx, Ny in sizes]
    ens = nse.Ensemble(members)
    for m in members:
        start(m, 0.0)
    ens.step(2)
    for m, s in zip(members, alone):
        start(m, 0.4)
        start(s, 0.4)
        s.step(3, use_graph=True)
    ens.step(3)
    assert all(same(m, s) for m, s in zip(members, alone))
    ens.close()


def test_a_state_with_walls_of_its_own(nse, cuda):
    """FP32: a state whose wall vorticity is not the closure's of its psi has wall constants of its own, which the
    steps captured before it do not hold; the same through an ensemble's graph."""
    for Nx, Ny in ((2048, 65), (16, 33)):
        a, b, c = (nse.Solver(Nx=Nx, Ny=Ny, precision=32, **CFG) for _ in range(3))
        ens = nse.Ensemble([c])
        for s in (a, c):
            start(s, 0.0)
        a.step(2, use_graph=True)
        a.run(max_steps=2)
        ens.step(2)
        start(b, 0.0)
        w, psi = b.fields()
        w[0] += 0.5
        w[-1] -= 0.25
        for s in (a, b, c):
            s.set_state(w, psi)
        for s in (a, b):
            s.step(2, use_graph=True)
            s.run(max_steps=2)
        ens.step(4)
        b_alone = b.time(), b.fields()
        assert same(a, b)
        assert b_alone[0] == c.time() and all(np.array_equal(x, y) for x, y in zip(b_alone[1], c.fields()))
        ens.close()


def test_a_models_settings_after_steps(nse, cuda):
    """Scales, gain, wall rows and the mean-flow switch of a model that is attached already."""
    Nx, Ny = 64, 33

    def attached():
        s = nse.Solver(Nx=Nx, Ny=Ny, **CFG)
        net = nse.Cnn(Nx, Ny, s.metric(0), 16, 1)
        net.init_params(3)
        net.set_scales([2.0, 0.75, 0.6, 0.1], 10.0)
        net.set_application(1, 0.25, True)
        s.set_closure(net, every_stage=True)
        start(s, 0.0)
        return s, net

    def change(net):
        net.set_scales([1.0, 0.5, 0.6, 0.2], 5.0)
        net.set_application(2, 0.125, False)
    (a, na), (b, nb) = attached(), attached()
    ens = nse.Ensemble([a])
    for run in (lambda s: s.step(2, use_graph=True), lambda s: s.run(max_steps=2), lambda s: ens.step(2) if s is a else s.step(2)):
        for n in (na, nb):
            n.set_scales([2.0, 0.75, 0.6, 0.1], 10.0)
            n.set_application(1, 0.25, True)
        start(a, 0.0)
        run(a)                                               # captured with the first settings
        change(na)
        change(nb)
        start(a, 0.0)
        start(b, 0.0)
        run(a)
        b.step(2)                                            # by plain launches, which hold nothing
        assert same(a, b)
    a.set_closure(None)                                      # and without the model
    b.set_closure(None)
    for s in (a, b):
        start(s, 0.0)
    ens.step(2)
    b.step(2)
    assert same(a, b)
    ens.close()
