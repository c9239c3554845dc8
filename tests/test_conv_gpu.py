"""The closure model's convolutions and weight gradients (csrc/conv_tc.cuh) at their edges, on a B200, against
the CPU oracle: every width of the hidden layers, batches, pixel counts that are not multiples of the 128 and
64 pixels of a tile (fewer pixels than one tile too), rows that are not powers of two, and fields of few rows,
where most taps meet a wall. Bars as in test_closure_gpu.py: the output within 1e-2 of its largest magnitude,
every gradient within 3e-2 in the relative L2 norm, the loss within 1e-3 (a hidden activation next to a BF16
rounding boundary can round the other way)."""
import numpy as np
import pytest

from conftest import load_oracle_module
from test_closure_gpu import SCALES, _dev, _net, _rel, _sample

pytestmark = pytest.mark.gpu

co = load_oracle_module("closure_oracle")


@pytest.mark.parametrize("Nx,Ny,H,idx", [(4, 5, 16, (0,)), (20, 9, 16, (1, 0)), (12, 7, 48, (2, 0, 3)), (34, 11, 48, (0,)),
                                         (64, 33, 64, (3, 1)), (128, 5, 32, (0, 1, 2, 3)), (96, 40, 32, (2,))])
def test_edges_match_the_oracle(nse, cuda, Nx, Ny, H, idx):
    torch = cuda
    net, y = _net(nse, Nx, Ny, H, 7, max_batch=len(idx) + 1)
    S = [_sample(Ny, Nx, 30 + s) for s in range(4)]
    out = torch.full((Ny, Nx), 7.0, dtype=torch.float64, device="cuda")
    net.forward(*[_dev(torch, f) for f in S[1][:4]], out)
    ref = co.predict(net.params(), *S[1][:4], y, SCALES, bf=True)
    assert np.abs(out.cpu().numpy() - ref).max() <= 1e-2 * np.abs(ref).max()
    stack = [_dev(torch, np.stack([smp[f] for smp in S])) for f in range(5)]
    loss = net.gradients(*stack, idx=idx)
    ref_loss, ref_grads = co.loss_and_grads(net.params(), [S[i] for i in idx], y, SCALES, bf=True)
    assert abs(loss - ref_loss) <= 1e-3 * ref_loss, (loss, ref_loss)
    for layer in range(4):
        gw, gb = net.get_grads(layer)
        assert _rel(gw, ref_grads[layer][0]) < 3e-2, (layer, _rel(gw, ref_grads[layer][0]))
        assert _rel(gb, ref_grads[layer][1]) < 3e-2, (layer, _rel(gb, ref_grads[layer][1]))


@pytest.mark.parametrize("Nx,Ny,H,idx", [(256, 6, 16, (0, 2)), (130, 7, 32, (1,)), (64, 130, 32, (0, 1, 2, 3)), (66, 40, 64, (3, 0)),
                                         (128, 150, 48, (1, 2)), (8, 161, 16, (0, 1, 2, 3))])
def test_strips_match_the_oracle(nse, cuda, Nx, Ny, H, idx):
    """Strips of one and of two rows, a row of one and of several strips, and tiles that run over the rows' ends."""
    test_edges_match_the_oracle(nse, cuda, Nx, Ny, H, idx)


@pytest.mark.parametrize("H", [16, 32, 48, 64])
def test_an_infinite_target_gives_infinite_gradients(nse, cuda, H):
    """One infinite tau at a pixel whose whole neighbourhood is away from the walls, with weights, biases and inputs
    that are all positive: its dZ is -inf in every channel of every layer and every activation that it meets is
    positive, so every gradient is -inf; a NaN would come of a split of dZ that subtracts infinities."""
    torch = cuda
    Nx, Ny = 32, 33
    net = nse.Cnn(Nx, Ny, np.linspace(0.5, 1.5, Ny), H, 1)
    rng = np.random.default_rng(H)
    for layer in range(4):
        ci, co_ = net.shape(layer)
        net.set_params(layer, rng.uniform(0.01, 0.02, (co_, 9, ci)), rng.uniform(0.1, 0.2, co_))
    net.set_scales(*SCALES)
    f = [rng.uniform(0.5, 1.0, (Ny, Nx)) for _ in range(5)]
    f[4][16, 9] = np.inf
    assert net.gradients(*[_dev(torch, a[None]) for a in f]) == np.inf
    for layer in range(4):
        for g in net.get_grads(layer):
            assert np.all(g == -np.inf), (layer, np.unique(g)[:4])


@pytest.mark.parametrize("H", [16, 32, 48, 64])
@pytest.mark.parametrize("Nx,Ny", [(128, 150), (250, 80)])
def test_strips_of_two_rows_and_two_tiles_match_the_oracle(nse, cuda, Nx, Ny, H):
    """Four fields whose strips of two rows fill the device twice, so that a CTA has two tiles, of one row each."""
    assert 4 * -(-Nx // 128) * -(-Ny // 2) >= 2 * 148
    test_edges_match_the_oracle(nse, cuda, Nx, Ny, H, (3, 0, 2, 1))


@pytest.mark.parametrize("H", [16, 32, 48, 64])
def test_sums_of_the_gradients_in_64_bits(nse, cuda, H):
    """The sums of the input gradient and of the weight gradients alone, against 64 bits. Everything around them is
    exact: constant activations of 20 (GELU' is 1), targets of 64 .. 127 times 2^24, beside which the output is lost in
    rounding, output weights of a few bits and a pixel count that is a power of two, so that dZ above the sums is the
    same to the bit and its rounding to BF16 too.

    A tensor core truncates at every step of a sum, 2^-24 of the sum on average over the step, of sums that grow from
    zero: n steps lose n 2^-26. Input gradient: 9 H / 16 steps in 1, 2, 2 or 3 accumulators, at most 14 steps each;
    weight gradient: 6 steps. Together 20 2^-26 = 3.0e-7, and 0.5e-7 for the additions in FP32."""
    torch = cuda
    Nx, Ny, B = 64, 34, 2
    rng = np.random.default_rng(H)
    net = nse.Cnn(Nx, Ny, np.zeros(Ny), H, B)
    net.set_scales([1.0] * 4, 1.0)
    W = []
    for layer in range(4):
        ci, c_out = net.shape(layer)
        w = rng.integers(-100, 101, (c_out, 9, ci)) / 2.0 ** 12 if layer == 3 else 0.005 * rng.standard_normal((c_out, 9, ci))
        net.set_params(layer, w, np.full(c_out, 20.0 if layer < 3 else 0.0))
        W.append(co.bf16(w))
    tau = rng.integers(64, 128, (B, Ny, Nx)) * 2.0 ** 24
    zero = torch.zeros((B, Ny, Nx), dtype=torch.float64, device="cuda")
    net.gradients(zero, zero, zero, zero, _dev(torch, tau), idx=range(B))
    h1 = np.full((Ny, Nx, H), 20.0)
    z1 = np.einsum("jitc,otc->jio", co.im2col(h1), W[1]) + 20.0
    assert z1.min() > 8.0
    h2 = co.bf16(z1)
    ref = {1: [0.0, 0.0], 2: [0.0, 0.0]}
    for s in range(B):
        d = np.zeros((Ny, Nx))
        d[1:-1] = -2.0 * tau[s, 1:-1] / (B * Nx * (Ny - 2))
        dz = {2: co.col2im(np.einsum("jio,otc->jitc", co.bf16(d[:, :, None]), W[3]))}
        dz[1] = co.col2im(np.einsum("jio,otc->jitc", co.bf16(dz[2]), W[2]))
        for layer, h in ((1, h1), (2, h2)):
            ref[layer][0] = ref[layer][0] + np.einsum("jio,jitc->otc", dz[layer], co.im2col(h))
            ref[layer][1] = ref[layer][1] + dz[layer].sum((0, 1))
    for layer in (1, 2):
        for got, want in zip(net.get_grads(layer), ref[layer]):
            assert _rel(got, want) < 3.5e-7, (layer, _rel(got, want))
