"""The training step's sums: gradients, loss and trained parameters equal to the last bit from run to
run (every partial sum is added in one order), the loss and the gradients against FP64, and the GEMM's
96-column tiles with FP32 stores.

Tolerances.  Loss: a thread adds at most batch * 16 / 256 squares, a tree of 8 levels follows, and d and
d^2 round once each: at most (batch / 16 + 12) 2^-24 relative.  Gradients: the restatement rounds to BF16
where the device does and sums exactly, so the two part only where the device's FP32 sums (off by some
1e-5 of a value, truncating accumulators included) fall on the other side of a BF16 rounding: 5e-3 of the
values by 2^-8, 3e-4 in norm a layer, and over the 12 layers of both passes in quadrature 1e-3; 4e-3 is
asked.  A row of a map left out or an offset lost at its border shows as several percent.
"""
import numpy as np
import pytest

import cnn_oracle as CO

pytestmark = pytest.mark.gpu


def _net(B, seed=1):
    from aldic_b200.learned import ProposalNet

    net = ProposalNet(0, max_batch=(B + 7) // 8 * 8)
    net.set_params(CO.init_params(seed))
    return net


def _batch(seed, B):
    import torch

    rng = np.random.default_rng(seed)
    X = rng.normal(size=(B, 72, 72, 2)).astype(np.float32)
    X[:, :, :, 0] = 0.0
    X[:, 16:56, 16:56, 0] = rng.normal(size=(B, 40, 40))
    T = rng.normal(scale=0.5, size=(B, 6)).astype(np.float32)
    return torch.from_numpy(X).cuda().to(torch.bfloat16), torch.from_numpy(T).cuda()


@pytest.mark.parametrize("B", [8, 72, 256, 512])
def test_training_repeats_to_the_bit(B):
    x, t = _batch(B, B)
    net = _net(B)
    try:
        p0, runs, loss = net.get_params(), [], []
        for _ in range(3):
            net.set_params(p0)
            loss.append([net.train_step(x, t, 1e-3, want_loss=True) for _ in range(8)])
            runs.append(net.get_params())
        assert not np.array_equal(runs[0], p0)
        assert all(np.array_equal(r, runs[0]) for r in runs[1:])
        assert all(v == loss[0] for v in loss[1:])
        net.set_params(p0)
        g = [net.gradients(x, t) for _ in range(4)]
        assert all(l == g[0][0] and np.array_equal(v, g[0][1]) for l, v in g[1:])
        net.status()
    finally:
        net.close()


@pytest.mark.parametrize("B", [8, 264, 4096])
def test_loss_against_fp64(B):
    import torch

    x, t = _batch(3, 8)
    x, t = x.repeat((B + 7) // 8, 1, 1, 1)[:B].contiguous(), torch.randn((B, 6), device="cuda")
    net = _net(B)
    try:
        y = torch.empty((B, 6), dtype=torch.float32, device="cuda")
        net.forward(x, y)
        loss, _ = net.gradients(x, t)
        want = float((y.double() - t.double()).square().mean())
        assert abs(loss - want) <= (B / 16 + 12) * 2.0 ** -24 * want
    finally:
        net.close()


@pytest.mark.parametrize("B", [24, 40])
def test_gradients_against_the_restatement(B):
    x, t = _batch(20 + B, B)
    net = _net(B, 2)
    try:
        _, g = net.gradients(x, t)
        _, want = CO.loss_and_gradients(CO.init_params(2), x.float().cpu().numpy(), t.cpu().numpy())
        for l, (ow, ob) in enumerate(CO.layout()[0]):
            for a, b in ((ow, ob), (ob, ob + CO.ROWS[l])):
                off = np.linalg.norm(g[a:b] - want[a:b]) / np.linalg.norm(want[a:b])
                assert off < 4e-3, (l, a, off)
    finally:
        net.close()


@pytest.mark.parametrize("M,N,K", [(8, 288, 32), (130, 288, 32), (4800, 288, 32), (300, 480, 64), (257, 576, 200)])
def test_gemm_columns_of_96(M, N, K):
    """FP32 stores of column tiles of 96 (288 and 576 columns; 480 takes tiles of 256), whole and ragged rows."""
    import torch

    from aldic_b200.learned import gemm_bf16

    gen = torch.Generator(device="cuda").manual_seed(M)
    a, b = (torch.randn((n, K), device="cuda", generator=gen).to(torch.bfloat16) for n in (M, N))
    c = torch.full((M, N + 4), 7.0, device="cuda")
    gemm_bf16(a, b, c[:, :N])
    torch.cuda.synchronize()
    want, scale = a.double() @ b.double().T, a.double().abs() @ b.double().abs().T
    assert float(((c[:, :N].double() - want).abs() / scale).max()) < 1e-5  # K 2^-24 at most, as summed in FP32
    assert bool((c[:, N:] == 7.0).all())
