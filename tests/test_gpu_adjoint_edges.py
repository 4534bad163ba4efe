"""The reconstruction and its adjoint at the edges of their tiling, in FP64,
against a dense sum over spikes and lags and its torch autograd: template lengths
around the 32-lag register slots, channels around the 32/64/128-channel groups and
past one cluster's eight chunks, batches that do not fill a column tile, spikes
whose windows reach outside the batch, templates without spikes.

Tolerance: both sides add at most n * nt * K * C products of unit-scale numbers in
FP64, each sum over m <= 2e4 terms errs by at most m * 2^-53 of its absolute sum;
1e-11 of the result's largest magnitude is 4x above that for these sizes.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _dense(U, W, amp, x, y, N):
    """R[c, s] by a scatter over spikes and lags; terms outside [0, N) dropped."""
    nt = W.shape[1]
    cols = x.long()[:, None] + torch.arange(nt, device=x.device) - nt // 2
    wave = torch.einsum('nkc,km->cnm', U[y.long()], W) * amp[None, :, None]
    pad = 512
    R = torch.zeros(U.shape[2], N + 2 * pad, device=U.device, dtype=U.dtype)
    return R.index_add(1, (cols + pad).reshape(-1), wave.reshape(U.shape[2], -1))[:, pad:pad + N]


@pytest.mark.parametrize('C, T, K, nt, N, n', [
    (1, 1, 1, 1, 1, 1),
    (8, 4, 3, 2, 63, 20),
    (31, 5, 6, 32, 65, 40),
    (33, 3, 16, 33, 200, 70),        # more spikes of a template than one batch of shares (64)
    (64, 7, 6, 61, 257, 60),
    (65, 2, 6, 64, 128, 150),
    (127, 6, 4, 65, 1000, 90),
    (129, 3, 2, 128, 999, 30),
    (130, 3, 2, 129, 700, 25),
    (520, 4, 3, 61, 300, 30),        # nine chunks of 64 channels: two rounds of a cluster of eight
    (300, 2, 2, 255, 600, 12),
])
def test_reconstruction_and_gradients_at_tile_edges(C, T, K, nt, N, n):
    from livespikesorter_b200.adjoint import Reconstruction
    g = torch.Generator().manual_seed(C * 1000 + nt)
    U = torch.randn(T + 1, K, C, generator=g, dtype=torch.float64).cuda()   # the last template has no spikes
    W = torch.randn(K, nt, generator=g, dtype=torch.float64).cuda()
    x = torch.randint(-nt, N + nt, (n,), generator=g, dtype=torch.int32).cuda()
    y = torch.randint(0, T, (n,), generator=g, dtype=torch.int32).cuda()
    a = (torch.rand(n, generator=g, dtype=torch.float64) + 0.5).cuda()
    G = torch.randn(C, N, generator=g, dtype=torch.float64).cuda()

    def run(fn):
        Uq, Wq, aq = (t.detach().clone().requires_grad_(True) for t in (U, W, a))
        R = fn(Uq, Wq, aq)
        return (R.detach(),) + torch.autograd.grad((R * G).sum(), (Uq, Wq, aq))

    got = run(lambda Uq, Wq, aq: Reconstruction.apply(Uq, Wq, aq, x, y, N))
    want = run(lambda Uq, Wq, aq: _dense(Uq, Wq, aq, x, y, N))
    for p, q in zip(got, want):
        assert (p - q).abs().max() <= 1e-11 * max(1.0, float(q.abs().max()))
    again = run(lambda Uq, Wq, aq: Reconstruction.apply(Uq, Wq, aq, x, y, N))
    assert all(torch.equal(p, q) for p, q in zip(got, again))               # deterministic
