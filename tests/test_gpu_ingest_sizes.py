"""Channel means and common-average reference over channel counts, batch lengths and values at the edges of the
median search (32 values per warp turn, brackets of at most 32 values, equal values, outliers, the int16 range) and of
the column tiles, against their definition in FP32: x = fl(raw - fl(mean)), x - lower median over the channels.

The whitening is the identity (products with 0 and 1: exact), so the batch must be equal bit for bit.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rows(kind, N, C, rng):
    if kind == 'noise':
        r = 30 * rng.standard_normal((N, C)) + rng.integers(-300, 300, C)
    elif kind == 'equal':
        r = np.full((N, C), -5)
    elif kind == 'range':
        r = rng.integers(-32768, 32768, (N, C))
    elif kind == 'two values':
        r = 7 * rng.integers(0, 2, (N, C))
    elif kind == 'outliers':
        r = np.where(rng.random((N, C)) < 0.3, -20000, 5 * rng.standard_normal((N, C)))
    else:  # skewed
        r = 20 * np.exp(2 * rng.standard_normal((N, C)))
    return np.clip(np.round(r), -32768, 32767).astype(np.int16)


@pytest.mark.parametrize('C', [1, 2, 31, 32, 33, 64, 65, 96, 200, 384, 385, 700, 1024])
@pytest.mark.parametrize('NT, nt', [(50, 5), (301, 61), (5000, 61)])
def test_mean_and_median(C, NT, nt):
    from livespikesorter_b200.sorter import Sorter
    g = torch.Generator().manual_seed(C)
    T, K = 4, 2
    W = torch.linalg.qr(torch.randn(nt, K, generator=g))[0].T.contiguous()
    rng = np.random.default_rng(C + NT)
    cmap = rng.permutation(C + 3)[:C]
    s = Sorter(U=torch.randn(T, K, C, generator=g), wPCA=W, ctc=torch.zeros(T, T, 2 * nt + 1), Wrot=torch.eye(C), NT=NT,
               n_chan_bin=C + 3, chan_map=cmap)
    N = NT + 2 * nt
    for kind in ('noise', 'equal', 'range', 'two values', 'outliers', 'skewed'):
        rows = _rows(kind, N, C + 3, rng)
        for ib, n in ((0, NT // 2), (1, N), (2, N - 7)):
            X = s.filter(rows[:n], ib, 3).cpu()
            r = rows[:n, cmap].T.astype(np.float64)
            if ib == 0:    # nt copies of the first row, then the rows, then zeros
                r = np.concatenate([np.repeat(r[:, :1], nt, 1), r, np.zeros((C, N - nt - n))], 1)
            else:          # the last row repeated
                r = np.concatenate([r, np.repeat(r[:, -1:], N - n, 1)], 1)
            mean = torch.from_numpy(r.sum(1) * (1.0 / N)).float()   # exact sums
            x = torch.from_numpy(r).float() - mean[:, None]
            x = x - torch.median(x, 0)[0]
            assert torch.equal(X, x), (kind, ib)
