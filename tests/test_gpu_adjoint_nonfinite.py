"""The reconstruction with infinite and NaN amplitudes and template values: they
reach the columns of their spike's window and no others, with the values that the
definition gives there, sum_i a_i (sum_k U[y_i, k, c] wPCA[k, s - x_i + nt/2]).

Tolerance: an element adds n K products in the tensors' precision, each rounded at
most three times, so it errs by at most (n K + 3) eps of the sum of its terms'
magnitudes.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('value', [float('inf'), -float('inf'), float('nan')])
@pytest.mark.parametrize('where', ['amplitude', 'template'])
@pytest.mark.parametrize('C, K, nt, N', [(5, 3, 21, 300), (130, 6, 61, 1000), (33, 1, 1, 70)])
def test_non_finite_values_stay_in_their_windows(dtype, value, where, C, K, nt, N):
    from livespikesorter_b200.adjoint import reconstruct
    T, n = 4, 12
    g = torch.Generator().manual_seed(C + nt)
    U = torch.randn(T, K, C, generator=g, dtype=torch.float64)
    W = torch.randn(K, nt, generator=g, dtype=torch.float64)
    a = torch.rand(n, generator=g, dtype=torch.float64) + 0.5
    x = torch.randint(0, N, (n,), generator=g)
    x[0], x[1], x[2] = 31, 64, N - 1          # windows that end beside a tile's columns, and at the batch's end
    y = torch.arange(n) % (T - 1)
    if where == 'amplitude':
        a[0] = a[2] = value
    else:
        y[0] = T - 1                          # this spike's template alone has the value, in one channel
        U[T - 1, K - 1, C // 2] = value
    U, W, a = U.to(dtype), W.to(dtype), a.to(dtype)
    got = reconstruct(U.cuda(), W.cuda(), x.cuda(), y.cuda(), a.cuda(), N).cpu().double().numpy()
    Un, Wn, an = U.double().numpy(), W.double().numpy(), a.double().numpy()
    want, mag = np.zeros((C, N)), np.zeros((C, N))
    with np.errstate(invalid='ignore'):
        for i in torch.argsort(x, stable=True).tolist():
            lo = int(x[i]) - nt // 2
            cols = np.arange(max(lo, 0), min(lo + nt, N))
            wave = np.einsum('kc,km->cm', Un[y[i]], Wn[:, cols - lo])
            want[:, cols] += an[i] * wave
            mag[:, cols] += np.abs(an[i]) * np.einsum('kc,km->cm', np.abs(Un[y[i]]), np.abs(Wn[:, cols - lo]))
    fin = np.isfinite(want)
    assert 0 < (~fin).sum() < fin.size
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[np.isinf(want)], want[np.isinf(want)])
    assert (np.abs(got[fin] - want[fin]) <= (n * K + 3) * torch.finfo(dtype).eps * mag[fin]).all()
