"""The reconstruction with infinite and NaN amplitudes and template values: they
reach the columns of their spike's window and no others, with the values that the
definition gives there, sum_i a_i (sum_k U[y_i, k, c] wPCA[k, s - x_i + nt/2]).

The gradients: infinite where the definition's are, which contracts a spike's window
of the incoming gradient before its amplitude is taken; finite elsewhere.

Tolerance: an element adds n K products in the tensors' precision, each rounded at
most three times, so it errs by at most (n K + 3) eps of the sum of its terms'
magnitudes. A gradient's entry adds n nt (templates), n C (basis) or K C nt
(amplitudes) products, bounded the same way.
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


@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('value', [float('inf'), -float('inf'), float('nan')])
@pytest.mark.parametrize('where', ['amplitude', 'template', 'gradient'])
@pytest.mark.parametrize('C, K, nt, N', [(5, 3, 21, 300), (130, 6, 61, 1000), (520, 2, 33, 200), (33, 1, 1, 70)])
def test_gradients_of_non_finite_values(dtype, value, where, C, K, nt, N):
    from livespikesorter_b200.adjoint import Reconstruction
    T, n = 4, 70                              # over 64 spikes: two batches of shares for a template
    g = torch.Generator().manual_seed(C + nt)
    U = torch.randn(T, K, C, generator=g, dtype=torch.float64)
    W = torch.randn(K, nt, generator=g, dtype=torch.float64)
    G = torch.randn(C, N, generator=g, dtype=torch.float64)
    a = torch.rand(n, generator=g, dtype=torch.float64) + 0.5
    x = torch.randint(nt, N - nt, (n,), generator=g)
    y = torch.zeros(n, dtype=torch.long)
    y[:3] = torch.tensor([T - 1, 1, 2])       # the value's template has one spike
    if where == 'amplitude':
        a[0] = value
    elif where == 'template':
        U[T - 1, K - 1, C // 2] = value
    else:
        G[C // 2, int(x[0])] = value
    U, W, a, G = (t.to(dtype) for t in (U, W, a, G))
    Uq, Wq, aq = (t.cuda().requires_grad_(True) for t in (U, W, a))
    R = Reconstruction.apply(Uq, Wq, aq, x.cuda(), y.cuda(), N)
    got = [v.cpu().double().numpy() for v in torch.autograd.grad(R, (Uq, Wq, aq), G.cuda())]
    Un, Wn, an, Gn = (t.double().numpy() for t in (U, W, a, G))

    def sums(Un, Wn, an, Gn):
        dU, dW, da = np.zeros_like(Un), np.zeros_like(Wn), np.zeros_like(an)
        for i in range(n):
            win = Gn[:, int(x[i]) - nt // 2:int(x[i]) - nt // 2 + nt]
            P = np.einsum('km,cm->kc', Wn, win)
            dU[y[i]] += an[i] * P
            dW += an[i] * np.einsum('kc,cm->km', Un[y[i]], win)
            da[i] = (Un[y[i]] * P).sum()
        return dU, dW, da

    with np.errstate(invalid='ignore'):
        want, mag = sums(Un, Wn, an, Gn), sums(*(np.abs(v) for v in (Un, Wn, an, Gn)))
    for p, q, m, terms in zip(got, want, mag, (n * nt, n * C, K * C * nt)):
        fin = np.isfinite(q)
        assert np.array_equal(np.isfinite(p), fin)
        if where != 'gradient':               # (there the kernels' order gives infinities where the sum above mixes signs)
            assert np.array_equal(np.isnan(p), np.isnan(q)) and np.array_equal(p[np.isinf(q)], q[np.isinf(q)])
        assert (np.abs(p[fin] - q[fin]) <= (terms + 3) * torch.finfo(dtype).eps * m[fin]).all()
    assert any((~np.isfinite(q)).any() for q in want) and any(np.isfinite(q).any() for q in want)
