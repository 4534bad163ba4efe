"""PC features of a sorted batch over component counts, template lengths and
crowded batches, against the definition in FP64 on the sorter's own spikes:

  xfeat[i, j, k] = sum_m Xres[ch_j, x_i + m - nt/2] wPCA[k, m] + amp_i Ucc[j, y_i, k]

with Xres the filtered batch minus every spike's waveform (template_matching.py:50-51).
Tolerance as for the other feature tests: 1e-3 of the largest feature (FP32 sums over
C * nt terms in another order, and the whitening applied after the projection).
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _features64(X, U, W, Ucc, iCC, iU, x, y, amp):
    T, K, C = U.shape
    nt = W.shape[1]
    h = nt // 2
    pad = 2 * nt
    Xr = torch.zeros(C, X.shape[1] + 2 * pad, dtype=torch.float64)
    Xr[:, pad:-pad] = X.double()
    lag = torch.arange(nt) - h + pad
    wave = torch.einsum('nkc,km->ncm', U[y].double(), W.double()) * amp.double()[:, None, None]
    for i in range(len(x)):
        Xr[:, x[i] + lag] -= wave[i]
    ch = iCC[:, iU[y]].T                                              # [n, nC]
    win = Xr[ch[:, :, None], (x[:, None] + lag)[:, None, :]]
    return win @ W.double().T + amp.double()[:, None, None] * Ucc[:, y].permute(1, 0, 2).double()


@pytest.mark.parametrize('K, nt, NT, T, th, noise, precision', [
    (1, 61, 1000, 20, 8.0, 10, 'fp32'),
    (3, 41, 1500, 20, 8.0, 10, 'fp32'),
    (4, 61, 1001, 30, 8.0, 10, 'bf16'),
    (5, 81, 1300, 20, 8.0, 10, 'fp32'),
    (6, 61, 2111, 40, 8.0, 10, 'fp32'),
    (7, 61, 1200, 20, 8.0, 10, 'bf16'),
    (8, 41, 1999, 30, 8.0, 10, 'fp32'),
    (6, 129, 1500, 16, 8.0, 10, 'fp32'),      # over 48 KB of shared memory
    (8, 129, 1500, 16, 8.0, 10, 'fp32'),      # basis correlations too large for the columns kernel
    (2, 5, 400, 200, 0.5, 200, 'fp32'),       # over 1024 spikes near 64 columns
])
def test_features_of_a_sorted_batch(K, nt, NT, T, th, noise, precision):
    from livespikesorter_b200 import setup_tensors as st
    from livespikesorter_b200 import synth
    from livespikesorter_b200.sorter import Sorter
    C, nC = 40, 10
    g = torch.Generator().manual_seed(100 * K + nt)
    W = torch.linalg.qr(torch.randn(nt, K, generator=g))[0].T.contiguous()
    mid = torch.rand(T, generator=g) * (C - 1)
    U = 30 * torch.randn(T, K, 1, generator=g) * torch.exp(-(torch.arange(C) - mid[:, None, None]) ** 2 / 4)
    probe = synth.probe_two_column(C)
    iCC, iU, Ucc = st.prepare_extract(probe.xc, probe.yc, U, nC)
    rng = np.random.default_rng(K + nt)
    rows = noise * rng.standard_normal((NT + 2 * nt, C))
    for _ in range(T * 2):
        t, x = rng.integers(T), rng.integers(nt, NT)
        rows[x:x + nt] += 2.0 * torch.einsum('kc,km->mc', U[t], W).numpy()
    rows = np.clip(np.round(rows), -32768, 32767).astype(np.int16)
    s = Sorter(U=U, wPCA=W, ctc=st.prepare_matching(W, U), Wrot=torch.eye(C), iCC=iCC, iU=iU, Ucc=Ucc, NT=NT, Th=th,
               do_CAR=False, precision=precision,
               max_rounds=300 if th < 1 else 30)   # at most 256 neighbours per spike are taken
    X = s.filter(rows, 1, 3).cpu()
    r = s.sort_batch(rows, 1, 3)
    n = len(r['time'])
    assert n > 20
    x = r['time'] - NT + nt + nt // 2 - 20
    y = r['template'].long()
    if th < 1:
        assert max(int(((x >= c - nt) & (x < c + 64 + nt)).sum()) for c in range(0, NT, 64)) > 1024
    want = _features64(X, U, W, Ucc, iCC, iU, x, y, r['amplitude'])
    assert (r['pc'].double() - want).abs().max() <= 1e-3 * want.abs().max()
