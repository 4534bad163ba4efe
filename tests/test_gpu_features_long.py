"""PC features of long and of crowded batches: more spikes near a CTA's columns than
its list holds, so that the columns are taken piece by piece. The features follow the
definition in FP64 (tolerance as for the other feature tests, 1e-3 of the largest: FP32
sums over C * nt terms in another order), and the stage's time grows with the spikes:
five times the batch may take three times as long per spike (work per spike is the
same at any length; the room is for timing noise and the last, partly filled wave)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
C, NC = 32, 10


def _sorter(K, nt, NT, max_rounds, precision='fp32'):
    from livespikesorter_b200 import setup_tensors as st
    from livespikesorter_b200 import synth
    from livespikesorter_b200.sorter import Sorter
    g = torch.Generator().manual_seed(100 * K + nt)
    T = 32
    W = torch.linalg.qr(torch.randn(nt, K, generator=g))[0].T.contiguous()
    mid = torch.rand(T, generator=g) * (C - 1)
    U = 30 * torch.randn(T, K, 1, generator=g) * torch.exp(-(torch.arange(C) - mid[:, None, None]) ** 2 / 4)
    probe = synth.probe_two_column(C)
    iCC, iU, Ucc = st.prepare_extract(probe.xc, probe.yc, U, NC)
    s = Sorter(U=U, wPCA=W, ctc=st.prepare_matching(W, U), Wrot=torch.eye(C), iCC=iCC, iU=iU, Ucc=Ucc, NT=NT, Th=1.0,
               do_CAR=False, max_rounds=max_rounds, max_spikes=8 * NT, precision=precision)
    rng = np.random.default_rng(K + nt)
    rows = np.round(30 * rng.standard_normal((NT + 2 * nt, C))).astype(np.int16)
    return s, (U, W, Ucc, iCC, iU), rows


@pytest.mark.parametrize('K, nt, NT, max_rounds, precision', [
    (6, 21, 60000, 150, 'fp32'),
    (3, 21, 60001, 150, 'bf16'),
    (6, 61, 300000, 100, 'fp32'),
])
def test_pieces_of_a_slice(K, nt, NT, max_rounds, precision):
    s, (U, W, Ucc, iCC, iU), rows = _sorter(K, nt, NT, max_rounds, precision)
    X = s.filter(rows, 1, 3).cpu().double()
    r = s.sort_batch(rows, 1, 3)
    x = r['time'] - NT + nt + nt // 2 - 20
    y, amp = r['template'].long(), r['amplitude'].double()
    # over 1024 spikes near the columns of one of 148 CTAs
    w = -(-s.N // 148)
    assert max(int(((x >= c - nt) & (x < c + w + nt)).sum()) for c in range(0, NT, w)) > 1024
    wave = torch.einsum('nkc,km->ncm', U.double(), W.double())
    lag = torch.arange(nt) - nt // 2
    big = float(r['pc'].abs().max())
    for lo in (nt, NT // 3, NT - 500):                      # a few hundred columns each
        near = torch.nonzero((x >= lo - 2 * nt) & (x < lo + 400 + 2 * nt)).ravel()
        Xr = X.clone()[:, lo - nt:] if lo == nt else X[:, lo - 4 * nt:lo + 400 + 4 * nt].clone()
        off = lo - nt if lo == nt else lo - 4 * nt
        for i in near.tolist():
            c = x[i] + lag - off
            ok = (c >= 0) & (c < Xr.shape[1])
            Xr[:, c[ok]] -= amp[i] * wave[y[i]][:, ok]
        mine = near[(x[near] >= lo) & (x[near] < lo + 400)]
        assert len(mine) > 50
        ch = iCC[:, iU[y[mine]]].T
        win = Xr[ch[:, :, None], (x[mine, None] + lag - off)[:, None, :]]
        want = win @ W.double().T + amp[mine, None, None] * Ucc[:, y[mine]].permute(1, 0, 2).double()
        assert (r['pc'][mine].double() - want).abs().max() <= 1e-3 * big


def test_time_grows_with_the_spikes():
    per = []
    for NT in (60000, 300000):
        s, _, rows = _sorter(6, 61, NT, 100)
        rows = torch.from_numpy(rows).cuda()
        s.set_profiling(True)
        ms = []
        for _ in range(4):
            n = len(s.sort_batch(rows, 1, 3, on_device=True)['time'])
            ms.append(s.stage_times()['feature_ms'])
        assert n > NT // 2
        per.append(min(ms) / n)
    assert per[1] < 3 * per[0], per
