"""The deferred rounds (mp_lazy.cu) at the sizes where they can go wrong.

Score fields of overlapping spikes on a few channels, whose templates all
interact, against the oracle's run_matching on the same field: spikes and
amplitudes bit-identical (every step is IEEE-exact elementwise work, so there is
no tolerance). Sizes: template counts around the 16-row blocks and the 32-block
groups, column counts around the 32-column chunks, slices narrower than a spike
window, rounds that fill the spike log (512 entries per slice) several times,
slices whose keys do not fit in shared memory, short and long templates.
Fields with infinite and NaN scores are compared with the rounds that update
every row.
"""
import numpy as np
import pytest
import torch

import ks4_oracle as ko

pytestmark = pytest.mark.gpu


def _field(T, N, nt, seed, K=2, C=6, density=0.02, noise=2.0):
    from livespikesorter_b200 import setup_tensors as st
    g = torch.Generator().manual_seed(seed)
    W = torch.linalg.qr(torch.randn(nt, K, generator=g))[0].T.contiguous()
    # footprints along the channels, so that the probe order means something
    c = torch.arange(C).float()
    mid = torch.rand(T, generator=g) * (C - 1)
    U = torch.randn(T, K, 1, generator=g) * torch.exp(-(c - mid[:, None, None]) ** 2)
    U = U + 0.05 * torch.randn(T, K, C, generator=g)
    ctc = st.prepare_matching(W, U)
    B = noise * torch.randn(T, N, generator=g) * (U ** 2).sum((1, 2)).sqrt()[:, None]
    n = max(1, int(density * N))
    x = torch.randint(0, N, (n,), generator=g)
    y = torch.randint(0, T, (n,), generator=g)
    a = 4.0 + 8.0 * torch.rand(n, generator=g)
    for xi, yi, ai in zip(x.tolist(), y.tolist(), a.tolist()):
        lo, hi = max(0, xi - nt), min(N, xi + nt + 1)
        B[:, lo:hi] += ai * ctc[:, yi, lo - xi + nt:hi - xi + nt]
    return U, W, ctc, B


def _sorter(U, W, ctc, N, th, max_rounds):
    from livespikesorter_b200.sorter import Sorter
    nm = (U ** 2).sum((1, 2))
    return nm, Sorter(U=U, wPCA=W, ctc=ctc, Wrot=torch.eye(U.shape[2]), NT=N - 2 * W.shape[1], Th=th, nm=nm,
                      max_rounds=max_rounds)


@pytest.mark.parametrize('T, N, nt, density, max_rounds', [
    (1, 95, 15, 0.05, 100),            # one template, three chunks
    (15, 64, 15, 0.1, 100),            # two whole chunks, a partial block
    (16, 97, 31, 0.1, 100),            # one whole block; slices narrower than a window
    (17, 1023, 61, 0.02, 100),
    (33, 4736, 15, 0.05, 100),         # one chunk per CTA on 148 SMs
    (40, 4737, 7, 0.1, 100),           # and one column more
    (31, 20011, 15, 0.08, 100),        # logs that fill up
    (8, 30000, 5, 0.15, 200),          # ... several times
    (530, 3001, 31, 0.02, 100),        # more than 32 blocks: two groups
    (60, 2500, 127, 0.01, 100),        # long templates
    (330, 190000, 15, 0.01, 4),        # keys of a slice in global memory
])
def test_deferred_rounds_bit_exact(T, N, nt, density, max_rounds):
    th = 6.0
    U, W, ctc, B = _field(T, N, nt, seed=T + N, density=density)
    nm, s = _sorter(U, W, ctc, N, th, max_rounds)
    st_o, amps_o, _ = ko.run_matching(torch.zeros(U.shape[2], N), U, ctc, W, th, nt, B=B, nm=nm,
                                      max_rounds=max_rounds)
    assert len(st_o) > 0
    s.set_round_kernel(True)
    for n in (N, N - 1) if N < 5000 else (N,):   # and a batch shorter than the handle's
        if n != N:
            st_o, amps_o, _ = ko.run_matching(torch.zeros(U.shape[2], n), U, ctc, W, th, nt, B=B[:, :n].contiguous(),
                                              nm=nm, max_rounds=max_rounds)
        st, amps = s.match_scores(B[:, :n].contiguous().cuda())
        assert torch.equal(st.cpu(), st_o)
        assert torch.equal(amps.cpu(), amps_o)


def test_infinite_and_nan_scores_as_with_every_row_updated():
    T, N, nt = 24, 3000, 31
    U, W, ctc, B = _field(T, N, nt, seed=3)
    rng = np.random.default_rng(0)
    for v in (float('inf'), -float('inf'), float('nan')):
        B[torch.from_numpy(rng.integers(0, T, 5)), torch.from_numpy(rng.integers(nt, N - nt, 5))] = v
    _, s = _sorter(U, W, ctc, N, 6.0, 30)
    got = {}
    for skip in (False, True):
        s.set_round_kernel(skip)
        got[skip] = s.match_scores(B.cuda())
    assert len(got[False][0]) > 0
    assert torch.equal(got[False][0], got[True][0])
    assert torch.equal(got[False][1], got[True][1], ) or torch.allclose(got[False][1], got[True][1], rtol=0, atol=0,
                                                                        equal_nan=True)


def test_a_flat_field_is_refused_by_both_kernels():
    """More than 31 equal peaks within 2nt samples of one another: refused with
    LSS_ERR_CAPACITY, whichever kernel runs the rounds."""
    from livespikesorter_b200._lib import LssError
    T, N, nt = 4, 600, 31
    U, W, ctc, B = _field(T, N, nt, seed=5, density=0.0, noise=0.0)
    B[:] = 0.0
    B[1, 200:300] = 1e4
    _, s = _sorter(U, W, ctc, N, 6.0, 5)
    for skip in (False, True):
        s.set_round_kernel(skip)
        with pytest.raises(LssError, match='31 peaks'):
            s.match_scores(B.cuda())
