"""Deferred rounds against the rounds that update every row where the numbering of a round's peaks matters: batches cut
off after a few rounds, more peaks than the list holds, over 30 peaks near one CTA's columns, peaks closer than two
template lengths (their order depends on the round's peaks before them) and none that close."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(T, N, nt, gap, seed, **kw):
    """Scores with a peak about every `gap` columns, and a sorter for them."""
    from livespikesorter_b200 import setup_tensors as st
    from livespikesorter_b200.sorter import Sorter
    g = torch.Generator().manual_seed(seed)
    K, C = 3, 6
    W = torch.linalg.qr(torch.randn(nt, K, generator=g))[0].T.contiguous()
    U = 5 * torch.randn(T, K, C, generator=g)
    nm = (U ** 2).sum((1, 2))
    B = 0.5 * torch.randn(T, N, generator=g) * nm[:, None].sqrt()
    x = torch.arange(nt + 1, N - nt - 1, gap) + torch.randint(0, 3, (len(range(nt + 1, N - nt - 1, gap)),), generator=g)
    x = x[x < N - nt - 1]
    y = torch.randint(0, T, (len(x),), generator=g)
    B[y, x] = nm[y].sqrt() * (8 + 4 * torch.rand(len(x), generator=g))
    s = Sorter(U=U, wPCA=W, ctc=st.prepare_matching(W, U), Wrot=torch.eye(C), NT=N - 2 * nt, Th=6.0, nm=nm, **kw)
    return s, B.cuda()


@pytest.mark.parametrize('T, N, nt, gap, max_rounds', [
    (20, 30000, 5, 7, 100),       # over 30 peaks near a CTA's columns, all of them close
    (20, 30000, 5, 14, 100),      # ... none close in the first round
    (40, 20000, 61, 70, 100),     # every pair close
    (40, 20000, 61, 150, 100),    # close pairs only in later rounds
    (40, 20000, 61, 500, 1),
    (40, 20000, 61, 70, 1),
    (40, 20000, 61, 70, 2),
    (33, 700, 61, 65, 3),
    (33, 300, 31, 35, 100),
])
def test_rounds_equal(T, N, nt, gap, max_rounds):
    s, B = _case(T, N, nt, gap, T + gap + max_rounds, max_rounds=max_rounds)
    got = []
    for deferred in (False, True):
        s.set_round_kernel(deferred)
        st, amps = s.match_scores(B)
        got.append((st, amps, s.stats()['rounds']))
    assert len(got[0][0]) > 0
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert got[0][2] == got[1][2]


@pytest.mark.parametrize('max_spikes', [1, 100, 150])
def test_overflowing_list_is_refused(max_spikes):
    from livespikesorter_b200._lib import LssError
    s, B = _case(20, 20000, 61, 130, 1, max_spikes=max_spikes)      # about 150 peaks in the first round
    for deferred in (False, True):
        s.set_round_kernel(deferred)
        with pytest.raises(LssError):
            s.match_scores(B)
