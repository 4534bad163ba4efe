"""Which rounds kernel a handle runs, and what it says about it. The deferred rounds
count the (spike, tile) updates that they meet (mp_items); the rounds that update
every row count none, which tells the two apart."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _sorter(T, N, nt=15, seed=0):
    from livespikesorter_b200 import setup_tensors as st
    from livespikesorter_b200.sorter import Sorter
    g = torch.Generator().manual_seed(seed)
    K, C = 2, 6
    W = torch.linalg.qr(torch.randn(nt, K, generator=g))[0].T.contiguous()
    U = 5 * torch.randn(T, K, C, generator=g)
    s = Sorter(U=U, wPCA=W, ctc=st.prepare_matching(W, U), Wrot=torch.eye(C), NT=N - 2 * nt, Th=6.0, max_rounds=3)
    return s


def _deferred(s, N):
    """Does a batch of this sorter run the deferred rounds?"""
    B = torch.zeros(s.T, N)
    B[0, N // 2] = 1e4
    st, _ = s.match_scores(B.cuda())
    assert len(st) > 0
    return s.stats()['mp_items'] > 0


def _c_get(s):
    v = ctypes.c_int32(-1)
    assert s._lib.lss_get_round_kernel(s._h, ctypes.byref(v)) == 0
    return v.value


@pytest.mark.parametrize('T', [3, 599, 600])
def test_reported_kernel_is_the_one_that_runs(T):
    N = 700
    s = _sorter(T, N)
    assert _deferred(s, N)                                   # a fresh handle defers
    assert _c_get(s) == 1 and s.rounds_deferred()
    s.set_round_kernel(s.rounds_deferred())                  # what it reports, set back: nothing changes
    assert _deferred(s, N)
    s.set_round_kernel(False)
    assert _c_get(s) == 0 and not s.rounds_deferred() and not s.round_kernel()
    assert not _deferred(s, N)
    s.set_round_kernel(s.rounds_deferred())
    assert not _deferred(s, N)
    s.set_round_kernel(True)
    assert _c_get(s) == 1 and s.rounds_deferred() and s.round_kernel()
    assert _deferred(s, N)


def test_slices_too_wide_for_the_deferred_rounds():
    """A slice takes about 45 bytes of shared memory per column: a million columns over
    148 SMs do not fit, and every row is updated whatever was asked for."""
    N = 1_000_000
    s = _sorter(1, N)
    for told in (None, True):
        if told is not None:
            s.set_round_kernel(told)
        assert not _deferred(s, N)
        assert _c_get(s) == 0 and not s.rounds_deferred()
