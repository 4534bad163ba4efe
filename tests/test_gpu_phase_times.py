"""The rounds' phase times are means over the CTAs that ran: every CTA's four phases
add up to the time of the rounds, so the four means do too, within the launch and
the read-back that the stage's device time holds beside them. 4768 columns are 150
chunks of 32: the deferred rounds take them with 75 CTAs of two chunks, about half of
the SMs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('deferred', [True, False])
@pytest.mark.parametrize('N', [4768, 4736, 700])
def test_phases_add_up_to_the_rounds(N, deferred):
    from livespikesorter_b200 import setup_tensors as st
    from livespikesorter_b200.sorter import Sorter
    g = torch.Generator().manual_seed(N)
    T, K, C, nt = 200, 3, 8, 31
    W = torch.linalg.qr(torch.randn(nt, K, generator=g))[0].T.contiguous()
    U = 20 * torch.randn(T, K, C, generator=g)
    s = Sorter(U=U, wPCA=W, ctc=st.prepare_matching(W, U), Wrot=torch.eye(C), NT=N - 2 * nt, Th=0.5, max_rounds=100,
               do_CAR=False)
    s.set_round_kernel(deferred)
    s.set_profiling(True)
    rows = (100 * torch.randn(N, C, generator=g)).round().to(torch.int16).cuda()
    share = []
    for _ in range(5):
        s.sort_batch(rows, 1, 3, on_device=True, with_pc=False)
        p = s.stats()['mp_phases_ms']
        share.append(sum(p[k] for k in ('peak', 'peak_wait', 'update', 'update_wait')) / s.stage_times()['mp_ms'])
    assert s.stats()['rounds'] > 50
    share = sorted(share)[2]
    assert 0.6 < share < 1.1, share
