"""lss_set_templates takes the templates and the basis from host, pinned or device
memory alike: the swapped handle scores and matches the same, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision', ['fp32', 'bf16'])
def test_templates_from_any_memory(precision):
    from livespikesorter_b200 import synth
    from livespikesorter_b200.sorter import Sorter
    a, rec = synth.config(0, duration_s=1.0, seed=21, T=24)
    b, _ = synth.config(0, duration_s=0.5, seed=22, T=24)
    U, W = b.U.float().contiguous(), b.wPCA.float().contiguous()
    got = []
    for place in (lambda t: t, lambda t: t.pin_memory(), lambda t: t.cuda()):
        s = Sorter.from_setup(a, precision=precision)
        u, w = place(U), place(W)
        torch.cuda.synchronize()
        assert s._lib.lss_set_templates(s._h, u.data_ptr(), w.data_ptr()) == 0
        X = torch.from_numpy(rec.raw[:5000].T.astype('float32')).contiguous()[:s.C].cuda()
        st, amps, _ = s.match(X)
        got.append((s.scores(X), st, amps))
    assert len(got[0][1]) > 0
    for g in got[1:]:
        assert all(torch.equal(p, q) for p, q in zip(g, got[0]))
