"""Calls of different sizes from two threads at the same time: a launch of one
thread takes as much shared memory as its own sizes ask for, whatever the other
thread's calls ask for meanwhile. Results are compared bit for bit with the same
calls made one after the other."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _together(jobs):
    """Runs the jobs at the same time, each on its own thread and stream; their errors."""
    errors, gate = [], threading.Barrier(len(jobs))

    def work(job):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                gate.wait()
                job()
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001 (reported by the test)
            errors.append(repr(e))

    ts = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    return errors


def _recon_job(K, nt, C, passes):
    """Forward and backward kernels at these sizes, straight through the C entry points
    (a few microseconds of host work each, so that the threads' calls interleave)."""
    from livespikesorter_b200 import _lib
    lib = _lib.load()
    T, n, N = 3, 10, 200
    g = torch.Generator().manual_seed(K)
    U, W, a, G = (torch.randn(*s, generator=g).cuda() for s in ((T, K, C), (K, nt), (n,), (C, N)))
    x = torch.randint(0, N, (n,), generator=g, dtype=torch.int32).sort().values.cuda()
    y = (torch.arange(n, dtype=torch.int32) * T // n).cuda()
    order = torch.arange(n, dtype=torch.int32).cuda()
    start = torch.searchsorted(y, torch.arange(T + 1, dtype=torch.int32).cuda()).int()
    out = [torch.zeros_like(t) for t in (G, U, W, a)] + [torch.zeros(T, K, nt, device='cuda')]
    R, dU, dW, da, work = out
    arrays = dict(U=U, W=W, x=x, y=y, a=a, o=order, s=start, G=G)
    ptr = {k: v.data_ptr() for k, v in arrays.items()}

    def once():
        st = torch.cuda.current_stream().cuda_stream
        _lib.check(lib.lss_recon_forward(0, ptr['U'], ptr['W'], T, K, C, nt, ptr['x'], ptr['y'], ptr['a'], n,
                                         R.data_ptr(), N, st))
        _lib.check(lib.lss_recon_backward(0, ptr['U'], ptr['W'], T, K, C, nt, ptr['x'], ptr['a'], ptr['o'], ptr['s'],
                                          ptr['G'], N, dU.data_ptr(), dW.data_ptr(), da.data_ptr(), work.data_ptr(), st))

    once()
    want = [t.clone() for t in out[:4]]
    torch.cuda.synchronize()

    def job(keep=arrays):
        for _ in range(passes):
            once()
        torch.cuda.current_stream().synchronize()
        assert all(torch.equal(p, q) for p, q in zip(out, want))
    return job


def test_reconstructions_of_different_sizes():
    assert not _together([_recon_job(K, nt, C, 5000) for K, nt, C in ((2, 21, 8), (16, 255, 40), (1, 5, 8), (8, 61, 64))])


def _match_job(T, nt, N, passes):
    from livespikesorter_b200 import setup_tensors as st
    from livespikesorter_b200 import synth
    from livespikesorter_b200.sorter import Sorter
    g = torch.Generator().manual_seed(T)
    K, C, nC = 3, 12, 10
    W = torch.linalg.qr(torch.randn(nt, K, generator=g))[0].T.contiguous()
    U = 20 * torch.randn(T, K, C, generator=g)
    probe = synth.probe_two_column(C)
    iCC, iU, Ucc = st.prepare_extract(probe.xc, probe.yc, U, nC)
    s = Sorter(U=U, wPCA=W, ctc=st.prepare_matching(W, U), Wrot=torch.eye(C), iCC=iCC, iU=iU, Ucc=Ucc, NT=N - 2 * nt,
               Th=6.0, do_CAR=False)
    rows = 10 * torch.randn(N, C, generator=g)
    for i in range(6):
        x = 2 * nt + i * (N - 4 * nt) // 6
        rows[x:x + nt] += 2 * torch.einsum('kc,km->mc', U[i % T], W)
    rows = rows.round().to(torch.int16).cuda()
    want = s.sort_batch(rows, 1, 3, on_device=True)
    assert len(want['time']) > 0
    torch.cuda.synchronize()

    def job():
        for _ in range(passes):
            r = s.sort_batch(rows, 1, 3, on_device=True)
            assert all(torch.equal(r[k], want[k]) for k in want)
    return job


def test_sorters_of_different_sizes():
    assert not _together([_match_job(*a, 600) for a in ((20, 21, 300), (150, 129, 900), (40, 61, 400), (100, 31, 600))])
