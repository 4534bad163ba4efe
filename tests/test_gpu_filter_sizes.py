"""The whitening product of the filter over channel counts and batch lengths at the edges of its tiles (64 and 128
channels, 256 columns, slabs of 16 terms, rows of whole 16- and 8-byte pieces and not), against FP64.

Without common-average reference and temporal filter the batch is (M @ Wrot) @ x, x the rows less each channel's
mean. Tolerance: two FP32 FMA chains of C terms each, every partial sum rounded once, and two roundings in x:
|error| <= (2 C + 2) u (|M| @ |Wrot| @ (|rows| + |mean|)), u = 2**-24, with the second-order terms covered by a factor
of 1.01.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('C, NT, nt', [
    (1, 500, 5), (15, 700, 5), (33, 3001, 41), (64, 20000, 61), (65, 20001, 61), (96, 19998, 41), (128, 18932, 41),
    (130, 10000, 61), (193, 5000, 61), (200, 9999, 61), (384, 8192, 61), (385, 7003, 61),
])
def test_whitening_product(C, NT, nt):
    from livespikesorter_b200.sorter import Sorter
    g = torch.Generator().manual_seed(C)
    T, K = 8, 3
    W = torch.linalg.qr(torch.randn(nt, K, generator=g))[0].T.contiguous()
    U = torch.randn(T, K, C, generator=g)
    Wrot = torch.randn(C, C, generator=g)
    rows = np.random.default_rng(C).integers(-300, 300, (NT + 2 * nt, C)).astype(np.int16)
    s = Sorter(U=U, wPCA=W, ctc=torch.zeros(T, T, 2 * nt + 1), Wrot=Wrot, NT=NT, do_CAR=False, n_chan_bin=C)
    M = torch.eye(C)
    for drift in (False, True):
        if drift:
            M = M + 0.1 * torch.randn(C, C, generator=g)
            s.set_drift(M)
        X = s.filter(rows, 1, 3).cpu().double()
        raw = torch.from_numpy(rows).double().T
        A = M.double() @ Wrot.double()
        mean = raw.mean(1, keepdim=True)
        mag = (M.abs().double() @ Wrot.abs().double()) @ (raw.abs() + mean.abs())
        assert X.shape == raw.shape
        assert bool(((X - A @ (raw - mean)).abs() <= 1.01 * (2 * C + 2) * 2.0 ** -24 * mag).all())
