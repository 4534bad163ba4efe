"""Scores over template lengths around the 64 taps that the projection takes from its kernel's arguments and all
component counts, against FP64.

B[t, s] = sum_{k, c} U[t, k, c] sum_m wPCA[k, m] X[c, s + m - nt/2]. Tolerance: every score sums C K products of a
projection (nt FMAs, each rounded once) with a template value in 3xTF32 (each product to 2^-21, the sum in FP32), so
|error| <= (nt + C K + 16) 2^-23 of the sum of the absolute terms, twice what the roundings above can add up to.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nt', [5, 41, 55, 57, 61, 63, 65, 81])
@pytest.mark.parametrize('K', [1, 2, 3, 4, 5, 6, 7, 8])
def test_scores_against_fp64(K, nt):
    from livespikesorter_b200.sorter import Sorter
    C, T, NT = 33, 20, 700
    g = torch.Generator().manual_seed(100 * K + nt)
    U, W = torch.randn(T, K, C, generator=g), torch.randn(K, nt, generator=g)
    X = torch.randn(C, NT + 2 * nt, generator=g)
    s = Sorter(U=U, wPCA=W, ctc=torch.zeros(T, T, 2 * nt + 1), Wrot=torch.eye(C), NT=NT)
    B = s.scores(X.cuda()).cpu().double()

    def scores(U, W, X):
        P = torch.nn.functional.conv1d(X.double()[:, None], W.double()[:, None], padding=nt // 2)   # [C, K, N]
        return torch.einsum('tkc,ckn->tn', U.double(), P)

    bound = (nt + C * K + 16) * 2.0 ** -23 * scores(U.abs(), W.abs(), X.abs())
    assert bool(((B - scores(U, W, X)).abs() <= bound).all())
