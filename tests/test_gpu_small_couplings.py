"""Stage (a) on states whose Grams are diagonal but for equal couplings among
small eigenvalues: k vectors of weight eps^2 each that belong to one singular
vector of weight k^2 eps^2, below FP32's resolution of the Gram and above the
1e-10 truncation cutoff.

The amplitude matrix between the two halves is diag(1 x m) and a k x k block of
eps, so the bonds are those of m + 1 singular vectors, where the k unresolved
ones would make m + k of them, or at a capacity of m + 1 lose all but one.
Bound of the target: a state of bond m + 1 is kept whole, so what is left is
the working precision's rounding of the n projections and contractions, 4 n
2^-23 (fast) or 4 n 2^-44 (exact), and per cut the amplitude g / sigma that a
coupling g at the rotations' floor (1e-13 or 1e-15 of the trace) takes from a
kept value sigma, which the cutoff keeps above 1e-5."""

import numpy as np
import pytest
import torch

from oracle import dense as D

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng(cuda_lib):
    from qmprs_gb300 import engine
    return engine.engine()


@pytest.mark.parametrize("precision", ["fast", "exact"])
@pytest.mark.parametrize("eps", [2e-5, 1e-4, 3e-4])
@pytest.mark.parametrize("n,m,k", [(4, 1, 2), (6, 1, 3), (8, 4, 5), (10, 8, 9), (12, 20, 11)])
def test_equal_small_couplings(eng, n, m, k, eps, precision):
    half = n // 2
    a = np.zeros((2 ** half, 2 ** half), complex)
    a[range(m), range(m)] = 1.0
    a[m: m + k, m: m + k] = eps
    v = (a / np.linalg.norm(a)).reshape(-1)
    for chi in (m + 1, 2 ** half):
        p = eng.plan([n], 1, chi, precision)
        sv = v.astype(p.npdtype)
        dev = torch.from_numpy(sv.view(np.float64 if precision == "exact" else np.float32)).cuda()
        _, bonds, target = eng.stage_mps(p, dev, chi)
        ref = D.tt_svd_right(sv.astype(complex), n, chi)
        assert [int(x) for x in bonds.cpu().numpy()[1:n]] == [t.shape[0] for t in ref[1:]], chi
        got = target.cpu().numpy().view(p.npdtype)
        rounding, floor = (2.0 ** -44, 1e-15) if precision == "exact" else (2.0 ** -23, 1e-13)
        assert np.linalg.norm(got - D.mps_to_dense(ref)) <= 4 * n * rounding + n * floor / 1e-5
