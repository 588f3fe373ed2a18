"""Stage (a)'s one-block eigensolver at Gram widths 2 to 64, odd bonds and
rank-deficient cuts among them: bonds as the oracle's, right-isometric site
tensors, the truncated target.

Bounds: the vectors are orthonormal to the double-float products' rounding,
w 2^-44 an entry.  The target's error is the working precision's rounding
over the n projections and contractions, 4 n 2^-23 (fast) or 4 n 2^-44
(exact), times the condition of a random MPS's kept spectrum (below 1e2).
"""

import numpy as np
import pytest
import torch

from oracle import dense as D
from oracle import states as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng(cuda_lib):
    from qmprs_gb300 import engine
    return engine.engine()


@pytest.mark.parametrize("precision", ["fast", "exact"])
@pytest.mark.parametrize("n,bonds,chi", [(2, [1, 2], 4), (5, [3], 3), (11, [1, 3, 5, 7], 16),
                                         (12, [21, 31, 32], 32), (13, [17, 32, 29], 24), (16, [4, 9], 8)])
def test_sites_and_target(eng, n, bonds, chi, precision):
    exact = precision == "exact"
    states = [S.random_mps(n, bd, 11 * n + bd) for bd in bonds]
    p = eng.plan([n] * len(bonds), 1, chi, precision)
    sv = torch.from_numpy(np.concatenate(states).astype(p.npdtype).view(np.float64 if exact else np.float32)).cuda()
    tensors, bd_dev, target = eng.stage_mps(p, sv, chi)
    ts = tensors.cpu().numpy().view(np.complex128)
    bh = bd_dev.cpu().numpy().reshape(len(bonds), -1)
    tv = target.cpu().numpy().view(p.npdtype)
    for b in range(len(bonds)):
        v = states[b].astype(p.npdtype).astype(np.complex128)
        ref = D.tt_svd_right(v, n, chi)
        assert [int(x) for x in bh[b, 1:n]] == [t.shape[0] for t in ref[1:]]
        ce, base = p.chi_eff(b), int(p.tensor_off[b])
        for s in range(1, n):
            l, r = int(bh[b, s]), int(bh[b, s + 1])
            off = base + s * 2 * ce * ce
            m = ts[off: off + l * 2 * r].reshape(l, 2 * r)
            assert np.max(np.abs(m @ m.conj().T - np.eye(l))) <= 2 * r * 2.0 ** -44, s
        got = tv[p.vec_off[b]: p.vec_off[b] + 2 ** n]
        tol = 4 * n * (2.0 ** -44 if exact else 2.0 ** -23) * 1e2
        assert np.linalg.norm(got - D.mps_to_dense(ref)) <= tol
