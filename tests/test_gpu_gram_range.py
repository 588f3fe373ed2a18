"""Stage (a) of statevectors whose norm^2 is at the ends of FP32's range: the
truncated target, relative to the norm, as at norm 1.  The capacity holds the
whole state; bound as for other random MPS (working precision over the n
projections and contractions, 4 n 2^-23, times a condition below 1e2)."""

import numpy as np
import pytest
import torch

from oracle import states as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norm", [1e-15, 1.0, 1.5e18, 1.7e19, 2.5e19])
@pytest.mark.parametrize("n", [4, 10, 16])
def test_target_at_any_norm(cuda_lib, n, norm):
    from qmprs_gb300 import engine
    eng = engine.engine()
    v = S.random_mps(n, 8, n)
    p = eng.plan([n], 1, 32)
    sv = torch.from_numpy((v * norm).astype(np.complex64).view(np.float32)).cuda()
    _, bonds, target = eng.stage_mps(p, sv, 32)
    assert int(bonds.cpu().max()) == min(8, 2 ** (n // 2))
    got = target.cpu().numpy().view(np.complex64).astype(complex) / norm
    assert np.linalg.norm(got - v) <= 4 * n * 2.0 ** -23 * 1e2
