"""Stage (a) of states of up to 10 qubits: the truncated target to its storage's
rounding.

The capacity holds the whole state, so the target is the state up to the
rounding of n - 1 projected remainders and n - 1 contracted ones and of the
vectors they are multiplied with, each entry uniform within half a unit of
complex64 (2^-24 / sqrt(3) of it, root mean square) and independent:
2^-24 / sqrt(3) sqrt(4 (n - 1)) of the norm, as root mean square over the
states.  FP32 accumulation over the bond adds as much again and more."""

import numpy as np
import pytest
import torch

from oracle import states as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [6, 8, 9, 10])
def test_target_is_the_state(cuda_lib, n):
    from qmprs_gb300 import engine
    eng = engine.engine()
    B = 12
    states = [S.uniform_complex(n, 300 + b).astype(np.complex64) for b in range(B)]
    p = eng.plan([n] * B, 1, 2 ** (n // 2))
    sv = torch.from_numpy(np.concatenate(states).view(np.float32)).cuda()
    _, _, target = eng.stage_mps(p, sv, 2 ** (n // 2))
    got = target.cpu().numpy().view(np.complex64).astype(complex)
    err = [np.linalg.norm(got[o: o + 2 ** n] - v) for o, v in zip(p.vec_off, states)]
    assert np.sqrt(np.mean(np.square(err))) <= 2.0 ** -24 / np.sqrt(3) * np.sqrt(4 * (n - 1))
