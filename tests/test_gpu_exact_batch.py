"""The exact mode's truncation of a batch, its states side by side in one
launch per step: every state as it is alone, bit for bit, for batches of one
launch's states and of more (24 to a launch), of one size and of mixed ones."""

import numpy as np
import pytest
import torch

from oracle import states as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [[2, 4, 3], [7] * 24, [2, 9, 5, 6, 8, 3] * 5])
def test_batch_equals_single_states(cuda_lib, ns):
    from qmprs_gb300 import engine
    eng = engine.engine()
    chi = 6
    states = [S.random_mps(n, 9, 100 + i) for i, n in enumerate(ns)]
    states = [v / np.linalg.norm(v) for v in states]

    def run(ids):
        p = eng.plan([ns[i] for i in ids], 1, chi, "exact")
        sv = torch.from_numpy(np.concatenate([states[i] for i in ids]).view(np.float64)).cuda()
        t, bonds, target = eng.stage_mps(p, sv, chi)
        t, target = t.cpu().numpy().view(np.complex128), target.cpu().numpy().view(np.complex128)
        bh = bonds.cpu().numpy().reshape(len(ids), -1)
        out = []
        for k, i in enumerate(ids):
            n, ce, base = ns[i], p.chi_eff(k), int(p.tensor_off[k])
            bd = [int(x) for x in bh[k, : n + 1]]
            sites = [t[base + c * 2 * ce * ce:][: bd[c] * 2 * bd[c + 1]] for c in range(n)]
            out.append((bd, sites, target[int(p.vec_off[k]):][: 2 ** n]))
        return out

    batch = run(range(len(ns)))
    for i in range(len(ns)):
        alone = run([i])[0]
        assert alone[0] == batch[i][0]
        for a, b in zip(alone[1] + [alone[2]], batch[i][1] + [batch[i][2]]):
            assert np.array_equal(a.view(np.uint64), b.view(np.uint64)), i
