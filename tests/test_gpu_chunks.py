"""The tile passes over chunks of every length the plan picks: one tile per
chunk (a few tiles), two, four, eight, three (a last chunk of two), and several
states sharing a launch.

Every gate's environment against the oracle.  An environment is a sum of
products of amplitudes that passed each gate at most twice through
split-FP16 products (2^-21 each, FP32 accumulation), bounded in the
Frobenius norm over all gates by 2 G 2^-21 of the largest's norm; a random
target's overlap is small, so the bound is taken against |t| = 1.
"""

import numpy as np
import pytest
import torch

from oracle import dense as D

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng(cuda_lib):
    from qmprs_gb300 import engine
    return engine.engine()


def _unitary(rng, m):
    q, r = np.linalg.qr(rng.standard_normal((m, m)) + 1j * rng.standard_normal((m, m)))
    return q * (np.diag(r) / np.abs(np.diag(r)))


@pytest.mark.parametrize("ns", [[14], [15, 12, 11, 3], [20], [21, 16], [22], [16] * 40])
def test_environments_over_chunk_lengths(eng, ns):
    L = 1
    rng = np.random.default_rng(sum(ns))
    p = eng.plan(ns, L, 4)
    store = np.zeros(p.gate_elems, complex)
    arity = np.zeros(p.gate_elems // 16, np.int8)
    layers, targets = [], []
    for b, n in enumerate(ns):
        gs = [_unitary(rng, 4) for _ in range(n - 1)] + [_unitary(rng, 2)]
        layers.append([[(0, n - 1, gs)]])
        t = D.circuit_state(layers[b], n)
        z = rng.standard_normal(2 ** n) + 1j * rng.standard_normal(2 ** n)
        t = t + z / np.linalg.norm(z)
        targets.append((t / np.linalg.norm(t)).astype(np.complex64))
        for s, g in enumerate(gs):
            off = int(p.gate_off[b]) + s * 16
            store[off: off + g.size] = g.reshape(-1)
            arity[off // 16] = 1 if s == n - 1 else 2
    gates = torch.from_numpy(store.view(np.float64)).cuda()
    ar = torch.from_numpy(arity).cuda()
    nl = torch.full((len(ns),), L, dtype=torch.int32, device="cuda")
    t = torch.from_numpy(np.concatenate(targets).view(np.float32)).cuda()
    env = eng.environments(p, t, gates, ar, nl).cpu().numpy().view(np.complex128)
    for b, n in enumerate(ns):
        want = D.environments(targets[b].astype(np.complex128), n, layers[b])
        for s, e in enumerate(want):
            off = int(p.gate_off[b]) + s * 16
            got = env[off: off + e.size].reshape(e.shape)
            assert np.linalg.norm(got - e) <= 2 * n * L * 2.0 ** -21, (n, s)
