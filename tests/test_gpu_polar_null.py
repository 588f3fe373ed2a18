"""Rank-deficient environments in a sweep: the new gate's action on the null
space, which the sweep's fidelity does not see, is the unitary nearest to the
current gate's there.

A sweep's first two steps (the last site's 2 x 2 gate, its neighbour's 4 x 4
one) against the oracle's rule.  The rank comes from the target (truncated to
Schmidt rank k between the two last qubits and the rest, or 1 between the last
and the rest) or from fresh |0> qubits (one layer on two or three qubits).

Bound: an environment is off by delta = 3 G eps of the vectors' norms (an
amplitude passes each of the G gates at most three times; eps is 2^-22 in the
fast mode, 2^-44 in the exact one).  With s the smallest singular value that
counts and x that of the current gate's component on the null space, the
factor moves by delta / s, the null space by delta / s, and the completion by
that over x, once for each of its three factors.  States with s below 0.05 or
x below 0.1 have no unique gate at that accuracy and are left out."""

import numpy as np
import pytest
import torch

from oracle import conventions as cv
from oracle import dense as D

pytestmark = pytest.mark.gpu


def _unitary(rng, m):
    q, r = np.linalg.qr(rng.standard_normal((m, m)) + 1j * rng.standard_normal((m, m)))
    return q * (np.diag(r) / np.abs(np.diag(r)))


def _condition(env, prev):
    """Smallest significant singular value, and that of (I - U U^H) W V_N."""
    u, s, vh = np.linalg.svd(env)
    k = int(np.sum(s > cv.POLAR_NULL_TOL * s[0]))
    if k == len(s):
        return k, s[-1], 1.0
    x = prev @ vh[k:].conj().T
    x = x - u[:, :k] @ (u[:, :k].conj().T @ x)
    return k, s[k - 1], np.linalg.svd(x)[1][-1]


@pytest.mark.parametrize("precision", ["fast", "exact"])
@pytest.mark.parametrize("n,L,cut,rank", [(6, 2, 2, 1), (6, 2, 2, 2), (6, 2, 2, 3), (6, 2, 1, 1),
                                          (2, 1, 0, 1), (3, 1, 0, 2)])
def test_completion_follows_the_gate(cuda_lib, n, L, cut, rank, precision):
    from qmprs_gb300 import engine
    eng = engine.engine()
    B = 24
    p = eng.plan([n] * B, L, 4, precision)
    store = np.zeros(p.gate_elems, complex)
    arity = np.zeros(p.gate_elems // 16, np.int8)
    targets, steps = [], []
    for b in range(B):
        rng = np.random.default_rng(50 * n + b)
        layers = [[(0, n - 1, [_unitary(rng, 4) for _ in range(n - 1)] + [_unitary(rng, 2)])] for _ in range(L)]
        t = D.circuit_state(layers, n) + 0.2 * (rng.standard_normal(2 ** n) + 1j * rng.standard_normal(2 ** n)) / 2 ** (n / 2)
        if cut:
            u, s, vh = np.linalg.svd(t.reshape(-1, 2 ** cut), full_matrices=False)
            t = ((u[:, :rank] * s[:rank]) @ vh[:rank]).reshape(-1)
        t = (t / np.linalg.norm(t)).astype(p.npdtype)
        targets.append(t)
        for l, layer in enumerate(reversed(layers)):
            for q, g in enumerate(layer[0][2]):
                off = int(p.gate_off[b]) + (l * n + q) * 16
                store[off: off + g.size] = g.reshape(-1)
                arity[off // 16] = 1 if q == n - 1 else 2
        psi, tt = D.circuit_state(layers, n), t.astype(complex)
        for q in (n - 1, n - 2):
            g = layers[-1][0][2][q]
            psi = D.apply_gate(psi, n, g.conj().T, q)
            env = D.environment(tt, psi, n, q, 1 if q == n - 1 else 2)
            w, _ = cv.polar_unitary_canonical(env, g.conj())
            steps.append((b, q, w.conj(), *_condition(env, g.conj())))
            tt = D.apply_gate(tt, n, w.T, q)
    dev = torch.from_numpy(store.view(np.float64)).cuda()
    t = torch.from_numpy(np.concatenate(targets).view(np.float64 if precision == "exact" else np.float32)).cuda()
    nl = torch.full((B,), L, dtype=torch.int32, device="cuda")
    eng.stage_sweeps(p, t, dev, torch.from_numpy(arity).cuda(), nl, 1)
    got = dev.cpu().numpy().view(complex)
    delta = 3 * n * L * 2.0 ** (-44 if precision == "exact" else -22)
    deficient = n - 1 if cut == 1 else n - 2
    seen = 0
    usable = {b: True for b in range(B)}
    for b, q, want, k, s, x in steps:
        usable[b] = usable[b] and s > 0.05 and x > 0.1
        if not usable[b]:
            continue
        off = int(p.gate_off[b]) + q * 16
        u = got[off: off + want.size].reshape(want.shape)
        bound = delta / s * (1 + 3 / x)
        if q == n - 2:      # the target already carries the first step's gate
            bound *= 2
        assert np.max(np.abs(u - want)) <= bound, (b, q, k, s, x)
        if q == deficient:
            assert k == rank
            seen += 1
    assert seen >= B // 4
