"""The sweep's polar factor by one warp, at the environments where it can go
wrong: 2 x 2 and 4 x 4, of full rank, rank deficient (fresh |0> inputs), of
rank one (product targets) and zero (a target orthogonal to the circuit).

Bounds: in the fast mode an amplitude passes each of the G gates at most
three times (rebuild, peel, target) at a relative rounding of at most 2^-22
(complex FP32 products; the split-FP16 products of states above 13 qubits
2^-20 with their accumulation), so a sweep's fidelity is within 3 G times
that of the oracle's; the new gates are unitary to FP64 rounding.  The exact
mode's double-float products round at 2^-44 and its gates are compared too,
where no choice of a null direction is left to rounding.
"""

import copy

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


def _layers(rng, n, L, kind):
    """Layers in circuit order."""
    out = []
    for _ in range(L):
        gates = [np.eye(4, dtype=complex) if kind == "zero" else _unitary(rng, 4) for _ in range(n - 1)]
        gates.append(np.eye(2, dtype=complex) if kind == "zero" else _unitary(rng, 2))
        out.append([(0, n - 1, gates)])
    return out


def _target(rng, n, kind):
    if kind == "zero":          # identity gates, a target without |0...0>
        t = np.zeros(2 ** n, complex)
        t[-1] = 1.0
        return t
    if kind == "product":
        t = np.ones(1, complex)
        for _ in range(n):
            t = np.kron(t, rng.standard_normal(2) + 1j * rng.standard_normal(2))
    else:
        t = rng.standard_normal(2 ** n) + 1j * rng.standard_normal(2 ** n)
    return t / np.linalg.norm(t)


@pytest.mark.parametrize("kind", ["random", "product", "zero"])
@pytest.mark.parametrize("ns", [[2], [3, 2, 4], [5, 13], [4, 14]])
@pytest.mark.parametrize("precision", ["fast", "exact"])
def test_sweep_gates_and_fidelity(eng, ns, kind, precision):
    L = 2
    exact = precision == "exact"
    rng = np.random.default_rng(100 + sum(ns))
    p = eng.plan(ns, L, 4, precision)
    store = np.zeros(p.gate_elems, complex)
    arity = np.zeros(p.gate_elems // 16, np.int8)
    layers, targets = [], []
    for b, n in enumerate(ns):
        layers.append(_layers(rng, n, L, kind))
        targets.append(_target(rng, n, kind).astype(p.npdtype))
        for l, layer in enumerate(reversed(layers[b])):
            for s, g in enumerate(layer[0][2]):
                off = int(p.gate_off[b]) + (l * n + s) * 16
                store[off: off + g.size] = g.reshape(-1)
                arity[off // 16] = 1 if s == n - 1 else 2
    gates = torch.from_numpy(store.view(np.float64)).cuda()
    ar = torch.from_numpy(arity).cuda()
    nl = torch.full((len(ns),), L, dtype=torch.int32, device="cuda")
    t = torch.from_numpy(np.concatenate(targets).view(np.float64 if exact else np.float32)).cuda()
    sf, sd = eng.stage_sweeps(p, t, gates, ar, nl, 1)
    got = gates.cpu().numpy().view(np.complex128)
    assert np.all(sd.cpu().numpy() == 1)
    for b, n in enumerate(ns):
        ref, f = D.sweep(targets[b].astype(np.complex128), n, copy.deepcopy(layers[b]))
        eps = 2.0 ** -44 if exact else 2.0 ** -20 if max(ns) > 13 else 2.0 ** -22
        assert abs(float(sf[b].cpu()) - f) <= 3 * n * L * eps, (n, kind)
        for i in range(L * n):
            m = 2 if (i + 1) % n == 0 else 4
            off = int(p.gate_off[b]) + i * 16
            u = got[off: off + m * m].reshape(m, m)
            assert np.max(np.abs(u @ u.conj().T - np.eye(m))) < 1e-13
            if exact and kind == "random":
                want = ref[L - 1 - i // n][0][2][i % n]
                assert np.max(np.abs(u - want)) < 1e-8
