"""The layer stage's cuts at their edges: a remainder of one row unit, of
exactly one (13 qubits) and of several (14 and 15), mixed batches, and
remainders of every width (rank-one cuts, two equal singular values).

Bounds: fidelities and reconstructions are gauge free.  A layer's overlap
moves by the relative rounding of the working state, which each of the n
projections and n gates leaves once: 2 n 2^-23 in complex64, 2 n 2^-44 in
double-float.  Two equal singular values leave the basis to rounding, so
only the first layer's overlap is compared there.
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


def _state(kind, n, seed):
    if kind == "mps":
        return S.random_mps(n, 6, seed)
    rng = np.random.default_rng(seed)
    v = np.ones(1, complex)
    if kind == "blocks":       # pairs of qubits: bonds 2 and 1 in turn
        for k in range(0, n, 2):
            w = 2 if k + 1 < n else 1
            v = np.kron(v, rng.standard_normal(2 ** w) + 1j * rng.standard_normal(2 ** w))
    else:                      # (|0..0> + |1..1>) / sqrt 2
        v = np.zeros(2 ** n, complex)
        v[0] = v[-1] = 1.0
    return v / np.linalg.norm(v)


@pytest.mark.parametrize("precision", ["fast", "exact"])
@pytest.mark.parametrize("kind", ["mps", "blocks", "ghz"])
@pytest.mark.parametrize("ns", [[2], [13], [14], [3, 15, 2, 14]])
def test_layers_at_unit_edges(eng, ns, kind, precision):
    exact = precision == "exact"
    L = 1 if kind == "ghz" else 2
    p = eng.plan(ns, L, 4, precision)
    states = [_state(kind, n, 7 + n) for n in ns]
    t = torch.from_numpy(np.concatenate(states).astype(p.npdtype).view(np.float64 if exact else np.float32)).cuda()
    gates, arity, nl, lf = eng.stage_layers(p, t, L, 1.0)
    got, ar = gates.cpu().numpy().view(np.complex128), arity.cpu().numpy()
    lf = lf.cpu().numpy().view(np.complex128).reshape(len(ns), L)
    for b, n in enumerate(ns):
        sv = states[b].astype(p.npdtype).astype(np.complex128)
        layers, fids = D.get_unitary_layers(sv, n, L, threshold=1.0)
        assert int(nl[b].cpu()) == len(fids)
        tol = 2 * n * (2.0 ** -44 if exact else 2.0 ** -23)
        for l, f in enumerate(fids):
            assert abs(abs(lf[b, l]) - abs(f)) <= tol * (l + 1), (n, l)
        # the first generated layer: its circuit state is the bond-2 truncation
        base = int(p.gate_off[b])
        blocks, gs, start = [], [], 0
        for s in range(n):
            k = int(ar[base // 16 + s])
            raw = got[base + s * 16: base + s * 16 + 4 ** k]
            gs.append(raw.reshape(2 ** k, 2 ** k))
            if k == 1:
                blocks.append((start, s, gs))
                start, gs = s + 1, []
        psi = D.circuit_state([blocks], n)
        assert abs(abs(np.vdot(psi, sv)) / np.linalg.norm(sv) - abs(fids[0])) <= tol


@pytest.mark.parametrize("precision", ["fast", "exact"])
@pytest.mark.parametrize("gap", [0.0, 1e-9, 1e-7, 1e-6, 1e-5, 1e-3])
def test_nearly_equal_singular_values(eng, gap, precision):
    """(|0..0> + (1 + gap) |1..1>) under a unitary on each qubit: bond two at
    every cut, so one layer prepares it to the working precision whichever
    basis the nearly equal singular values take."""
    exact = precision == "exact"
    ns = [2, 5, 13]
    p = eng.plan(ns, 1, 2, precision)
    rng = np.random.default_rng(17)
    states = []
    for n in ns:
        v = np.zeros([2] * n, complex)
        v[(0,) * n], v[(1,) * n] = 1.0, 1.0 + gap
        for k in range(n):
            u = np.linalg.qr(rng.standard_normal((2, 2)) + 1j * rng.standard_normal((2, 2)))[0]
            v = np.moveaxis(np.tensordot(u, v, (1, k)), 0, k)
        states.append(v.reshape(-1) / np.linalg.norm(v))
    t = torch.from_numpy(np.concatenate(states).astype(p.npdtype).view(np.float64 if exact else np.float32)).cuda()
    lf = eng.stage_layers(p, t, 1, 1.0)[3].cpu().numpy().view(np.complex128)
    for b, n in enumerate(ns):
        assert abs(abs(lf[b]) - 1.0) <= 2 * n * (2.0 ** -44 if exact else 2.0 ** -23), n
