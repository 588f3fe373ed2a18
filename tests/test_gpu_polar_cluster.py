"""The grouped sweep's polar kernel where the blocks of a cluster share the
sum over a state's chunks: 64, 128 and 256 chunks (two, four, eight blocks),
one state and two of different sizes.

One group's steps on a state at its fixed point: the target is the circuit's
own state, so every environment's polar factor is the gate that is there and
a sweep's fidelity is one.  An environment sums 2^n products that passed each
gate at most twice through split-FP16 products (2^-21 each): G 2^-20."""

import numpy as np
import pytest
import torch

from oracle import dense as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [[17], [18], [19], [20], [18, 13]])
def test_fixed_point(cuda_lib, ns):
    from qmprs_gb300 import engine
    eng = engine.engine()
    L = 1
    rng = np.random.default_rng(sum(ns))
    p = eng.plan(ns, L, 4)
    store = np.zeros(p.gate_elems, complex)
    arity = np.zeros(p.gate_elems // 16, np.int8)
    targets = []
    for b, n in enumerate(ns):
        gs = []
        for s in range(n):
            m = 4 if s < n - 1 else 2
            q, r = np.linalg.qr(rng.standard_normal((m, m)) + 1j * rng.standard_normal((m, m)))
            gs.append(q * (np.diag(r) / np.abs(np.diag(r))))
            off = int(p.gate_off[b]) + s * 16
            store[off: off + m * m] = gs[-1].reshape(-1)
            arity[off // 16] = 1 if s == n - 1 else 2
        targets.append(D.circuit_state([[(0, n - 1, gs)]], n).astype(np.complex64))
    gates = torch.from_numpy(store.view(np.float64)).cuda()
    ar = torch.from_numpy(arity).cuda()
    nl = torch.full((len(ns),), L, dtype=torch.int32, device="cuda")
    t = torch.from_numpy(np.concatenate(targets).view(np.float32)).cuda()
    fid, _ = eng.stage_sweeps(p, t, gates, ar, nl, 1)
    fid = fid.cpu().numpy().reshape(len(ns), -1)
    for b, n in enumerate(ns):
        assert abs(fid[b, 0] - 1.0) <= n * 2.0 ** -20, n
    new = gates.cpu().numpy().view(np.complex128)
    for b, n in enumerate(ns):
        gs = []
        for s in range(n):
            m = 4 if s < n - 1 else 2
            off = int(p.gate_off[b]) + s * 16
            gs.append(new[off: off + m * m].reshape(m, m))
        got = D.circuit_state([[(0, n - 1, gs)]], n)
        assert abs(np.vdot(got, targets[b].astype(np.complex128))) >= 1.0 - n * 2.0 ** -20, n


@pytest.mark.parametrize("ns", [[14], [20], [15, 12, 11, 3], [16] * 40, [21, 16]])
def test_passes_repeat_bit_for_bit(cuda_lib, ns):
    """Passes and polar kernels start while their predecessor runs: two runs
    of two sweeps on the same inputs give the same bits, with states that
    stop after the first (an exact target) and states that go on."""
    from qmprs_gb300 import engine
    eng = engine.engine()
    L = 2
    rng = np.random.default_rng(len(ns))
    p = eng.plan(ns, L, 4)
    store = np.zeros(p.gate_elems, complex)
    arity = np.zeros(p.gate_elems // 16, np.int8)
    for b, n in enumerate(ns):
        for i in range(L * n):
            m = 2 if (i + 1) % n == 0 else 4
            q = np.linalg.qr(rng.standard_normal((m, m)) + 1j * rng.standard_normal((m, m)))[0]
            off = int(p.gate_off[b]) + i * 16
            store[off: off + m * m] = q.reshape(-1)
            arity[off // 16] = 1 if m == 2 else 2
    ar = torch.from_numpy(arity).cuda()
    nl = torch.full((len(ns),), L, dtype=torch.int32, device="cuda")
    g0 = torch.from_numpy(store.view(np.float64)).cuda()
    t = eng.stage_circuit(p, g0, ar, nl)
    z = torch.randn(t.shape, dtype=t.dtype, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    for b, n in enumerate(ns):
        if b % 2:   # away from the circuit's own state
            lo = 2 * int(p.vec_off[b])
            v = t[lo: lo + 2 ** (n + 1)] + z[lo: lo + 2 ** (n + 1)] * 2.0 ** (-n / 2)
            t[lo: lo + 2 ** (n + 1)] = v / torch.linalg.norm(v)
    out = []
    for _ in range(3):
        g = g0.clone()
        fid, done = eng.stage_sweeps(p, t, g, ar, nl, 2, 1.0 - 1e-4)
        out.append((g.cpu().numpy(), fid.cpu().numpy(), done.cpu().numpy()))
    for o in out[1:]:
        for a, b in zip(out[0], o):
            assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
