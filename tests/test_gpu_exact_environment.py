"""The exact mode's environments summed to FP64: the gate of a sweep's first
step, the polar factor of an environment of 2^(n-1) products per entry, against
that of the environment in 80-bit sums.

Gates with entries of 0, (+-1 +- i) / 2 and their like make every amplitude of
the circuit state a power of two times a phase, exactly, and the target is
given in double-float, so products carry no rounding and only the sums do.  In
units of the environment's norm (about one: the target is near the circuit), a
thread's sums and the first two steps over a warp's lanes are double-float,
three roundings of 2^-49 per addition, independent between the 256, 128 and 64
sums of a block: 3 x 2^-49 (1/16 + 1/11 + 1/8) at most.  FP64 takes the rest,
and four of its units through the polar factor.  Together 2.4e-15 would be
reached if all added up; as independent parts, in the root mean square over
the states, 2^-49 is not.  A sum that is rounded to double-float at its end is
off by 2^-48 from that alone."""

import numpy as np
import pytest
import torch

from oracle import conventions as cv

pytestmark = pytest.mark.gpu

ROOT_X = np.array([[1 + 1j, 1 - 1j], [1 - 1j, 1 + 1j]]) / 2


def _double_float(x):
    hi = x.astype(np.complex64).astype(complex)
    return hi + (x - hi).astype(np.complex64).astype(complex)


def _phases(rng, m):
    return np.diag(1j ** rng.integers(0, 4, m))


@pytest.mark.parametrize("n,B", [(9, 96), (12, 64), (14, 48)])
def test_first_gate_of_a_sweep(cuda_lib, n, B):
    from qmprs_gb300 import engine
    eng = engine.engine()
    p = eng.plan([n] * B, 1, 4, "exact")
    store = np.zeros(p.gate_elems, complex)
    arity = np.full(p.gate_elems // 16, 2, np.int8)
    targets, want = [], []
    for b in range(B):
        rng = np.random.default_rng(1000 * n + b)
        gates = [_phases(rng, 4) @ np.kron(ROOT_X if q == 0 else np.eye(2), ROOT_X) for q in range(n - 1)]
        gates.append(_phases(rng, 2))
        x = np.zeros(2 ** n, complex)
        x[0] = 1
        for q, g in enumerate(gates[:-1]):
            x = np.einsum("ab,ibj->iaj", g, x.reshape(2 ** q, 4, -1)).reshape(-1)
        noise = rng.standard_normal(2 ** n) + 1j * rng.standard_normal(2 ** n)
        t = _double_float(np.einsum("ab,ib->ia", gates[-1], x.reshape(-1, 2)).reshape(-1)
                          + 0.3 * noise / np.linalg.norm(noise))
        env = np.einsum("ia,ib->ab", t.astype(np.clongdouble).reshape(-1, 2).conj(),
                        x.astype(np.clongdouble).reshape(-1, 2)).astype(complex)
        w, s = cv.polar_unitary_canonical(env, gates[-1].conj())
        want.append((w.conj(), s.sum()))
        targets.append(t)
        for q, g in enumerate(gates):
            off = int(p.gate_off[b]) + q * 16
            store[off: off + g.size] = g.reshape(-1)
        arity[off // 16] = 1
    dev = torch.from_numpy(store.view(np.float64)).cuda()
    t = torch.from_numpy(np.concatenate(targets).view(np.float64)).cuda()
    nl = torch.ones(B, dtype=torch.int32, device="cuda")
    eng.stage_sweeps(p, t, dev, torch.from_numpy(arity).cuda(), nl, 1)
    got = dev.cpu().numpy().view(complex)
    err = []
    for b, (w, s) in enumerate(want):
        off = int(p.gate_off[b]) + (n - 1) * 16
        err.append(np.max(np.abs(got[off: off + 4].reshape(2, 2) - w)) * s)
    rms = np.sqrt(np.mean(np.square(err)))
    assert rms <= 2.0 ** -49, rms
