"""The exact mode's layer Grams to FP64: the gate of the last site, whose columns
are the eigenvectors of the first cut's 2 x 2 Gram, against those of the Gram
in 80-bit sums.

Amplitudes are given in double-float, so both sides start from the same
numbers.  The Gram's entries are sums of 2^(n-1) products that FP64 would round
last, and an entry's error over the eigenvalues' difference turns the vectors.
Bound, root mean square over the states: the error times the difference (in
units of the trace) is one unit of FP64, 2^-52: the roundings of the entries,
of the products with the vectors and of the vectors themselves, 2^-53 each and
independent.  Sums over a warp's lanes in double-float, or entries rounded to
it, are off by more."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _double_float(x):
    hi = x.astype(np.complex64).astype(complex)
    return hi + (x - hi).astype(np.complex64).astype(complex)


def _eigenvectors(g):
    """Of a 2 x 2 Hermitian matrix (closed form, in its precision): columns by
    descending eigenvalue, the first of the largest entries positive; and the
    eigenvalues' difference over their sum."""
    a, d, c = g[0, 0].real, g[1, 1].real, g[0, 1]
    h = (a - d) / 2
    r = np.sqrt(h * h + abs(c) ** 2)
    v = np.array([c, r - h]) if h < 0 else np.array([r + h, np.conj(c)])
    v = v / np.sqrt((abs(v) ** 2).sum())
    out = np.stack([v, [-np.conj(v[1]), np.conj(v[0])]], axis=1)
    for k in range(2):
        mag = np.abs(out[:, k])
        z = out[int(np.nonzero(mag >= (1 - 1e-6) * mag.max())[0][0]), k]
        out[:, k] *= np.conj(z) / abs(z)
    return out, float(2 * r / (a + d))


@pytest.mark.parametrize("n,B", [(8, 256), (10, 192), (12, 128)])
def test_last_sites_gate(cuda_lib, n, B):
    from qmprs_gb300 import engine
    eng = engine.engine()
    p = eng.plan([n] * B, 1, 2, "exact")
    states = []
    for b in range(B):
        rng = np.random.default_rng(100 * n + b)
        m = rng.standard_normal((2 ** (n - 1), 2)) + 1j * rng.standard_normal((2 ** (n - 1), 2))
        m = m @ np.array([[1.0, 0.4], [0.0, 0.5]])
        states.append(_double_float(m.reshape(-1) / np.linalg.norm(m)))
    sv = torch.from_numpy(np.concatenate(states).view(np.float64)).cuda()
    gates = eng.stage_layers(p, sv, 1, 1 - 1e-6)[0].cpu().numpy().view(complex)
    err = []
    for b, v in enumerate(states):
        m = v.astype(np.clongdouble).reshape(-1, 2)
        want, gap = _eigenvectors(m.conj().T @ m)
        off = int(p.gate_off[b]) + (n - 1) * 16
        err.append(float(np.max(np.abs(gates[off: off + 4].reshape(2, 2) - want.conj()))) * gap)
    rms = np.sqrt(np.mean(np.square(err)))
    assert rms <= 2.0 ** -52, rms
