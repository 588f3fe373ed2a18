"""Stage (a)'s one-block eigensolver at Gram widths 2 to 64, odd bonds and
rank-deficient cuts among them: bonds as the oracle's, right-isometric site
tensors, the truncated target.

Bounds: the vectors are orthonormal to the double-float products' rounding,
w 2^-44 an entry.  The target's error is the working precision's rounding
over the n projections and contractions, 4 n 2^-23 (fast) or 4 n 2^-44
(exact), times the condition of a random MPS's kept spectrum (below 1e2).
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


@pytest.mark.parametrize("precision", ["fast", "exact"])
@pytest.mark.parametrize("n,bonds,chi", [(2, [1, 2], 4), (5, [3], 3), (11, [1, 3, 5, 7], 16),
                                         (12, [21, 31, 32], 32), (13, [17, 32, 29], 24), (16, [4, 9], 8),
                                         (9, [9, 11, 12], 12)])
def test_sites_and_target(eng, n, bonds, chi, precision):
    exact = precision == "exact"
    states = [S.random_mps(n, bd, 11 * n + bd) for bd in bonds]
    p = eng.plan([n] * len(bonds), 1, chi, precision)
    sv = torch.from_numpy(np.concatenate(states).astype(p.npdtype).view(np.float64 if exact else np.float32)).cuda()
    tensors, bd_dev, target = eng.stage_mps(p, sv, chi)
    ts = tensors.cpu().numpy().view(np.complex128)
    bh = bd_dev.cpu().numpy().reshape(len(bonds), -1)
    tv = target.cpu().numpy().view(p.npdtype)
    for b in range(len(bonds)):
        v = states[b].astype(p.npdtype).astype(np.complex128)
        ref = D.tt_svd_right(v, n, chi)
        assert [int(x) for x in bh[b, 1:n]] == [t.shape[0] for t in ref[1:]]
        ce, base = p.chi_eff(b), int(p.tensor_off[b])
        for s in range(1, n):
            l, r = int(bh[b, s]), int(bh[b, s + 1])
            off = base + s * 2 * ce * ce
            m = ts[off: off + l * 2 * r].reshape(l, 2 * r)
            assert np.max(np.abs(m @ m.conj().T - np.eye(l))) <= 2 * r * 2.0 ** -44, s
        got = tv[p.vec_off[b]: p.vec_off[b] + 2 ** n]
        tol = 4 * n * (2.0 ** -44 if exact else 2.0 ** -23) * 1e2
        assert np.linalg.norm(got - D.mps_to_dense(ref)) <= tol


@pytest.mark.parametrize("kind", ["rank_one", "two_blocks", "flat"])
@pytest.mark.parametrize("n,chi", [(4, 4), (8, 12), (10, 20), (11, 32)])
def test_spectra_at_padded_widths(eng, n, chi, kind):
    """Spectra the Jacobi sweeps meet at their edges: nothing to rotate, an
    exact block structure with zero entries, all eigenvalues equal up to
    rounding.  The bonds are within the capacity, so the target is the state
    itself; the bound is test_sites_and_target's."""
    rng = np.random.default_rng(n)
    if kind == "rank_one":
        v = np.ones(1)
        for _ in range(n):
            v = np.kron(v, rng.standard_normal(2) + 1j * rng.standard_normal(2))
    elif kind == "two_blocks":   # (|0>|a> + |1>|b>) |0> |c>, a and b product states
        a, b, c = np.ones(1), np.ones(1), np.ones(1)
        for _ in range((n - 2) // 2):
            a, b, c = (np.kron(x, rng.standard_normal(2) + 1j * rng.standard_normal(2)) for x in (a, b, c))
        rest = n - 2 - (n - 2) // 2 * 2
        v = np.kron(np.kron(np.concatenate([a, b]), [1.0, 0.0]), np.kron(c, [1.0] + [0.0] * (2 ** rest - 1)))
    else:   # pairs (q, q + k) maximally entangled, k < chi's bits
        k = int(np.log2(chi))
        v = np.zeros([2] * n)
        for bits in range(2 ** k):
            idx = [0] * n
            for j in range(k):
                idx[j] = idx[n - k + j] = (bits >> j) & 1
            v[tuple(idx)] = 1.0
        v = v.reshape(-1).astype(complex)
    v = v / np.linalg.norm(v)
    p = eng.plan([n], 1, chi, "fast")
    v32 = v.astype(p.npdtype)
    _, bd, target = eng.stage_mps(p, torch.from_numpy(v32.view(np.float32)).cuda(), chi)
    assert int(bd.cpu().max()) <= (1 if kind == "rank_one" else 2 if kind == "two_blocks" else chi)
    got = target.cpu().numpy().view(p.npdtype)
    assert np.linalg.norm(got - v32) <= 4 * n * 2.0 ** -23 * 1e2


@pytest.mark.parametrize("kind", ["mps", "mixture"])
@pytest.mark.parametrize("n,chi", [(6, 8), (9, 9), (12, 20), (13, 32)])
def test_exact_finish(eng, n, chi, kind):
    """The exact mode's FP64 finish on spectra it takes in one step and on
    decaying ones that go on to FP64 sweeps: right-isometric sites, and kept
    weight as the oracle's.  Bounds: isometry as in test_sites_and_target; the
    kept weight moves by the square of the vectors' error, so by the rounding
    of its sum, 2^n terms at 2^-44."""
    v = S.random_mps(n, 8, n) if kind == "mps" else S.gaussian_mixture(n, n)
    v = (v / np.linalg.norm(v)).astype(complex)
    p = eng.plan([n], 1, chi, "exact")
    tensors, bonds, target = eng.stage_mps(p, torch.from_numpy(v.view(np.float64)).cuda(), chi)
    t, tv = tensors.cpu().numpy().view(np.complex128), target.cpu().numpy().view(np.complex128)
    bd = [int(x) for x in bonds.cpu().numpy()[: n + 1]]
    ce, base = p.chi_eff(0), int(p.tensor_off[0])
    for c in range(1, n):
        keep, w = bd[c], 2 * bd[c + 1]
        m = t[base + c * 2 * ce * ce:][: keep * w].reshape(keep, w)
        assert np.max(np.abs(m @ m.conj().T - np.eye(keep))) <= w * 2.0 ** -44, c
    ref = D.mps_to_dense(D.tt_svd_right(v, n, chi))
    assert abs(abs(np.vdot(tv, v)) - abs(np.vdot(ref, v))) <= 2 ** (n / 2) * 2.0 ** -44
