"""The blocked eigensolver where a sweep has few rounds: Gram widths 66 to
130, padded to 3 to 5 subproblems, of flat and of decaying spectra.

Bounds: the refinement repeats until its last correction is below 1e-4, and
a step squares the error: vectors to 1e-8, summed over up to 65 columns;
the truncated target additionally carries the working precision's rounding
of the n projections and contractions, 4 n 2^-23 times the condition of the
kept spectrum (below 1e2)."""

import numpy as np
import pytest
import torch

from oracle import dense as D
from oracle import states as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["flat", "mixture", "mps"])
@pytest.mark.parametrize("n,chi", [(13, 33), (13, 47), (14, 65)])
def test_few_rounds(cuda_lib, n, chi, kind):
    from qmprs_gb300 import engine
    eng = engine.engine()
    sv = (S.uniform_complex(n, 5) if kind == "flat" else S.gaussian_mixture(n, 5) if kind == "mixture"
          else S.random_mps(n, chi, 5))
    p, svd = eng.upload([sv], 1, chi)
    before = eng.wide_stats(p)["grams"]
    tensors, bonds, target = eng.stage_mps(p, svd, chi)
    torch.cuda.synchronize()
    assert eng.wide_stats(p)["grams"] > before
    v = sv.astype(np.complex64).astype(np.complex128)
    ref = D.mps_to_dense(D.tt_svd_right(v / np.linalg.norm(v), n, chi)) * np.linalg.norm(v)
    got = target.cpu().numpy().view(np.complex64).astype(np.complex128)
    # compared with the truncation error's own weight: which vectors of a
    # close pair are dropped moves the target by at most their difference
    assert abs(np.vdot(got, v)) >= abs(np.vdot(ref, v)) * (1 - 4 * n * 2.0 ** -23 * 1e2)
    bd = [int(x) for x in bonds.cpu().numpy()[: n + 1]]
    ce, base = p.chi_eff(0), int(p.tensor_off[0])
    t = tensors.cpu().numpy().view(np.complex128)
    for c in range(1, n):
        keep, w = bd[c], 2 * bd[c + 1]
        a = t[base + c * 2 * ce * ce: base + c * 2 * ce * ce + keep * w].reshape(keep, w)
        assert np.max(np.abs(a @ a.conj().T - np.eye(keep))) <= 65 * 1e-8, (c, keep, w)
