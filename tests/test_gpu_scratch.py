"""Stage (a)'s scratch in a batch of small states with one large one.

Per state it holds the Gram partials, eight of the widest Gram a plan can have
(128 wide: 2 MB), and three matrices of that width (0.75 MB).  More partials,
one per tile, are for the states that have the tiles: at most 1216 blocks take
one 64-wide partial (64 KB) each, 76 MB for a whole batch.  32 MB are allowed
for the allocator's granularity and for kernels loaded on first use."""

import pytest
import torch

pytestmark = pytest.mark.gpu

MB = 2 ** 20


@pytest.mark.parametrize("ns", [[8] * 400, [8] * 400 + [20], [9] * 150 + [18, 19, 20]])
def test_scratch_of_small_states(cuda_lib, ns):
    from qmprs_gb300 import engine as E
    eng = E.engine()
    warm = E.Plan(eng.hd, ns[:1], 1, 16)
    p = E.Plan(eng.hd, ns, 1, 16)
    for q in (warm, p):
        sv = q.vec().zero_()
        sv[torch.as_tensor(2 * q.vec_off, device="cuda")] = 1.0
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        eng.stage_mps(q, sv, 16)
        torch.cuda.synchronize()
        used = free - torch.cuda.mem_get_info()[0]
    buffers = 2 * q.tensor_elems * 8 + 2 * q.vec_elems * 4 + MB     # the outputs
    assert used <= len(ns) * 2.75 * MB + 76 * MB + 32 * MB + buffers, used / MB
