"""The warm-start network's GEMM at the edges of its 128 x 64 tiles and four
stages, with outputs that allow 16-byte stores and outputs that do not, and
the column sums at the edges of their 32 x 32 blocks.

Bounds: products of BF16 values are exact in FP32; K sums round at 2^-24
each, so an entry is within K 2^-24 of the sum of |products|.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ws(cuda_lib):
    from qmprs_gb300 import warmstart
    return warmstart


@pytest.mark.parametrize("M,N,K,ksplit", [(128, 80, 64, 0), (256, 144, 272, 0), (128, 208, 320, 0), (128, 64, 528, 0),
                                          (256, 240, 784, 0), (128, 96, 1040, 272)])
@pytest.mark.parametrize("offset", [0, 1])
def test_gemm_tiles(ws, M, N, K, ksplit, offset):
    rng = np.random.default_rng(M + N + K)
    a = torch.as_tensor(rng.standard_normal((M, K)), device="cuda").to(torch.bfloat16).contiguous()
    b = torch.as_tensor(rng.standard_normal((N, K)), device="cuda").to(torch.bfloat16).contiguous()
    bias = torch.as_tensor(rng.standard_normal(N), device="cuda").float()
    res_store = torch.as_tensor(rng.standard_normal(M * (N + offset) + offset), device="cuda").float()
    c_store = torch.full((M * (N + offset) + offset,), float("nan"), device="cuda")
    h_store = torch.zeros(M * (N + offset) + offset, dtype=torch.bfloat16, device="cuda")
    ht = torch.zeros(N, M, dtype=torch.bfloat16, device="cuda")
    c, h, res = c_store[offset:], h_store[offset:], res_store[offset:]
    S = -(-K // ksplit) if ksplit else 1
    part = torch.zeros(S * M * N, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert ws.N.load().qmprs_gemm_bf16(ws._p(a), K, ws._p(b), K, M, N, K, ksplit, ws._p(bias), ws._p(res),
                                       N + offset, 0, ws._p(c), N + offset, ws._p(h), ws._p(ht), M, ws._p(part),
                                       ws._p(err), ws._sp(None)) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    r = res.view(M, N + offset)[:, :N].double()
    want = a.double() @ b.double().t() + bias.double() + r
    mag = a.double().abs() @ b.double().abs().t() + bias.double().abs() + r.abs()
    got = c.view(M, N + offset)[:, :N].double()
    assert bool(((got - want).abs() <= (K + 2) * 2.0 ** -24 * mag).all())
    assert torch.equal(h.view(M, N + offset)[:, :N], c.view(M, N + offset)[:, :N].to(torch.bfloat16))
    assert torch.equal(ht.t(), h.view(M, N + offset)[:, :N])
    if offset:   # nothing between the rows is written
        assert bool(torch.isnan(c.view(M, N + 1)[:, N]).all()) and bool((h.view(M, N + 1)[:, N] == 0).all())


@pytest.mark.parametrize("B", [1, 31, 33, 1000])
@pytest.mark.parametrize("N", [1, 32, 33, 256])
def test_column_sums(ws, B, N):
    x = torch.randn(B, N, generator=torch.Generator().manual_seed(B + N)).cuda()
    out = torch.full((N,), float("nan"), device="cuda")
    assert ws.N.load().qmprs_mlp_col_sum(ws._p(x), B, N, ws._p(out), ws._sp(None)) == 0
    bound = (B + 1) * 2.0 ** -24 * x.double().abs().sum(0)
    assert bool(((out.double() - x.double().sum(0)).abs() <= bound).all())
