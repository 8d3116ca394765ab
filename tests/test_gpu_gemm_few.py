"""The few-token product without tensor memory at the edges of its tiles and of its dispatch, every epilogue, against 64-bit sums."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# features on both sides of every change of tile, odd ones; k that is one piece, no multiple of a warp's blocks, several rounds of them
@pytest.mark.parametrize("N,K", [(66, 8), (130, 200), (2050, 104), (9, 8192), (130, 1000), (1024, 1024), (1026, 520), (4736, 456), (4738, 504), (8192, 1000), (600, 8192)])
@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 24, 32])
def test_every_epilogue(M, N, K):
    from rustinfer_b200.ops import kernels as k, library as L
    torch.manual_seed(M)
    x, w = torch.randn(M, K, device=DEV).bfloat16(), (torch.randn(N, K, device=DEV) / K ** 0.5).bfloat16()
    want = x.double() @ w.double().T
    # bf16 products are exact in 32 bits.  Chains of eight additions that cut off, up to half a unit of 2^-23 each, joined by some twenty
    # rounded ones: a few units of 6e-8 whatever K is; measured 1.5e-7, and 4.7e-7 with K of 8,192 in one chain a warp
    tol = 3e-7
    rel = lambda a, b: ((a.double() - b).norm() / b.norm()).item()
    out = torch.full((M, N), float("nan"), device=DEV)
    k.gemm_tc(x, w, out, k.EPI_F32)
    assert rel(out, want) < tol
    again = torch.empty_like(out)
    k.gemm_tc(x, w, again, k.EPI_F32)
    assert torch.equal(out, again)                           # no order of arrival in the sums
    h = torch.randn(M, N, device=DEV)
    added = h.clone()
    k.gemm_tc(x, w, added, k.EPI_RESIDUAL)
    assert rel(added, h.double() + want) < tol
    wide = torch.zeros(M, N + 5, dtype=torch.bfloat16, device=DEV)       # rows that are not whole pieces
    k.gemm_tc(x, w, wide[:, :N], k.EPI_BF16)
    assert rel(wide[:, :N], want) < 3e-3 and not wide[:, N:].any()
    relu = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    k.gemm_tc(x, w, relu, k.EPI_RELU2)
    assert rel(relu, want.clamp(min=0) ** 2) < 3e-3
    if N % 2 == 0:
        gate, up = want[:, 0::2], want[:, 1::2]
        for epi, act in ((k.EPI_SILU, torch.nn.functional.silu(gate)), (k.EPI_GELU, torch.nn.functional.gelu(gate, approximate="tanh"))):
            pair = torch.empty(M, N // 2, dtype=torch.bfloat16, device=DEV)
            k.gemm_tc(x, w, pair, epi)
            assert rel(pair, act * up) < 4e-3
    shape = L.gemm_tc().ri_gemm_few_shape
    assert shape(33, 1024, 1024) == -1 and shape(8, 4096, 448) == -1 and shape(8, 9, 456) >= 0 and shape(8, 28672, 4096) == -1 and shape(24, 16384, 2048) == -1 and shape(8, 1024, 1024) >= 0
    assert shape(M, N, K) >= 0
    assert [shape(8, 32 * L.num_sms() + d, 1024) for d in (0, 2)] == [1, 2]    # two CTAs of 16 features an SM


# K of up to seven k-blocks; features that few tokens would find one, two and four tiles a CTA for
@pytest.mark.parametrize("N,K", [(9, 8), (1024, 64), (1024, 128), (1026, 264), (4096, 128), (8192, 448)])
def test_short_sums_have_the_same_bits_in_any_step(N, K):
    from rustinfer_b200.ops import kernels as k
    torch.manual_seed(K)
    x, w = torch.randn(700, K, device=DEV).bfloat16(), torch.randn(N, K, device=DEV).bfloat16()
    all_rows = torch.empty(700, N, device=DEV)
    k.gemm_tc(x, w, all_rows, k.EPI_F32)
    for m in (1, 8, 16, 17, 32, 33, 64, 65, 130, 300):
        out = torch.empty(m, N, device=DEV)
        k.gemm_tc(x[:m], w, out, k.EPI_F32)
        assert torch.equal(out, all_rows[:m]), m
