"""Products of mid sizes (more than 64 rows, too few tiles for the GPU) under the plan they get, against 64-bit sums."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# tiles of 64 and 128 features, their remainders, a K in several slices, the last size before whole tiles of 256
@pytest.mark.parametrize("M,N,K", [(65, 72, 64), (65, 1000, 200), (129, 1024, 4096), (300, 3072, 520), (511, 2056, 2048), (1024, 2048, 1024),
                                   (2048, 1024, 8192), (1030, 130, 4104)])
def test_mid_sizes(M, N, K):
    from rustinfer_b200.ops import kernels as k
    torch.manual_seed(N)
    x, w = torch.randn(M, K, device=DEV).bfloat16(), (torch.randn(N, K, device=DEV) / K ** 0.5).bfloat16()
    want = x.double() @ w.double().T
    # bf16 products are exact in 32 bits.  An addition of 16 of them cuts off half a unit of the last of 24 bits on average, relative to a
    # sum of the end's size 3e-8, and the sums are smaller on the way: measured 1.5e-8 to 1.8e-8 an addition of a chain.  Chains are of 16
    # additions, or of a slice where tiles of 256 columns stay
    bn, splits = k.gemm_tc_plan(M, N, K)[1:3]
    tol = 2.5e-8 * (16 if bn < 256 else K / splits / 16)
    assert bn < 256 or K >= 8192                             # the narrow tiles take all but the longest
    rel = lambda a, b: ((a.double() - b).norm() / b.norm()).item()
    out, half, pair = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV).bfloat16(), torch.empty(M, N // 2, device=DEV).bfloat16()
    k.gemm_tc(x, w, out, k.EPI_F32)
    assert rel(out, want) < tol
    h = torch.randn(M, N, device=DEV)
    added = h.clone()
    k.gemm_tc(x, w, added, k.EPI_RESIDUAL)
    assert rel(added, h.double() + want) < tol
    k.gemm_tc(x, w, half, k.EPI_BF16)
    k.gemm_tc(x, w, pair, k.EPI_SILU)
    assert rel(half, want) < 3e-3 and rel(pair, torch.nn.functional.silu(want[:, 0::2]) * want[:, 1::2]) < 4e-3
    assert k.gemm_tc_error(out.device) == 0


@pytest.mark.parametrize("bn", [64, 128])
@pytest.mark.parametrize("M,N,K,splits", [(70, 200, 576, 6), (130, 128, 704, 1), (300, 136, 1160, 4), (128, 64, 512, 1)])
def test_chains_and_slices(M, N, K, splits, bn):
    """Tiles that sum short chains: an uneven last chain, slices that get no k-block, rows of the stream with and without vector adds."""
    from rustinfer_b200.ops import kernels as k
    torch.manual_seed(K)
    x, w = torch.randn(M, K, device=DEV).bfloat16(), (torch.randn(N, K, device=DEV) / K ** 0.5).bfloat16()
    want = x.double() @ w.double().T
    rel = lambda a, b: ((a.double() - b).norm() / b.norm()).item()
    h = torch.randn(M, N + 3, device=DEV)
    for out in (h[:, :N].contiguous(), h.clone()[:, :N]):    # rows of whole vectors, rows that are not
        was = out.double()
        k.gemm_tc(x, w, out, k.EPI_RESIDUAL, (0, bn, splits, 128))
        assert rel(out, was + want) < 4e-7
        k.gemm_tc(x, w, out, k.EPI_F32, (0, bn, splits, 128))
        assert rel(out, want) < 4e-7
        again = torch.empty_like(out)
        k.gemm_tc(x, w, again, k.EPI_F32, (0, bn, splits, 128))
        assert torch.equal(out, again)                       # slices are added in their order, not in that of their arrival
    assert k.gemm_tc_error(out.device) == 0
