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
    tol = 1e-6 + K / 16 * 6e-8                               # a chain of K / 16 additions that cut off
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
