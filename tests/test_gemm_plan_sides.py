"""Products of 33 to 64 rows: which operand lies on the 128-row side, and their sums against 64 bits."""
import pytest
import torch

from rustinfer_b200.ops import kernels as K


@pytest.mark.parametrize("M,N,Kd,epilogue,weights", [
    (32, 16384, 2048, 0, True), (33, 16384, 2048, 0, False), (64, 2048, 2048, 0, False), (64, 2048, 2048, K.EPI_RESIDUAL, True),
    (36, 28672, 4096, 0, False), (48, 16384, 8192, 0, True), (48, 12288, 6144, 2, True), (48, 10240, 14336, 0, False),
    (40, 4096, 14336, 0, False), (65, 16384, 8192, 0, False), (64, 72, 64, 1, False),
])
def test_side(M, N, Kd, epilogue, weights):
    swap, bn, splits, rows = K.gemm_tc_plan(M, N, Kd, 148, epilogue)
    assert bool(swap) == weights
    tiles = -(-N // rows) * -(-M // bn) if swap else -(-M // rows) * -(-N // bn)
    assert splits == 1 or epilogue == K.EPI_RESIDUAL or tiles * splits * bn * 128 <= K._TC_WORKSPACE_FLOATS


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,Kd", [(33, 1000, 200), (33, 24, 4096), (48, 1536, 520), (64, 2056, 2048), (64, 130, 4104), (40, 12288, 6144)])
def test_sums(M, N, Kd):
    torch.manual_seed(M)
    x, w = torch.randn(M, Kd, device="cuda:0").bfloat16(), (torch.randn(N, Kd, device="cuda:0") / Kd ** 0.5).bfloat16()
    want = x.double() @ w.double().T
    rel = lambda a, b: ((a.double() - b).norm() / b.norm()).item()
    _swap, bn, splits, _rows = K.gemm_tc_plan(M, N, Kd, None, K.EPI_F32)
    # an addition of 16 exact products cuts off 2.5e-8 of the sum at the most (measured 1.5e-8 to 1.8e-8); chains are of 16 additions in
    # tiles of 64 and 128 columns, else of a slice
    tol = 2.5e-8 * max(16, Kd / splits / 16)
    out, half, pair = torch.empty(M, N, device="cuda:0"), torch.empty(M, N, device="cuda:0").bfloat16(), torch.empty(M, N // 2, device="cuda:0").bfloat16()
    K.gemm_tc(x, w, out, K.EPI_F32)
    assert rel(out, want) < tol
    again = torch.empty_like(out)
    K.gemm_tc(x, w, again, K.EPI_F32)
    assert torch.equal(out, again)
    K.gemm_tc(x, w, half, K.EPI_BF16)
    K.gemm_tc(x, w, pair, K.EPI_SILU)
    assert rel(half, want) < 3e-3 and rel(pair, torch.nn.functional.silu(want[:, 0::2]) * want[:, 1::2]) < 4e-3
    assert K.gemm_tc_error(out.device) == 0
