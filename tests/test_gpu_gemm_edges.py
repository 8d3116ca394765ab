"""Products whose features end inside a tile: the columns have the bits they have in a wider product, and nothing behind a row's end
is written, whatever the rows' alignment (vector stores of 32 or 16 bytes, or none)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("plan", [(0, 256, 1, 128), (0, 128, 1, 128), (0, 64, 1, 128)])
@pytest.mark.parametrize("N", [320, 264, 272, 280, 258, 16, 2])
@pytest.mark.parametrize("epilogue", ["EPI_F32", "EPI_BF16", "EPI_SILU", "EPI_RESIDUAL", "EPI_RELU2"])
def test_columns_at_the_edge(plan, N, epilogue):
    from rustinfer_b200.ops import kernels as K
    M, Kd, wide = 515, 192, 512                              # rows from 512 on: the kernel of CTA pairs (256 columns)
    torch.manual_seed(N)
    epi = getattr(K, epilogue)
    half = 2 if epi == K.EPI_SILU else 1
    x, w = torch.randn(M, Kd, device=DEV).bfloat16(), torch.randn(wide, Kd, device=DEV).bfloat16()
    dt = torch.float32 if epi in (K.EPI_F32, K.EPI_RESIDUAL) else torch.bfloat16
    base = torch.randn(M, wide // half, device=DEV).to(dt)
    want = base.clone()
    K.gemm_tc(x, w, want, epi, plan)
    block = torch.full((M * (N // half) + 64,), 7.0, dtype=dt, device=DEV)
    got = block[: M * (N // half)].view(M, N // half)
    got.copy_(base[:, : N // half])
    K.gemm_tc(x, w[:N].contiguous(), got, epi, plan)
    assert torch.equal(got, want[:, : N // half])
    assert (block[M * (N // half):] == 7.0).all()


@pytest.mark.parametrize("M", [33, 36, 37, 64])
@pytest.mark.parametrize("N,Kd", [(2048, 1024), (72, 2048), (3104, 520), (16, 1024)])
def test_rows_from_33_on_as_in_a_prompt(M, N, Kd):
    """33 to 64 rows go the way of 65: their sums have the bits they have there."""
    from rustinfer_b200.ops import kernels as K
    torch.manual_seed(Kd)
    x, w = torch.randn(65, Kd, device=DEV).bfloat16(), torch.randn(N, Kd, device=DEV).bfloat16()
    for epi, dt in ((K.EPI_F32, torch.float32), (K.EPI_BF16, torch.bfloat16)):
        few, many = torch.empty(M, N, dtype=dt, device=DEV), torch.empty(65, N, dtype=dt, device=DEV)
        K.gemm_tc(x[:M], w, few, epi)
        K.gemm_tc(x, w, many, epi)
        assert torch.equal(few, many[:M])
