"""The exact fp32 product at the edges of its tiles: every tile adds the same chain over k, so a row's bits do not depend on how many
rows (and so which tile) it is computed with."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# row counts on both sides of every change of tile; sizes that are multiples of the tiles, that are not, and rows that are not aligned
@pytest.mark.parametrize("N,K,offset", [(3072, 256, 0), (2048, 64, 0), (129, 100, 0), (61, 45, 0), (2050, 52, 3), (16400, 20, 1)])
def test_a_row_has_the_same_bits_in_every_tile(N, K, offset):
    from rustinfer_b200.ops import kernels
    torch.manual_seed(N)
    rows = [1, 2, 8, 9, 16, 17, 32, 33, 64, 65, 100, 130, 300, 321]
    a = torch.randn(rows[-1], K + 4, device=DEV)[:, offset: offset + K]
    w = torch.randn(N, K, device=DEV)
    chain = torch.zeros(rows[-1], N, dtype=torch.float64, device=DEV)
    for k in range(K):                                       # the same chain: an exact product, one rounding to 32 bits a step
        chain = (chain + a[:, k: k + 1].double() * w[:, k].double()).float().double()
    for m in rows:
        out = torch.full((m, N), 7.0, device=DEV)
        kernels.gemm_f32(a[:m], w, out)
        same = out == chain[:m].float()
        # the sum in 64 bits rounds twice where its 53 bits end in a tie of the 24: next to never
        assert same.float().mean() > 0.9999 and torch.allclose(out, chain[:m].float(), rtol=0, atol=1e-5 * K ** 0.5)
        if m == rows[0]:
            first = out
        assert torch.equal(out[:1], first)
