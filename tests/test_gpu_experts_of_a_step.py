"""The router's loops for few and for many tokens give a token the same bits; the experts' products with three and with four stages."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("E,d,top", [(4, 40, 1), (8, 512, 2), (33, 1000, 4), (64, 513, 8)])
def test_a_token_among_few_and_many(E, d, top, dt):
    from rustinfer_b200.ops import kernels as K
    gen = torch.Generator().manual_seed(E)
    x, router = torch.randn(600, d, generator=gen).to(dt).to(DEV), (torch.randn(E + 1, d, generator=gen) / d ** 0.5).to(DEV)

    def route(part):
        T = part.shape[0]
        ids, wts, counts, gate = torch.empty((T, top), dtype=torch.int32, device=DEV), torch.empty((T, top), device=DEV), \
            torch.zeros(E, dtype=torch.int32, device=DEV), torch.empty(T, device=DEV)
        K.moe_route(None, None, top, 0, 0, True, ids, wts, counts, x=part, router=router, score="softmax", gate=gate)
        assert counts.sum().item() == T * top
        return ids, wts, gate
    whole = route(x)                                          # four tokens a CTA
    for n in (1, 148, 149, 300):                              # CTAs that all fit at once, and those that do not
        for a, b in zip(route(x[:n].contiguous()), whole):
            assert torch.equal(a, b[:n])
    z = x.double() @ router.double().T
    best = torch.softmax(z[:, :E], -1).topk(top, -1).values
    # the sums of d products and the exponentials: d^0.5 2^-24 of numbers of size 1
    assert torch.allclose(whole[1].double(), best / best.sum(-1, keepdim=True), rtol=1e-4, atol=0)
    assert torch.allclose(whole[2].double(), torch.sigmoid(z[:, E]), rtol=1e-4, atol=0)


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("E,rows,N,K_", [(4, 9, 64, 200), (32, 32, 2112, 64), (32, 70, 2112, 264)])       # one wave; two of four CTAs an SM; two either way
def test_products(E, rows, N, K_, gated):
    from rustinfer_b200.ops import kernels as K
    gen = torch.Generator().manual_seed(rows)
    a, w = torch.randn(rows, K_, generator=gen).bfloat16().to(DEV), (torch.randn(E, 2 * N if gated else N, K_, generator=gen) / K_ ** 0.5).bfloat16().to(DEV)
    owner = torch.randint(0, E, (rows,), generator=gen).sort().values
    offsets = torch.searchsorted(owner, torch.arange(E + 1)).to(torch.int32).to(DEV)
    out = torch.full((rows, N), float("nan"), device=DEV, dtype=torch.bfloat16 if gated else torch.float32)
    K.moe_product(a, w, out, offsets, None, 1, gated)
    want = torch.einsum("rk,rnk->rn", a.double(), w[owner.to(DEV)].double())
    if gated:
        want = torch.nn.functional.silu(want[:, 0::2]) * want[:, 1::2]
    # gated: half a place of bf16; else sums of K_ exact products in 32 bits
    assert ((out.double() - want).norm() / want.norm()).item() < (4e-3 if gated else 1e-6)
