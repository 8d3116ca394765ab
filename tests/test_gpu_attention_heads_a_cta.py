"""`attention_plain`: the query heads that a CTA takes together (by how many tiles a call has) against one head a CTA, bit for bit, and
against the formula in 64 bits, at edges of tiles (16 tokens), half chunks and chunks of keys (32 and 64), pages and windows."""
import pytest
import torch

from test_gpu_kernels import PagedCase, close, dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("Hq,Hkv,hd,page,window", [
    (8, 2, 64, 16, None),                                    # four heads a key head: two a CTA
    (12, 4, 64, 8, 40),                                      # three: one a CTA
    (8, 2, 128, 32, 65),
    (4, 1, 48, 4, None),                                     # output pieces that not every lane has
    (4, 2, 256, 16, None),                                   # chunks of 32 keys
])
def test_heads_a_cta(dt, Hq, Hkv, hd, page, window):
    from rustinfer_b200.ops import kernels as K
    kv_lens, q_lens = [1, 32, 33, 64, 65, 130, 300], [1, 16, 33, 1, 17, 130, 2]
    case = PagedCase(dt, Hq, Hkv, hd, page, kv_lens, q_lens, seed=hd + Hq)
    te, tq = case.tiles(16)
    outs = []
    for n in (0, 700 // Hq):                                 # tiles that are skipped: one and two heads a CTA
        skip = torch.full((n,), -1, dtype=torch.int32, device=dev())
        out = torch.full_like(case.q_all, float("nan"))
        K.attention_plain(case.q_all, out, case.cache, case.table, case.cu_q, case.kv_len, torch.cat([te, skip]),
                          torch.cat([tq, torch.zeros_like(skip)]), Hq, Hkv, hd, hd ** -0.5, window)
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    close(outs[0], case.reference(hd ** -0.5, window), dt)
