"""Prompt attention on tcgen05 with unrounded softmax weights (`attention_prefill_exact`) against the formula in 64 bits, at
edges of its tiles (128 rows over a key head's query heads, 64 keys), with biases that end before, inside and behind a tile."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("H,G,lens,past,window,bias_len,sink,gate,page", [
    (8, 2, [32], 0, None, 128, False, True, 16),             # one full tile of 4 heads a key head
    (8, 2, [33, 2, 31], 0, None, 1, True, False, 16),        # a tile and a row; a bias that is one number
    (6, 2, [43, 129], 63, None, 30, True, True, 8),          # 42 tokens a tile, two rows of padding
    (4, 4, [129], 64, 70, 70, False, False, 32),             # a head a key head, a window
    (8, 1, [17], 200, None, 300, False, True, 64),           # a bias longer than the prompt
    (8, 2, [260], 65, 1, 0, True, True, 16),                 # every query sees its own key alone
    (4, 2, [500], 0, None, 128, False, True, 16),            # near tiles, far tiles and the diagonal
])
def test_exact_prompt_attention(hd, H, G, lens, past, window, bias_len, sink, gate, page):
    from rustinfer_b200.ops import kernels as K
    from rustinfer_b200.parts.base import StepShape, token_tiles
    dev, gen = "cuda:0", torch.Generator().manual_seed(5)
    lens = np.array(lens)
    n, cu = len(lens), np.concatenate([[0], np.cumsum(lens)])
    T, pages = int(cu[-1]), -(-(past + int(lens.max())) // page)
    i32 = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.int32, device=dev)
    rnd = lambda *shape: torch.randn(shape, generator=gen).to(dev)
    table = torch.randperm(n * pages + 3, generator=gen)[: n * pages].reshape(n, pages)
    kv = rnd(n * pages + 3, 2, G, page, hd).to(BF)
    for i in range(n):                                       # slots behind a request's last key hold no numbers
        last = past + int(lens[i])
        flat = kv[table[i].to(dev)].transpose(2, 3).reshape(pages, 2, page, G, hd).clone()
        at = torch.arange(pages * page, device=dev).reshape(pages, 1, page, 1, 1)
        kv[table[i].to(dev)] = torch.where(at < last, flat, torch.full_like(flat, float("nan"))).transpose(2, 3)
    q = rnd(T, H * hd).to(BF)
    bias = rnd(H, bias_len) if bias_len else None
    sinks, gates = rnd(H) if sink else None, rnd(T, H) if gate else None
    assert K.tc_exact_supports(H, G, hd, page, bias_len)
    tiles = [i32(a) for a in token_tiles(K.tc_tokens_per_tile(H, G), False).build(StepShape(lens, np.full(n, past), cu, past + lens, np.arange(n)))]
    out = torch.full((T, H * hd), float("nan"), dtype=BF, device=dev)
    K.attention_prefill_exact(q, out, kv, i32(table), i32(cu), i32(past + lens), *tiles, H, G, hd, hd ** -0.5, window, sinks, bias,
                              gates, 0.5)
    got = out.double().view(T, H, hd)
    for i in range(n):
        keys = past + int(lens[i])
        kk = kv[table[i].to(dev)].double().permute(1, 2, 0, 3, 4).reshape(2, G, -1, hd)[:, :, :keys]
        far = torch.arange(past, keys, device=dev)[:, None] - torch.arange(keys, device=dev)[None]
        hide = far < 0 if window is None else (far < 0) | (far >= window)
        for h in range(H):
            rows = slice(int(cu[i]), int(cu[i + 1]))
            s = q[rows, h * hd: (h + 1) * hd].double() @ kk[0, h // (H // G)].T * hd ** -0.5
            if bias is not None:
                s = s + bias[h].double()[far.clamp(0, bias_len - 1)]
            s = s.masked_fill(hide, -math.inf)
            if sinks is not None:
                s = torch.cat([s, sinks[h].double().expand(s.shape[0], 1)], dim=1)
            want = torch.softmax(s, dim=-1)[:, :keys] @ kk[1, h // (H // G)]
            if gates is not None:
                want = want * 0.5 * torch.sigmoid(gates[rows, h, None].double())
            # half a place of bf16 (8 significant bits: 2^-8 of the number at most), and 2e-5 of the largest value: scores below 2^6 in units of log2 move a weight by 2^-18 of
            # itself, some 60 cut-off additions of the tensor core a sum by 2^-18
            assert ((got[rows, h] - want).abs() <= 2.0 ** -8 * want.abs() + 2e-5 * kk[1].abs().max()).all()
