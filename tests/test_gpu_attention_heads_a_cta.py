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


def formula(q, keys, values, positions, Hq, Hkv, maps, scale, window, block, softcap, sink, sink_values, slopes, bias, gate, gate_scale):
    """One entry in 64 bits: q [tokens, Hq, hd], keys [keys, Hkv * maps, hd], values [keys, Hkv, vd]; out [tokens, Hq, vd]."""
    q, keys, values = q.double(), keys.double(), values.double()
    per = Hq // (Hkv * maps)
    far = positions[:, None] - torch.arange(keys.shape[0], device=q.device)[None]
    hide = far < 0
    if window:
        hide |= far >= window
    if block:
        hide |= torch.arange(keys.shape[0], device=q.device)[None] < positions[:, None] // block * block
    out = []
    for h in range(Hq):
        g = h // maps // per
        s = q[:, h] @ keys[:, g * maps + h % maps].T * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        if slopes is not None:
            s = s - slopes[h].double() * far
        if bias is not None:
            s = s + bias[h].double()[far.clamp(0, bias.shape[1] - 1)]
        s = s.masked_fill(hide, float("-inf"))
        if sink:
            first = sink_values[h].double() if sink_values is not None else torch.zeros((), dtype=torch.float64, device=q.device)
            s = torch.cat([s, first.expand(s.shape[0], 1)], dim=1)
        o = torch.softmax(s, dim=-1)[:, : keys.shape[0]] @ values[:, g]
        out.append(o * gate_scale * torch.sigmoid(gate[:, h, None].double()) if gate is not None else o)
    return torch.stack(out, dim=1)


@pytest.mark.parametrize("Hq,Hkv,maps,hd,vd,page,in_key,opts", [
    (8, 1, 2, 64, 48, 16, False, ()),                        # two maps a head: every second head reads the same keys
    (8, 2, 2, 64, 128, 8, False, ("window", "sinks")),
    (12, 1, 3, 33, 32, 4, False, ("softcap", "slopes")),     # rows that are no whole pieces of four
    (8, 2, 1, 64, 64, 16, False, ("bias", "gate")),
    (8, 2, 1, 64, 64, 16, False, ("slopes", "sink", "block")),
    (4, 1, 1, 128, 128, 32, False, ("bias", "sinks", "gate", "window")),
    (16, 1, 1, 33, 32, 16, True, ("softcap",)),              # values inside the keys
    (8, 1, 1, 48, 32, 16, True, ("sinks", "gate", "block")),
    (8, 2, 1, 23, 9, 8, False, ("gate", "softcap", "window")),
])
def test_heads_a_cta_with_options(Hq, Hkv, maps, hd, vd, page, in_key, opts):
    from rustinfer_b200.ops import kernels as K
    gen = torch.Generator().manual_seed(hd + vd + Hq)
    rnd = lambda *shape: torch.randn(shape, generator=gen).to(dev())
    i32 = lambda a: torch.as_tensor(a, dtype=torch.int32, device=dev())
    kv_lens, q_lens = [1, 33, 64, 130, 300], [1, 33, 2, 130, 17]
    n, T, Hk, pages = len(q_lens), sum(q_lens), Hkv * maps, -(-max(kv_lens) // page)
    q, keys = rnd(T, Hq * hd), rnd(n, pages * page, Hk, hd)
    values = keys[..., :vd] if in_key else rnd(n, pages * page, Hkv, vd)
    paged = lambda x: x.view(n * pages, page, *x.shape[2:]).transpose(1, 2).reshape(n * pages, -1)       # [head][slot][channel]
    parts = [paged(keys)] if in_key else [paged(keys), paged(values)]
    cache = torch.cat(parts, dim=1).contiguous()
    if hd == vd and maps == 1 and not in_key:
        cache = cache.view(n * pages, 2, Hkv, page, hd)
    kw = dict(softcap=3.0 if "softcap" in opts else None, sink="sink" in opts or "sinks" in opts, sink_values=rnd(Hq) if "sinks" in opts else None,
              slopes=rnd(Hq).abs() / 16 if "slopes" in opts else None, bias=rnd(Hq, 70) if "bias" in opts else None,
              gate=rnd(T, Hq) if "gate" in opts else None, gate_scale=0.5, block=48 if "block" in opts else None)
    window, scale = 40 if "window" in opts else None, hd ** -0.5
    cu = [sum(q_lens[:i]) for i in range(n + 1)]
    tiles = [(i, t) for i in range(n) for t in range(0, q_lens[i], 16)]
    outs = []
    for skip in (0, 700 // Hq):                              # one and two heads a CTA
        every = tiles + [(-1, 0)] * skip
        out = torch.full((T, Hq * vd), float("nan"), device=dev())
        K.attention_plain(q, out, cache, i32(list(range(n * pages))).view(n, pages), i32(cu), i32(kv_lens), i32([e for e, _ in every]),
                          i32([t for _, t in every]), Hq, Hkv, hd, scale, window, value_dim=vd, maps=maps, value_in_key=in_key, **kw)
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    for i in range(n):
        rows, k = slice(cu[i], cu[i + 1]), kv_lens[i]
        own = dict(kw, gate=kw["gate"][rows] if kw["gate"] is not None else None)
        want = formula(q[rows].view(-1, Hq, hd), keys[i, :k], values[i, :k], torch.arange(k - q_lens[i], k, device=dev()), Hq, Hkv, maps, scale,
                       window, own.pop("block"), **own)
        # a score is a sum of hd products with a rounding each (sizes up to 8: 2^-20 at most), the exponentials and the cap 2^-22 of
        # theirs, a weight's quotient as much; the weighted sum of up to 300 keys adds 2^-21 of the largest value
        err = (outs[1][rows].view(-1, Hq, vd).double() - want).abs().max()
        assert err <= 2.0 ** -17 * values.abs().max()
