"""Recurrences over long portions in chunks (recurrent_chunks.cu) against the token-by-token recurrence in 64 bits, at the edges of
chunks, beside entries that walk, and with decays of zero and values that are no numbers."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, F64 = "cuda:0", torch.float64


def K():
    from rustinfer_b200.ops import kernels
    return kernels


@pytest.fixture(autouse=True)
def chunks_whatever_they_cost(monkeypatch, request):
    """Portions of a few hundred tokens go in chunks, so that their edges are met without long prompts."""
    if "keep_the_walk" not in request.node.name:
        monkeypatch.setattr(K(), "_CHUNK_FIXED_US", {False: -1e9, True: -1e9})


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def rel_err(x, want):
    return ((x.to(F64) - want).norm() / want.norm()).item()


def walk(q, k, v, a, state, cu, slots):
    """q, k [T, H, dk], v [T, H, dv], a [T, H, dk or 1] in float64; state [slots, H, dv, dk], updated in place."""
    out = torch.empty_like(v)
    for e, slot in enumerate(slots):
        S = state[slot].transpose(1, 2).clone()
        for t in range(cu[e], cu[e + 1]):
            S = a[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None]
            out[t] = (S * q[t][:, :, None]).sum(1)
        state[slot] = S.transpose(1, 2)
    return out


def lengths(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return cu, list(range(len(lens)))[::-1]


# a chunk is 64 tokens: portions that end on one, one before and one behind it, and in a quarter; entries too short for chunks
@pytest.mark.parametrize("lens", [[256], [257], [319, 1, 17, 320], [300, 255, 410]])
@pytest.mark.parametrize("H,G,dk,dv,kind,dtype", [(4, 4, 128, 128, "fixed", torch.float32), (8, 2, 128, 64, "steps", torch.float32),
                                                  (3, 3, 64, 192, "steps", torch.float32), (2, 1, 64, 64, "fixed", torch.bfloat16)])
def test_one_decay_a_head(lens, H, G, dk, dv, kind, dtype):
    torch.manual_seed(len(lens))
    (cu, slots), T = lengths(lens), sum(lens)
    x = torch.randn(T, 2 * G * dk + H * dv + 4, device=DEV).to(dtype)
    q, k, v = x[:, : G * dk], x[:, G * dk: 2 * G * dk], x[:, 2 * G * dk: 2 * G * dk + H * dv]
    gain = None
    if kind == "fixed":
        decay = torch.linspace(0.6, 0.9997, H, device=DEV)
    else:
        gain = torch.rand(T, H, device=DEV) + 0.1
        decay = torch.exp(-gain * torch.linspace(0.05, 6.0, H, device=DEV)) * (torch.rand(T, H, device=DEV) > 0.02)   # some are zero
    state = torch.randn(len(lens) + 1, H, dv, K().recurrent_state_rows(dk), device=DEV)
    want_state, out = state.to(F64), torch.empty(T, H * dv, device=DEV)
    spread = lambda t: t.to(F64).view(T, G, dk).repeat_interleave(H // G, 1)
    vals = v.to(F64).view(T, H, dv) * (gain.to(F64)[:, :, None] if gain is not None else 1.0)
    want = walk(spread(q) * 0.3, spread(k), vals, decay.to(F64).expand(T, H)[:, :, None], want_state, cu, slots)
    untouched = state[-1].clone()
    K().head_scan(q, k, v, decay, 0.3, out, state, i32(cu), i32(slots), len(lens), H, dk, dv, gain=gain, key_heads=G, longest=max(lens))
    # 32-bit sums of up to dk + 64 products and of a state of hundreds of tokens: a few roundings of 6e-8 each
    assert rel_err(out, want.view(T, -1)) < 1e-6
    assert rel_err(state[:-1], want_state[:-1]) < 1e-6
    assert torch.equal(state[-1], untouched)


@pytest.mark.parametrize("lens", [[384], [385], [447, 1, 33, 448], [500, 383, 511]])
@pytest.mark.parametrize("H,dk,dv,shift", [(2, 128, 256, 2.0), (3, 64, 64, -60.0), (2, 128, 192, 0.0)])
def test_a_decay_a_key_channel(lens, H, dk, dv, shift):
    torch.manual_seed(len(lens))
    (cu, slots), T = lengths(lens), sum(lens)
    x = torch.randn(T, 2 * H * dk + H * dv + 4, device=DEV).bfloat16()
    q, k, v = x[:, : H * dk], x[:, H * dk: 2 * H * dk], x[:, 2 * H * dk: 2 * H * dk + H * dv]
    z = torch.randn(T, H * dk, device=DEV) * 40.0 + shift                 # decays down to zero
    state = torch.randn(len(lens) + 1, H, dv, K().recurrent_state_rows(dk), device=DEV)
    want_state, out = state.to(F64), torch.empty(T, H * dv, device=DEV)
    untouched = state[-1].clone()
    K().gated_scan(q, k, v, z, None, 0.3, 1.0, out, state, i32(cu), i32(slots), len(lens), H, dk, dv, longest=max(lens))
    # z now holds the decays the recurrence used
    part = lambda t, n: t.to(F64).view(T, H, n)
    want = walk(part(q, dk) * 0.3, part(k, dk), part(v, dv), part(z, dk), want_state, cu, slots)
    assert rel_err(out, want.view(T, -1)) < 1e-6
    assert rel_err(state[:-1], want_state[:-1]) < 1e-6
    assert torch.equal(state[-1], untouched)


@pytest.mark.parametrize("kind,params", [
    ("gated_linear_attention", dict(num_heads=2, key_dim=128, value_dim=128, tau=16.0, decay_rank=16)),
    ("lightning_attention", dict(num_heads=2, key_dim=64, value_dim=128, decay=[0.9, 0.999])),
    ("retention", dict(num_heads=2, key_dim=128, value_dim=64, decay=[0.97, 0.9998])),
    ("mamba2", dict(num_heads=4, value_dim=64, state_dim=128, groups=2, conv_taps=4, norm_groups=2))])
def test_a_layer_in_chunks_is_the_layer_that_walks(kind, params, monkeypatch):
    import numpy as np
    import rustinfer_b200.models.decoder  # noqa: F401
    from rustinfer_b200.parts.base import MIXERS, BuildContext, StateLayerCache, StepContext
    from rustinfer_b200.parts.spec import PartSpec
    torch.manual_seed(5)
    part = MIXERS.build(PartSpec(kind, dict(hidden_size=128, norm_eps=1e-5, **params)))
    part.prepare(BuildContext(torch.device(DEV), torch.bfloat16, 1024, 16, max_batch_seqs=4))
    part.load({n: (torch.randn([16 if s == -1 else s for s in d.shape], device=DEV) * 0.1).bfloat16() for n, d in part.param_decls().items()})
    lens = [400, 9, 450]
    cu, slots = lengths(lens)
    T = sum(lens)
    step = StepContext(T, 3, i32([0] * T), i32(np.concatenate([np.arange(n) for n in lens])), i32(cu), i32(lens), i32(slots), [], [], 450, 450, False)
    needs = part.cache_need()
    needs = needs if isinstance(needs, tuple) else (needs,)
    start = [torch.randn((3,) + tuple(n.shape), device=DEV) for n in needs]
    x, got = torch.randn(T, 128, device=DEV).bfloat16(), []
    for fixed in (-1e9, 1e9):
        monkeypatch.setattr(K(), "_CHUNK_FIXED_US", {False: fixed, True: fixed})
        caches = tuple(StateLayerCache(t.clone()) for t in start)
        out = part.forward(x, step, caches if len(caches) > 1 else caches[0])
        got.append((out.float(), [c.state for c in caches]))
    # the recurrence's 32-bit sums in another order, rounded to bf16 behind the norm: a rounding tips here and there
    assert rel_err(got[0][0], got[1][0].to(F64)) < 2e-3
    assert all(rel_err(a, b.to(F64)) < 1e-5 for a, b in zip(got[0][1], got[1][1]))


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_a_value_that_is_no_number_reaches_later_tokens_only(gated, value):
    torch.manual_seed(0)
    T, H, dk, dv, at, column = 450, 2, 64, 64, 139, 70
    x = torch.randn(T, 2 * H * dk + H * dv, device=DEV).to(torch.bfloat16 if gated else torch.float32)
    decay = torch.full((T, H * dk) if gated else (T, H), 0.9, device=DEV)

    def run(x):
        q, k, v = x[:, : H * dk], x[:, H * dk: 2 * H * dk], x[:, 2 * H * dk:]
        out, state = torch.empty(T, H * dv, device=DEV), torch.zeros(1, H, dv, K().recurrent_state_rows(dk), device=DEV)
        if gated:
            K().gated_scan(q, k, v, torch.logit(decay), None, 1.0, 1.0, out, state, i32([0, T]), i32([0]), 1, H, dk, dv, longest=T)
        else:
            K().head_scan(q, k, v, decay, 1.0, out, state, i32([0, T]), i32([0]), 1, H, dk, dv, longest=T)
        return out, state
    clean, _ = run(x)
    x[at, 2 * H * dk + column] = value
    got, state = run(x)
    others = torch.arange(H * dv, device=DEV) != column
    assert torch.equal(got[:, others], clean[:, others]) and torch.equal(got[:at, column], clean[:at, column])
    assert not torch.isfinite(got[at:, column]).any() and not torch.isfinite(state.view(H * dv, -1)[column]).any()


def test_calls_that_keep_the_walk():
    """Short entries, batches that walk as fast, sizes the chunks are not made for, rows that are not aligned and callers that do not
    ask for chunks."""
    chunks = lambda T, n, longest, H=16, dk=128, dv=128, gated=False: K()._scan_chunks(T, n, longest, H, dk, dv, gated, 148)
    assert chunks(255, 1, 255) == 0 and chunks(4096, 16, 0) == 0
    assert chunks(8192, 1, 8192, H=1024) == 0                             # more scratch than a call takes
    assert chunks(1138, 5, 272, H=64, dv=64) == 0                         # one entry that could, four that walk beside it
    assert chunks(2048, 1, 2048) >= 32 and chunks(1749, 2, 999) >= 28 and chunks(2056, 9, 2048) >= 33
    assert chunks(384, 1, 384, H=8, dv=256, gated=True) == 0 and chunks(2048, 1, 2048, H=8, dv=256, gated=True) >= 32
    lib = __import__("rustinfer_b200.ops.library", fromlist=["recurrent"]).recurrent(64)
    ok = lambda stride, dv: lib.ri_chunks_ok(256, stride, 256, stride, 256, stride, 0, dv, 0)
    assert ok(128, 64) and not ok(129, 64) and not ok(128, 48)
    assert not lib.ri_chunks_ok(256, 128, 256, 128, 256, 128, 0, 64, 1)    # the gated form takes bf16


@pytest.mark.parametrize("gated", [False, True])
def test_a_call_without_room_for_scratch_walks(gated, monkeypatch):
    torch.manual_seed(1)
    T, H, dk, dv = 450, 2, 64, 64
    x = torch.randn(T, 2 * H * dk + H * dv, device=DEV).bfloat16()
    q, k, v = x[:, : H * dk], x[:, H * dk: 2 * H * dk], x[:, 2 * H * dk:]

    def run(longest):
        out, state = torch.empty(T, H * dv, device=DEV), torch.ones(1, H, dv, K().recurrent_state_rows(dk), device=DEV)
        args = (out, state, i32([0, T]), i32([0]), 1, H, dk, dv)
        if gated:
            K().gated_scan(q, k, v, torch.ones(T, H * dk, device=DEV), None, 1.0, 4.0, *args, longest=longest)
        else:
            K().head_scan(q, k, v, torch.full((H,), 0.9, device=DEV), 1.0, *args, longest=longest)
        return out, state
    walked, empty = run(0), torch.empty
    in_chunks = run(T)

    def full(*size, **kw):
        if kw.get("dtype") == torch.uint8:
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(*size, **kw)
    monkeypatch.setattr(torch, "empty", full)
    got = run(T)
    assert all(torch.equal(a, b) for a, b in zip(got, walked)) and not torch.equal(in_chunks[0], walked[0])


@pytest.mark.parametrize("gated", [False, True])
def test_outputs_off_their_boundary_walk(gated, monkeypatch):
    monkeypatch.setattr(K(), "_CHUNK_FIXED_US", {False: -1e9, True: -1e9})
    torch.manual_seed(2)
    T, H, dk, dv = 450, 2, 64, 64
    x = torch.randn(T, 2 * H * dk + H * dv, device=DEV).bfloat16()
    q, k, v = x[:, : H * dk], x[:, H * dk: 2 * H * dk], x[:, 2 * H * dk:]
    got = {}
    for at, longest in ((0, 0), (0, T), (1, T)):
        out = torch.empty(T * H * dv + 1, device=DEV)[at: at + T * H * dv].view(T, H * dv)
        state = torch.ones(1, H, dv, K().recurrent_state_rows(dk), device=DEV)
        args = (out, state, i32([0, T]), i32([0]), 1, H, dk, dv)
        if gated:
            K().gated_scan(q, k, v, torch.ones(T, H * dk, device=DEV), None, 1.0, 4.0, *args, longest=longest)
        else:
            K().head_scan(q, k, v, torch.full((H,), 0.9, device=DEV), 1.0, *args, longest=longest)
        got[at, longest] = out, state
    walked, in_chunks, off = got.values()
    assert all(torch.equal(a, b) for a, b in zip(off, walked)) and not torch.equal(in_chunks[0], walked[0])
