"""Kernels that take rows in aligned fours: against the general ones, which the same rows reach when they start one element later, and
against the same formulas in 64 bits."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16


def K():
    from rustinfer_b200.ops import kernels
    return kernels


def both(x):
    """x [rows, n] as a view whose rows come in aligned fours, and as one whose rows do not."""
    n = x.shape[1]
    a = torch.zeros(x.shape[0], (n + 7) // 4 * 4, dtype=x.dtype, device=DEV)
    b = torch.zeros(x.shape[0], n + 3 - (n % 2), dtype=x.dtype, device=DEV)
    a[:, :n], b[:, 1: n + 1] = x, x
    return a[:, :n], b[:, 1: n + 1]


def close(a, b, dtype):
    # the sums of a row are added in another order: a few roundings of 32 bits, which may tip one of bf16
    return ((a.float() - b.float()).norm() / b.float().norm()).item() < (2e-6 if dtype == torch.float32 else 1e-3)


@pytest.mark.parametrize("parts,n", [(1, 4), (3, 124), (2, 128), (4, 132), (1, 512), (2, 516), (1, 1024)])
@pytest.mark.parametrize("gate_first", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, BF])
def test_norm_by_parts(parts, n, gate_first, dtype):
    torch.manual_seed(n)
    T, C = 9, parts * n
    o, w = torch.randn(T, C, device=DEV), torch.randn(C, device=DEV)
    skip, got = torch.randn(C // 4, device=DEV), []
    for z, x in zip(both(torch.randn(T, C, device=DEV)), both(torch.randn(T, C, device=DEV))):
        out = torch.empty(T, C, dtype=dtype, device=DEV)
        K().part_norm_gate(o, z, w, parts, 1e-5, gate_first, out, skip=(skip, x))
        got.append(out)
    assert close(*got, dtype)


@pytest.mark.parametrize("heads,dk,rot", [(1, 8, 8), (5, 24, 16), (33, 128, 128)])
def test_rotation(heads, dk, rot):
    T = 7
    cos, sin = torch.randn(50, rot // 2, device=DEV), torch.randn(50, rot // 2, device=DEV)
    pos = torch.arange(T, dtype=torch.int32, device=DEV) * 7
    a, b = both(torch.randn(T, heads * dk, device=DEV))
    for x in (a, b):
        K().rotate_cols(x, pos, cos, sin, heads, dk, rot, False)
    assert close(a, b, torch.float32)


@pytest.mark.parametrize("H,dv", [(1, 4), (3, 100), (2, 128), (3, 132), (1, 256), (2, 512)])
@pytest.mark.parametrize("dtype", [torch.float32, BF])
@pytest.mark.parametrize("per_head", [False, True])
def test_norm_of_a_head_with_its_gate(H, dv, dtype, per_head):
    T = 11
    o, w, got = torch.randn(T, H * dv, device=DEV), torch.randn(H * dv if per_head else dv, device=DEV).to(dtype), []
    for gate in both(torch.randn(T, H * dv, device=DEV).to(dtype)):
        out = torch.empty(T, H * dv, dtype=dtype, device=DEV)
        K().gated_head_norm(o, gate, w, per_head, K().GATE_SILU, 1e-5, out, H, dv)
        got.append(out)
    assert close(*got, dtype)


@pytest.mark.parametrize("H,d", [(2, 64), (1, 128)])
@pytest.mark.parametrize("dtype", [torch.float32, BF])
def test_vectors_of_the_delta_rule(H, d, dtype):
    T, got = 5, []
    r, v, zw, ab = (torch.randn(T, H * d, device=DEV).to(dtype) for _ in range(4))
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    a = torch.randn(T, H * d, device=DEV).to(dtype)
    for k in both(torch.randn(T, H * d, device=DEV).to(dtype)):
        out, state = torch.empty(T, H * d, device=DEV), torch.zeros(1, H, d, K().recurrent_state_rows(d), device=DEV)
        z = zw.float().clone()
        K().delta_scan(r, k, v, a, ab[0].contiguous(), z, None, 0.6, 1e-6, out, state, i32([0, T]), i32([0]), 1, H, d, d)
        got += [out, z]
    assert close(got[0], got[2], torch.float32) and close(got[1], got[3], torch.float32)


@pytest.mark.parametrize("Hq,Hkv,dk,dv,rot,inter", [(4, 2, 24, 40, 0, False), (3, 3, 16, 8, 16, False), (4, 1, 32, 32, 24, True), (2, 1, 8, 4, 8, False)])
@pytest.mark.parametrize("dtype", [torch.float32, BF])
def test_queries_keys_and_values(Hq, Hkv, dk, dv, rot, inter, dtype):
    T, page, n = 6, 4, Hq * dk + Hkv * (dk + dv)
    cos, sin = (torch.randn(40, rot // 2, device=DEV) for _ in range(2)) if rot else (None, None)
    pos = torch.arange(T, dtype=torch.int32, device=DEV) * 5
    slots = torch.tensor([3, -1, 0, 9, 4, 7], dtype=torch.int32, device=DEV)
    bias, scale, got = torch.randn(n, device=DEV), torch.rand(40, device=DEV), []
    for qkv in both(torch.randn(T, n, device=DEV)):
        cache = torch.full((3, page * Hkv * (dk + dv)), 9.0, dtype=dtype, device=DEV)
        q = torch.empty(T, Hq * dk, dtype=dtype, device=DEV)
        K().qkv_prepare(qkv, bias, None, None, 0, 0.0, pos, cos, sin, rot, inter, slots, cache, q, Hq, Hkv, dk, dv, True, q_scale=scale)
        got += [q, cache]
    assert close(got[0], got[2], dtype) and close(got[1], got[3], dtype)


@pytest.mark.parametrize("rot,inter", [(64, False), (24, True), (0, False)])
@pytest.mark.parametrize("dtype", [torch.float32, BF])
def test_queries_stored_over_their_projection(rot, inter, dtype):
    T, Hq, dk = 300, 16, 64
    cos, sin = (torch.randn(T, rot // 2, device=DEV) for _ in range(2)) if rot else (None, None)
    pos, x = torch.arange(T, dtype=torch.int32, device=DEV), torch.randn(T, Hq * dk, device=DEV).to(dtype)
    apart, over = torch.empty_like(x), x.clone()
    for src, dst in ((x, apart), (over, over)):
        K().qkv_prepare(src, None, None, None, 0, 0.0, pos, cos, sin, rot, inter, None, None, dst, Hq, 1, dk, dk, False)
    assert close(over, apart, dtype)


# ---- against 64 bits: rows that come in fours and rows that do not
def near(a, want, dtype):
    # 32-bit sums and functions of a few units of 6e-8 each; a rounding to bf16 is 2^-9 at most, 1.1e-3 in the mean of squares
    return ((a.double() - want).norm() / want.norm()).item() < (2e-6 if dtype == torch.float32 else 2e-3)


@pytest.mark.parametrize("parts,n", [(3, 124), (2, 516), (1, 1024)])
@pytest.mark.parametrize("gate_first", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, BF])
def test_norm_by_parts_in_64_bits(parts, n, gate_first, dtype):
    torch.manual_seed(n + 1)
    T, C = 5, parts * n
    o, w, skip = torch.randn(T, C, device=DEV), torch.randn(C, device=DEV), torch.randn(C // 4, device=DEV)
    z0, x0 = torch.randn(T, C, device=DEV), torch.randn(T, C, device=DEV)
    y = o.double() + skip.double().repeat_interleave(4) * x0.double()
    gate = torch.nn.functional.silu(z0.double())
    rms = lambda t: (t.view(T, parts, n) / torch.sqrt((t.view(T, parts, n) ** 2).mean(-1, keepdim=True) + 1e-5)).view(T, C)
    want = rms(y * gate) * w.double() if gate_first else rms(y) * w.double() * gate
    for z, x in zip(both(z0), both(x0)):
        out = torch.empty(T, C, dtype=dtype, device=DEV)
        K().part_norm_gate(o, z, w, parts, 1e-5, gate_first, out, skip=(skip, x))
        assert near(out, want, dtype)


@pytest.mark.parametrize("H,dv", [(3, 100), (2, 512)])
@pytest.mark.parametrize("dtype", [torch.float32, BF])
@pytest.mark.parametrize("gate", ["silu", "sigmoid"])
def test_norm_of_a_head_with_its_gate_in_64_bits(H, dv, dtype, gate):
    torch.manual_seed(dv)
    T = 7
    o, w, g0 = torch.randn(T, H * dv, device=DEV), torch.randn(H * dv, device=DEV).to(dtype), torch.randn(T, H * dv, device=DEV).to(dtype)
    y, g = o.double().view(T, H, dv), g0.double()
    act = torch.nn.functional.silu(g) if gate == "silu" else torch.sigmoid(g)
    want = (y / torch.sqrt((y * y).mean(-1, keepdim=True) + 1e-5)).view(T, -1) * w.double() * act
    for x in both(g0):
        out = torch.empty(T, H * dv, dtype=dtype, device=DEV)
        K().gated_head_norm(o, x, w, True, K().GATE_SILU if gate == "silu" else K().GATE_SIGMOID, 1e-5, out, H, dv)
        assert near(out, want, dtype)


def turned(x, cos, sin, rot, inter):
    """x [T, heads, dk] in 64 bits, cos, sin [T, rot/2] of the tokens' positions."""
    x, c, s = x.clone(), cos.double()[:, None], sin.double()[:, None]
    a, b = (x[..., 0:rot:2].clone(), x[..., 1:rot:2].clone()) if inter else (x[..., : rot // 2].clone(), x[..., rot // 2: rot].clone())
    u, v = a * c - b * s, b * c + a * s
    if inter:
        x[..., 0:rot:2], x[..., 1:rot:2] = u, v
    else:
        x[..., : rot // 2], x[..., rot // 2: rot] = u, v
    return x


@pytest.mark.parametrize("heads,dk,rot", [(5, 24, 16), (33, 128, 128)])
def test_rotation_in_64_bits(heads, dk, rot):
    T = 6
    cos, sin = torch.randn(50, rot // 2, device=DEV), torch.randn(50, rot // 2, device=DEV)
    pos, x0 = torch.arange(T, dtype=torch.int32, device=DEV) * 7, torch.randn(T, heads * dk, device=DEV)
    want = turned(x0.double().view(T, heads, dk), cos[pos.long()], sin[pos.long()], rot, False).view(T, -1)
    for x in both(x0):
        K().rotate_cols(x, pos, cos, sin, heads, dk, rot, False)
        assert near(x, want, torch.float32)


@pytest.mark.parametrize("H,d", [(2, 64), (1, 128)])
@pytest.mark.parametrize("dtype", [torch.float32, BF])
def test_vectors_of_the_delta_rule_in_64_bits(H, d, dtype):
    """A request of one token from a state: the decays, and the state behind it, which unit key and rate go into."""
    torch.manual_seed(d)
    rnd = lambda *n: torch.randn(*n, device=DEV).to(dtype)
    r, v, a, ab, wb, k0, zw = rnd(1, H * d), rnd(1, H * d), rnd(1, H * d), rnd(H * d), rnd(H * d), rnd(1, H * d), torch.randn(1, H * d, device=DEV)
    S0 = torch.randn(1, H, d, K().recurrent_state_rows(d), device=DEV)
    row = lambda t: t.double().view(H, d)
    u = row(k0) / torch.sqrt((row(k0) ** 2).sum(-1, keepdim=True) + 1e-6)
    w = torch.exp(-0.6 * torch.sigmoid(row(zw) + row(wb)))
    S = S0[0].double().transpose(1, 2)
    S = w[:, :, None] * S - (torch.sigmoid(row(a) + row(ab)) * u)[:, :, None] * (S * u[:, :, None]).sum(1)[:, None] + row(k0)[:, :, None] * row(v)[:, None]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    for k in both(k0):
        z, state, out = zw.clone(), S0.clone(), torch.empty(1, H * d, device=DEV)
        K().delta_scan(r, k, v, a, ab, z, wb, 0.6, 1e-6, out, state, i32([0, 1]), i32([0]), 1, H, d, d)
        assert near(z.view(H, d), w, torch.float32) and near(state[0], S.transpose(1, 2), torch.float32)
        assert near(out.view(H, d), (S * row(r)[:, :, None]).sum(1), torch.float32)


@pytest.mark.parametrize("Hq,Hk,Hv,dk,dv,rot,inter,has_kv", [(4, 4, 2, 24, 40, 16, False, True), (4, 2, 1, 32, 8, 24, True, True),
                                                              (3, 3, 3, 16, 16, 0, False, True), (5, 1, 1, 64, 64, 64, False, False)])
@pytest.mark.parametrize("took,dtype", [(torch.float32, torch.float32), (torch.float32, BF), (BF, BF)])
def test_queries_keys_and_values_in_64_bits(Hq, Hk, Hv, dk, dv, rot, inter, has_kv, took, dtype):
    torch.manual_seed(dk)
    T, page = 6, 4
    n = Hq * dk + (Hk * dk + Hv * dv if has_kv else 0)
    cos, sin = (torch.randn(40, rot // 2, device=DEV) for _ in range(2)) if rot else (None, None)
    pos = torch.arange(T, dtype=torch.int32, device=DEV) * 5
    slots = torch.tensor([3, -1, 0, 9, 4, 7], dtype=torch.int32, device=DEV)
    bias, scale, x0 = torch.randn(n, device=DEV), torch.rand(40, device=DEV), torch.randn(T, n, device=DEV).to(took)
    y = x0.double() + bias.double()
    turn = lambda t: turned(t, cos[pos.long()], sin[pos.long()], rot, inter) if rot else t
    want_q = (turn(y[:, : Hq * dk].view(T, Hq, dk)) * scale.double()[pos.long()][:, None, None]).view(T, -1)
    want = torch.full((3, page * (Hk * dk + Hv * dv)), 9.0, dtype=torch.float64, device=DEV)
    if has_kv:
        keys, vals = turn(y[:, Hq * dk: (Hq + Hk) * dk].reshape(T, Hk, dk)), y[:, (Hq + Hk) * dk:].reshape(T, Hv, dv)
        for t, slot in enumerate(slots.tolist()):
            if slot >= 0:
                at = want[slot // page]
                at[: Hk * page * dk].view(Hk, page, dk)[:, slot % page] = keys[t]
                at[Hk * page * dk:].view(Hv, page, dv)[:, slot % page] = vals[t]
    for qkv in both(x0):
        cache = torch.full(want.shape, 9.0, dtype=dtype, device=DEV) if has_kv else None
        q = torch.empty(T, Hq * dk, dtype=dtype, device=DEV)
        K().qkv_prepare(qkv, bias, None, None, 0, 0.0, pos, cos, sin, rot, inter, slots if has_kv else None, cache, q, Hq, Hk, dk, dv, has_kv,
                        value_heads=Hv, q_scale=scale)
        assert near(q, want_q, dtype) and (not has_kv or near(cache, want, dtype))
