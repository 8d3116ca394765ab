"""The delta rule in chunks (recurrent_chunks.cu) against the recurrence in 64 bits and against the walk: chunks cut short, entries of
several lengths beside one another, value sizes other than the keys', the strongest decays it takes, numbers that are none."""
import math

import numpy as np
import pytest
import torch

BF = torch.bfloat16


def K():
    from rustinfer_b200.ops import kernels
    return kernels


def test_which_calls_go_in_chunks():
    k = K()
    sizes = k._delta_chunk_sizes(16, 128, 128)
    take = lambda T, n, longest, heads=16, dk=128: k._chunks_or_walk(
        T, n, longest, heads, dk, dk, 148, k.DELTA_CHUNK_MIN_TOKENS, k._delta_chunk_sizes(heads, dk, dk), k._DELTA_WALK_US, k._DELTA_CHUNK_FIXED_US,
        k._DELTA_CHUNK_US)
    assert take(512, 1, 512) == 9 and take(2048, 1, 2048) == 33 and take(2444, 4, 761) >= 42
    assert take(100, 1, 100) == 0 and take(192, 1, 192) == 0 and take(8, 8, 1) == 0
    assert 6 * 16 * 64 * 128 == sizes[4] == sizes[5] and sizes[3] == 6 * 16 * 64 * (64 + 128) and sum(sizes) * 300 > k.CHUNK_SCRATCH_BYTES
    assert take(300 * 64, 1, 300 * 64) == 0                  # no room in the scratch: a walk


def make(lens, H, dk, dv, low=-6.0, high=0.0):
    dev, gen = "cuda:0", torch.Generator().manual_seed(11)
    lens = np.array(lens)
    cu, n = np.concatenate([[0], np.cumsum(lens)]), len(lens)
    T = int(cu[-1])
    rnd = lambda *shape: torch.randn(shape, generator=gen).to(dev)
    wide = rnd(T, H * (3 * dk + dv) + 8).to(BF)              # columns of one product, as a layer has them
    r, k, za, v = (wide[:, a: a + m] for a, m in ((0, H * dk), (H * dk, H * dk), (2 * H * dk, H * dk), (3 * H * dk, H * dv)))
    i32 = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.int32, device=dev)
    return dict(r=r, k=k, v=v, za=za, zw=0.3 * rnd(T, H * dk), bias=(torch.rand(H * dk, generator=gen) * (high - low) + low).to(dev),
                state=0.3 * rnd(n + 1, H, dv, dk), cu=cu, cu_q=i32(cu), slots=i32(np.arange(n)[::-1] + 1), n=n, T=T, H=H, dk=dk, dv=dv)


def scan(c, longest, rate):
    out, state, zw = torch.full((c["T"], c["H"] * c["dv"]), float("nan"), device=c["r"].device), c["state"].clone(), c["zw"].clone()
    K().delta_scan(c["r"], c["k"], c["v"], c["za"], None, zw, c["bias"], rate, 1e-6, out, state, c["cu_q"], c["slots"], c["n"], c["H"], c["dk"],
                   c["dv"], longest=longest)
    return out.view(c["T"], c["H"], c["dv"]), state


def exact(c, rate):
    T, H, dk, dv = c["T"], c["H"], c["dk"], c["dv"]
    r, k, za = (c[x].double().view(T, H, dk) for x in ("r", "k", "za"))
    v, state, out = c["v"].double().view(T, H, dv), c["state"].double(), torch.empty(T, H, dv, dtype=torch.float64, device=c["r"].device)
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    w = torch.exp(-rate * torch.sigmoid(c["zw"].double() + c["bias"].double())).view(T, H, dk)
    au = torch.sigmoid(za) * u
    for i in range(c["n"]):
        slot = int(c["slots"][i])
        S = state[slot].transpose(1, 2).clone()
        for t in range(int(c["cu"][i]), int(c["cu"][i + 1])):
            dot = (S * u[t][:, :, None]).sum(1)
            S = w[t][:, :, None] * S - au[t][:, :, None] * dot[:, None] + k[t][:, :, None] * v[t][:, None]
            out[t] = (S * r[t][:, :, None]).sum(1)
        state[slot] = S.transpose(1, 2)
    return out, state


off = lambda a, b: float((a.double() - b).norm() / b.norm())


@pytest.mark.gpu
@pytest.mark.parametrize("lens,H,dk,dv,rate,low,high", [
    ([192], 2, 128, 128, math.exp(-0.5), -6.0, 0.0),                      # whole chunks
    ([193, 255, 64, 1], 3, 128, 128, math.exp(-0.5), -6.0, 0.0),          # one token over, one short; entries that walk
    ([260], 10, 128, 128, math.exp(-0.5), -6.0, 0.0),                     # 32 value channels a CTA of the scan from 149 blocks on
    ([200] * 4, 10, 128, 128, math.exp(-0.5), -6.0, 0.0),                 # 64 from 297 on
    ([321], 2, 64, 192, math.exp(-0.5), -6.0, 0.0),                       # other sizes of keys and values
    ([200], 2, 128, 64, math.exp(-0.5), -9.0, -8.0),                      # hardly any decay
    ([230], 2, 128, 128, 1.0, 2.0, 6.0),                                  # the strongest: e^-1 a token
])
def test_chunks_as_near_as_the_walk(lens, H, dk, dv, rate, low, high, monkeypatch):
    monkeypatch.setattr(K(), "_DELTA_CHUNK_FIXED_US", -1e9)
    c = make(lens, H, dk, dv, low, high)
    want, walked, got = exact(c, rate), scan(c, 0, rate), scan(c, max(lens), rate)
    assert not torch.equal(walked[0], got[0])                # the chunks ran
    short = torch.as_tensor(np.repeat(np.array(lens) < K().DELTA_CHUNK_MIN_TOKENS, lens), device=got[0].device)
    assert torch.equal(walked[0][short], got[0][short])
    for a, b, x in zip(got, walked, want):
        # both ways round every product and sum to 2^-24; a chunk's score adds a factor's and a reciprocal's rounding to a term
        assert off(a, x) <= 1.25 * off(b, x) + 2.0 ** -23


@pytest.mark.gpu
def test_stronger_decays_walk(monkeypatch):
    monkeypatch.setattr(K(), "_DELTA_CHUNK_FIXED_US", -1e9)
    c = make([256], 2, 128, 128)
    for a, b in zip(scan(c, 256, 1.01), scan(c, 0, 1.01)):
        assert torch.equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["k", "zw", "v"])
def test_a_number_that_is_none_spares_earlier_tokens_and_other_heads(where, monkeypatch):
    monkeypatch.setattr(K(), "_DELTA_CHUNK_FIXED_US", -1e9)
    c = make([300], 3, 128, 128)
    clean = scan(c, 300, 0.6)
    c[where] = c[where].clone()
    c[where][150, 1 * 128 + 5] = float("nan")
    out, state = scan(c, 300, 0.6)
    assert torch.equal(out[:, [0, 2]], clean[0][:, [0, 2]]) and torch.equal(state[1, [0, 2]], clean[1][1, [0, 2]])
    hit = slice(5, 6) if where == "v" else slice(0, 128)     # a value channel's column, or the head
    rest = [i for i in range(128) if i != 5] if where == "v" else []
    assert torch.isnan(out[150:, 1, hit]).all() and torch.isnan(state[1, 1, hit]).all()
    assert off(out[:150, 1], clean[0][:150, 1].double()) <= 1e-6          # the chunk's later tokens are left out of its sums
    assert torch.equal(out[:, 1, rest], clean[0][:, 1, rest]) and torch.equal(state[1, 1, rest], clean[1][1, 1, rest])


@pytest.mark.gpu
@pytest.mark.parametrize("out_at,zw_at", [(1, 0), (0, 1), (0, 2), (3, 3)])
def test_arrays_off_their_boundaries_walk(out_at, zw_at, monkeypatch):
    monkeypatch.setattr(K(), "_DELTA_CHUNK_FIXED_US", -1e9)
    c = make([256], 2, 128, 128)
    n, got = c["T"] * 2 * 128, []
    for longest in (0, 256):                                  # the walk, and the call that could go in chunks
        out, zw = (torch.full((n + 4,), float("nan"), device=c["r"].device)[at: at + n].view(c["T"], -1) for at in (out_at, zw_at))
        zw.copy_(c["zw"])
        state = c["state"].clone()
        K().delta_scan(c["r"], c["k"], c["v"], c["za"], None, zw, c["bias"], 0.6, 1e-6, out, state, c["cu_q"], c["slots"], 1, 2, 128, 128,
                       longest=longest)
        got.append((out, state))
    assert all(torch.equal(a, b) for a, b in zip(*got)) and torch.isfinite(got[0][0]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("noise", [0.0, 0.05, 0.5])
@pytest.mark.parametrize("dk", [64, 128])
def test_keys_that_resemble_one_another(noise, dk, monkeypatch):
    """Where the triangular system is far from the identity: keys around a common vector, hardly any decay, nearly all of u^T S taken away."""
    monkeypatch.setattr(K(), "_DELTA_CHUNK_FIXED_US", -1e9)
    c = make([320], 2, dk, dk, -9.0, -8.0)
    gen = torch.Generator().manual_seed(3)
    common = torch.randn((1, 2 * dk), generator=gen).to(c["k"].device)
    c["k"] = (common + noise * torch.randn((c["T"], 2 * dk), generator=gen).to(common.device)).to(BF)
    c["za"] = torch.full_like(c["k"], 6.0)
    rate = math.exp(-0.5)
    want, walked, got = exact(c, rate), scan(c, 0, rate), scan(c, 320, rate)
    assert not torch.equal(walked[0], got[0])
    for a, b, x in zip(got, walked, want):
        # repeated keys: earlier values are erased by differences of scores that are equal but for their roundings (2^-23 each), 64 in a chunk
        assert off(a, x) <= 1.25 * off(b, x) + (2.0 ** -23 if noise else 64 ** 0.5 * 2 * 2.0 ** -23)


@pytest.mark.gpu
def test_reciprocals():
    """Every significand of one power of two, and the range that products of 32 decays of at least e^-1 have."""
    from rustinfer_b200.ops import library as L
    lib = L.recurrent(128)
    for bits in (torch.arange(0x3f800000, 0x40000000, dtype=torch.int32, device="cuda:0"),
                 torch.arange(0x28000000, 0x57800000, 251, dtype=torch.int32, device="cuda:0")):          # 2^-47 .. 2^48
        x = bits.view(torch.float32)
        y = torch.empty_like(x)
        L.check(lib.ri_delta_chunk_reciprocals(x.data_ptr(), y.data_ptr(), x.numel(), L.stream_ptr()), "reciprocals")
        # a rounding, and the square of the approximation's error (2^-46): half a unit of the last place, as CUDA's own is
        assert float((y.double() * x.double() - 1).abs().max()) <= 2.0 ** -24 * (1 + 2.0 ** -10)
        assert int((y.view(torch.int32) - torch.reciprocal(x).view(torch.int32)).abs().max()) <= 1
