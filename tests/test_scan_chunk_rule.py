"""Which calls of the recurrences go in chunks, as far as that is decided on the host."""
from __future__ import annotations

import pytest
import torch

from rustinfer_b200.ops import kernels as K


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("H,dk,dv", [(8, 128, 256), (16, 128, 64), (64, 64, 64), (64, 128, 64), (1, 64, 64)])
def test_scratch_stays_below_its_bound(H, dk, dv, gated):
    # every array of a chunk in bytes: its state, the decays' products, the state in front of it in three bf16 pieces; gated: 64 x 64
    # scores and 64 x dk queries in three bf16 pieces too
    a_chunk = 10 * H * dk * dv + (4 * H * dk + 3 * 2 * H * 64 * (64 + dk) if gated else 8 * H)
    most = 0
    for T in [2 ** k + d for k in range(9, 22) for d in (0, 63)] + list(range(15000, 40000, 511)):
        chunks = K._scan_chunks(T, 1, T, H, dk, dv, gated, 148)
        assert chunks == 0 or chunks * 64 >= T
        assert chunks * a_chunk <= 1.26 * 2 ** 30
        most = max(most, chunks)
    assert (H == 1) or most > 0                              # the bound leaves ordinary prompts their chunks


@pytest.mark.parametrize("rows,tokens,parts,fits", [(128, 64, 36864, True), (128, 0, 0, True), (128, 32, 36864, False), (128, 64, 18432, False),
                                                    (132, 64, 36864, False)])
def test_a_library_that_counts_otherwise_is_refused(rows, tokens, parts, fits):
    lib = type("Library", (), dict(ri_recurrent_state_rows=lambda self: rows, ri_recurrent_chunk_tokens=lambda self: tokens,
                                   ri_gated_chunk_parts=lambda self: parts))()
    if fits:
        K._recurrent_sizes_agree(lib, 128, "scan")
    else:
        with pytest.raises(K.KernelError):
            K._recurrent_sizes_agree(lib, 128, "scan")


@pytest.mark.parametrize("out_at,zw_at,takes", [(0, 0, True), (1, 0, False), (2, 0, True), (0, 1, False), (0, 2, False), (0, 4, True), (0, None, True),
                                                (1, None, False)])
def test_arrays_off_their_boundaries_walk(out_at, zw_at, takes):
    lib = type("Library", (), dict(ri_chunks_ok=lambda self, *a: a[6:] == (1, 64, 1)))()
    memory = torch.zeros(64)                                  # (its own address is a multiple of 16)
    assert memory.data_ptr() % 16 == 0
    decays = memory[zw_at:] if zw_at is not None else None
    assert K._chunks_take(lib, (256, 128) * 3, torch.bfloat16, 64, True, memory[out_at:], decays) == takes


def test_a_state_off_its_boundary_is_refused(monkeypatch):
    monkeypatch.setattr(K, "_rows_checked", {64})
    cu = torch.zeros(2, dtype=torch.int32)
    state, out = torch.zeros(2 * 64 * 64 + 1), torch.zeros(5, 128)
    K._scan_common(state[:-1].view(1, 2, 64, 64), out, cu, cu, 5, 2, 64, 64, "scan")
    with pytest.raises(K.KernelError, match="16-byte"):
        K._scan_common(state[1:].view(1, 2, 64, 64), out, cu, cu, 5, 2, 64, 64, "scan")


@pytest.mark.parametrize("form,H,dk,dv,T,entries,longest,chunks", [
    ("delta", 8, 64, 64, 6400, 16, 400, False), ("delta", 8, 64, 64, 512, 1, 512, True), ("delta", 4, 128, 128, 192, 1, 192, False),
    ("delta", 16, 128, 128, 2444, 4, 761, True), ("gated", 32, 64, 64, 6400, 16, 400, False), ("gated", 8, 128, 256, 507, 8, 500, True),
    ("gated", 64, 128, 64, 2048, 1, 2048, False), ("gated", 64, 128, 64, 5000, 1, 5000, True), ("head", 32, 64, 64, 300, 1, 300, True),
    ("head", 64, 128, 64, 1138, 5, 272, False), ("head", 16, 128, 128, 900, 3, 300, True), ("head", 16, 100, 128, 2048, 1, 2048, False),
])
def test_the_sooner_way(form, H, dk, dv, T, entries, longest, chunks):
    if form == "delta":
        got = K._chunks_or_walk(T, entries, longest, H, dk, dv, 148, K.DELTA_CHUNK_MIN_TOKENS, K._delta_chunk_sizes(H, dk, dv), K._DELTA_WALK_US,
                                K._DELTA_CHUNK_FIXED_US, K._DELTA_CHUNK_US)
    else:
        got = K._scan_chunks(T, entries, longest, H, dk, dv, form == "gated", 148)
    assert (got > 0) == chunks
