"""Which calls of the recurrences go in chunks, as far as that is decided on the host."""
from __future__ import annotations

import pytest

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
