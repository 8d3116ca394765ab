"""The ring of the products' operand stages takes its size from the environment when the library is loaded and when a runner is made."""
from types import SimpleNamespace

from rustinfer_b200.ops import library as L


def test_a_size_set_after_the_first_product_counts(monkeypatch):
    sizes = []
    lib = SimpleNamespace(ri_gemm_tc_set_stream_budget=type("Call", (), dict(__call__=lambda self, n: sizes.append(n)))())
    monkeypatch.setattr(L, "_loaded", {})
    monkeypatch.setattr(L, "_load", lambda name, *a: L._loaded.setdefault(name, lib))
    monkeypatch.delenv("RUSTINFER_B200_STREAM_KB", raising=False)
    assert L.gemm_tc() is lib and sizes == []
    monkeypatch.setenv("RUSTINFER_B200_STREAM_KB", "96")
    L.read_stream_budget()
    assert L.gemm_tc() is lib and sizes == [96 * 1024]
    monkeypatch.setattr(L, "_loaded", {})
    assert L.gemm_tc() is lib and sizes == [96 * 1024] * 2
