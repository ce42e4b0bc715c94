"""Python's way to give back what closed plans left in the scratch pool."""
import meep_torch_b200


def test_release_scratch_reaches_the_library(monkeypatch):
    import types

    from meep_torch_b200 import _lib as L
    calls = []
    monkeypatch.setattr(L, "load", lambda: types.SimpleNamespace(
        mtb_release_scratch=lambda: calls.append(1)))
    meep_torch_b200.release_scratch()
    assert calls == [1]
