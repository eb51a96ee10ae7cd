"""The autotuner's file of choices: a choice holds for the library it was timed with and for
the gap-continuation class it was timed at."""
from test_autotune_logic import _Batch, _Engine
from vardepth_b200 import autotune, native


class _Params:
    def __init__(self, ext=0.1):
        self.anchored, self.ext = 0, ext


def _tuned(ext=0.1):
    eng = _Engine(lambda batch, t: 5.0 if t["pair_mask"] == 0 else 8.0)
    best = autotune.autotune(eng, _Batch(20), _Params(ext), repeats=1)
    return best["cached"], eng


def test_choices_are_kept_per_library_and_gap_continuation(monkeypatch, tmp_path):
    lib = tmp_path / "lib.so"
    lib.write_bytes(b"one")
    monkeypatch.setattr(native, "LIB_PATH", lib)
    monkeypatch.setattr(autotune, "CACHE", tmp_path / "tuning.json")
    assert not _tuned()[0]
    cached, eng = _tuned()
    assert cached and eng.tuning()["pair_mask"] == 0 and not eng.timed
    assert not _tuned(ext=0.05)[0]
    assert not _tuned(ext=0.005)[0]
    assert _tuned(ext=0.3)[0]  # the class of 0.1
    lib.write_bytes(b"two")
    cached, eng = _tuned()
    assert not cached and eng.timed
