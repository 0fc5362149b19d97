"""The bulk autotuner's cache, on the CPU with the library and the timing replaced: an
entry made before the tensor-core kernel is not applied but timed anew, one of the
present kernels is applied without timing, and other entries stay in the file."""
import json

from mrg8_gb300 import autotune
from mrg8_gb300._lib import F64_SHIFTED, U32

KINDS = (F64_SHIFTED, U32)


class Library:
    def __init__(self):
        self.set = {}

    def mrg8g_tune_plain(self, kind, V, bps):
        self.set[kind] = (V, bps)
        return 0


def tune(monkeypatch, path):
    import torch
    lib, timed = Library(), []

    def time_plain(kind, n, V, bps, reps=5, out=None):
        timed.append((kind, V, bps))
        return 1.0 if (V, bps) == (0, 0) else 2.0

    monkeypatch.setattr(autotune._lib, "load", lambda: lib)
    monkeypatch.setattr(autotune, "_device_name", lambda torch: "GPU")
    monkeypatch.setattr(autotune, "time_plain", time_plain)
    monkeypatch.setattr(torch, "empty", lambda *a, **k: None)
    result = autotune.tune_plain(kinds=KINDS, n=1024, cache=str(path))
    return lib.set, timed, result


def test_entries_of_earlier_kernels_are_not_applied(monkeypatch, tmp_path):
    path = tmp_path / "cache.json"
    old = {"GPU": {name: {"V": 2, "blocks_per_sm": 0, "gsamples_per_s": 793.0} for name in autotune.KIND_NAMES.values()}}
    path.write_text(json.dumps(old))
    applied, timed, result = tune(monkeypatch, path)
    assert timed and applied == {k: (0, 0) for k in KINDS}
    saved = json.loads(path.read_text())
    assert saved["GPU"] == old["GPU"] and len(saved) == 2
    applied, timed, again = tune(monkeypatch, path)
    assert not timed and applied == {k: (0, 0) for k in KINDS} and again == result
