"""The table of saved launch choices: entries measured on another engine are not installed."""
import json

import pytest

from brook_b200 import _native, tuning


class _Library:
    def __init__(self):
        self.installed = {}

    def brook_context_set_tuning(self, context, workload_class, choice):
        self.installed[workload_class] = choice._obj.prepare_cluster_voxels
        return _native.SUCCESS


@pytest.mark.parametrize("engine", [None, tuning.ENGINE - 1, tuning.ENGINE, tuning.ENGINE + 1])
def test_entries_of_another_engine_are_left_out(monkeypatch, tmp_path, engine):
    entry = dict(trace_cluster_ctas=8, trace_cluster_voxels=1000, prepare_cluster_voxels=4096, lone_first_percent=25)
    if engine is not None:
        entry["engine"] = engine
    path = tmp_path / "tuning.json"
    path.write_text(json.dumps({tuning._gpu_name(0): {"1a0b": entry}, "another GPU": {"2": dict(entry, engine=tuning.ENGINE)}}))
    monkeypatch.setenv("BROOK_B200_TUNING_CACHE", str(path))
    library = _Library()
    monkeypatch.setattr(tuning._native, "load", lambda: library)
    tuning.install_saved(None, 0)
    assert library.installed == ({0x1a0b: 4096} if engine == tuning.ENGINE else {})
