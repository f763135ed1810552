"""bench.py's other configurations belong to one-GPU jobs."""
import sys
from pathlib import Path
from types import SimpleNamespace

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("ws,no_configs,expect", [(1, False, True), (1, True, False), (2, False, False), (8, False, False)])
def test_configs_on_one_gpu_only(monkeypatch, ws, no_configs, expect):
    sys.path.insert(0, str(ROOT))
    import bench

    monkeypatch.setattr(bench, "other_configs", lambda args: {"ran": True})
    got = bench.configs_record(SimpleNamespace(no_configs=no_configs), ws)
    assert got == ({"configs": {"ran": True}} if expect else {})
