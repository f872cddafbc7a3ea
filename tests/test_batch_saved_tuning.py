"""A saved batch tuning is used only for the launches it was timed on."""
import json

import pytest

import test_batch_gpu
from fd3d_tsn_b200.batch import Batch

pytestmark = pytest.mark.gpu


def autotuned(path):
    b = Batch(1 << 29, 4)
    b.add(test_batch_gpu.small_models(1)[0])
    t = b.autotune(steps=4, cache_path=str(path), key="one model")
    b.close()
    return t


def test_a_line_of_older_launches_is_timed_again(tmp_path):
    path = tmp_path / "tune.jsonl"
    first = autotuned(path)
    line = json.loads(path.read_text())
    assert line["key"].startswith("one model|") and "|launches" in line["key"]
    # the same key as it was written for the cooperative kernel, with a depth that is no candidate
    line["key"] = line["key"].split("|launches")[0]
    line.update(schedule=0, kchunk=7, ctas_per_sm=3)
    old = json.dumps(line) + "\n"
    path.write_text(old)
    t = autotuned(path)
    assert t["kchunk"] in (4, 8, 16, 32) and t["schedule"] == first["schedule"] == "graph"
    assert path.read_text().startswith(old) and len(path.read_text().splitlines()) == 2
    assert autotuned(path) == t and len(path.read_text().splitlines()) == 2  # its own line is used
