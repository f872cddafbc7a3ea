"""The batch's two sets of launches, one per half-step and one per region, over the scenarios of
test_batch_gpu.py and test_gpu_fspace.py.  By size alone those small batches would all take the
first."""
import pytest

import test_batch_gpu
import test_gpu_fspace
from fd3d_tsn_b200.batch import Batch

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["1", "0"], ids=["per_half_step", "per_region"])
def launches(request, monkeypatch):
    monkeypatch.setenv("FD3D_BATCH_MERGED", request.param)
    b = Batch(1 << 29, 2)
    b.add(test_batch_gpu.small_models(1)[0])
    assert b.step_info()["merged"] == (request.param == "1")
    b.close()


def test_equal_single_model_runs(launches):
    test_batch_gpu.test_batch_equals_single_model_runs("graph")


def test_mixed_laws_and_uneven_lengths(launches):
    test_batch_gpu.test_batch_mixed_laws_and_uneven_lengths("graph")


def test_joining_later_and_leaving(launches):
    test_batch_gpu.test_models_joining_later_and_leaving("graph")


def test_against_oracle(launches):
    test_batch_gpu.test_batch_models_against_oracle("graph")


def test_full_space_models(launches):
    test_gpu_fspace.test_fspace_model_in_a_batch("graph")


def test_size_rule_and_overrides(monkeypatch):
    """About 120 items per SM of a velocity half-step separate the two."""
    for kchunk, merged in ((1, False), (8, True)):
        b = Batch(2 << 30, 4)
        for seed in (31, 32, 33):
            b.add(test_batch_gpu.configs.tiny_sw(seed=seed, nxT=161, nyT=65, nzT=145, nsteps=4))
        b.set_tuning(kchunk, 0)
        info = b.step_info()
        assert info["merged"] is merged, info
        b.close()
    monkeypatch.setenv("FD3D_BATCH_MERGED", "1")
    monkeypatch.setenv("FD3D_BATCH_BRANCHES", "1")  # parallel branches are launches per region
    b = Batch(1 << 29, 2)
    b.add(test_batch_gpu.small_models(1)[0])
    assert not b.step_info()["merged"]
    b.close()
