"""A z-slab's PML sweeps keep the occupancy of a whole model's."""
import pytest

from fd3d_tsn_b200 import configs
from fd3d_tsn_b200.slab import plan
from fd3d_tsn_b200.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,h", [("f32", 200.0), ("f32", 180.8), ("f32", 225.2), ("f64", 200.0)])
def test_slab_pml_sweeps_fit_as_many_ctas_as_the_whole_models(precision, h):
    m = configs.tiny_sw(nxT=36, nyT=11, nzT=22, h=h, precision=precision)
    with Solver(m) as s:
        s.set_profiling(True)  # the separate launches, as a slab takes them
        whole = s.step_info()
    assert not whole["one_launch"]
    for rng in plan(m, 2):
        with Solver(m, slab=rng) as s:
            assert s.step_info() == whole
