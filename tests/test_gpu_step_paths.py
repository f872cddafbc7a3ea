"""Which launches a step takes, by size: the sizes at which test_gpu_dispatch.py compares the two
sides of the rule really lie on the two sides."""
import pytest

from fd3d_tsn_b200 import configs
from fd3d_tsn_b200.solver import Solver

pytestmark = pytest.mark.gpu


# CTAs of a velocity half-step (12 x 148 = 1776 is the border): 62 to 338, 1625, 2219 and 2000; for slip
# weakening in double precision 9.5 x 148 = 1406: 1171 and 1359, 1438 and 1556
@pytest.mark.parametrize("law,precision,fspace,size,one_launch", [
    ("sw", "f32", False, (14, 9, 13), True),
    ("sw", "f32", False, (33, 12, 41), True),
    ("sw", "f32", True, (65, 17, 26), True),
    ("sw", "f64", False, (37, 11, 23), True),
    ("sw", "f64", True, (31, 14, 33), True),
    ("fvw", "f32", False, (41, 15, 29), True),
    ("fvw", "f64", True, (40, 13, 28), True),
    ("sw", "f32", False, (121, 47, 83), True),
    ("sw", "f32", False, (161, 61, 93), False),
    ("sw", "f32", True, (129, 55, 87), False),
    ("sw", "f64", False, (90, 50, 70), True),
    ("sw", "f64", False, (101, 47, 73), True),
    ("sw", "f64", False, (96, 56, 80), False),
    ("sw", "f64", False, (160, 40, 70), False),
    ("fvw", "f64", False, (160, 40, 70), True),
    ("sw", "f32", False, (160, 40, 70), True),
])
def test_one_launch_per_half_step_by_size(law, precision, fspace, size, one_launch, monkeypatch):
    nx, ny, nz = size
    m = (configs.tiny_sw if law == "sw" else configs.tiny_fvw)(nxT=nx, nyT=ny, nzT=nz, precision=precision, fspace=fspace)
    with Solver(m) as s:
        assert s.step_info()["one_launch"] is one_launch
        s.set_profiling(True)
        assert not s.step_info()["one_launch"]
    monkeypatch.setenv("FD3D_OVERLAP", "0")
    with Solver(m) as s:
        assert not s.step_info()["one_launch"]
