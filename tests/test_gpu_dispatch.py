"""Both sides of every size rule of the step give the same bits.

The step picks kernels by grid size (one launch per half-step with launches overlapped, or
separate launches; 576 or 256 threads per fault tile) and by the divisors of the absorbing
strips (precomputed quotient pairs, or FP64 division).  Profiling always takes the separate
launches, so it is the general path that the others are compared with; where a rule cannot
be switched, the oracle is.  Slip weakening and every same-device comparison are bitwise; the
rate-and-state law against the oracle keeps the tolerances of the parity tests (CUDA
against libm transcendentals)."""
import numpy as np
import pytest

from fd3d_tsn_b200 import configs
from fd3d_tsn_b200.batch import Batch, bytes_needed
from fd3d_tsn_b200.solver import Solver
from oracle.oracle import F64, MIXED, Oracle

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "w", "xx", "yy", "zz", "xy", "yz", "xz")


def everything(s):
    out = {f"history {f}": s.history(f) for f in range(s.nf)}
    out["stations"] = s.stations()
    out.update({n: s.field(n) for n in FIELDS})
    out.update(s.final())
    return out


def same(a, b):
    assert a.keys() == b.keys()
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


# the border lies at 12 CTAs per SM: about 0.9 M cells in single precision, both sides here
@pytest.mark.parametrize("law,precision,fspace,medium3d,size", [
    ("sw", "f32", False, False, (14, 9, 13)),
    ("sw", "f32", False, True, (33, 12, 41)),
    ("sw", "f32", True, False, (65, 17, 26)),
    ("sw", "f64", False, False, (37, 11, 23)),
    ("sw", "f64", True, True, (31, 14, 33)),
    ("fvw", "f32", False, False, (41, 15, 29)),
    ("fvw", "f64", True, False, (40, 13, 28)),
    ("sw", "f32", False, False, (121, 47, 83)),
    ("sw", "f32", False, False, (161, 61, 93)),
    ("sw", "f32", True, True, (129, 55, 87)),
])
def test_one_launch_per_half_step_equals_separate_launches(law, precision, fspace, medium3d, size):
    steps = 37
    nx, ny, nz = size
    make = configs.tiny_sw if law == "sw" else configs.tiny_fvw
    m = make(nxT=nx, nyT=ny, nzT=nz, nsteps=steps, precision=precision, fspace=fspace)
    runs = []
    for profiled in (False, True):
        with Solver(m) as s:
            if medium3d:
                rng = np.random.default_rng(3)
                s.upload_medium_arrays(*(a * (1.0 + 0.05 * rng.uniform(-1.0, 1.0, a.shape)) for a in configs.medium_3d(m)))
            s.set_profiling(profiled)
            s.run(steps)
            s.sync()
            runs.append(everything(s))
    assert np.abs(runs[0]["history 0"]).max() > 0.0, "the model must slip"
    same(*runs)


# 32 x 8 fault tiles: 4 x 37 = 148 of them and a column or a row more
@pytest.mark.parametrize("law,precision", [("sw", "f64"), ("fvw", "f32"), ("fvw", "f64")])
@pytest.mark.parametrize("nx,nz", [(128, 296), (129, 296), (128, 297)])
def test_fault_tiles_on_both_sides_of_the_sm_count(law, precision, nx, nz):
    steps = 12
    make = configs.tiny_sw if law == "sw" else configs.tiny_fvw
    m = make(nxT=nx, nyT=9, nzT=nz, nsteps=steps, precision=precision)
    oh, os_ = Oracle(m, F64 if precision == "f64" else MIXED).step(steps)
    with Solver(m) as s:
        s.run(steps)
        s.sync()
        for f in range(s.nf):
            got, ref = s.history(f), oh[:, f]
            if law == "sw":
                np.testing.assert_array_equal(got, ref, err_msg=f"history field {f}")
            else:
                tol = 1e-9 if precision == "f64" else 1e-5
                assert np.linalg.norm(got - ref) <= tol * np.linalg.norm(ref), f


@pytest.mark.parametrize("precision,fspace,size", [("f32", False, (39, 11, 25)), ("f64", False, (22, 9, 31)),
                                                   ("f32", True, (67, 10, 14))])
def test_layers_filled_on_the_device_equal_the_arrays(precision, fspace, size):
    nx, ny, nz = size
    lay = configs.layered(np.random.default_rng(5), 4, nz * 200.0)
    m = configs.tiny_sw(nxT=nx, nyT=ny, nzT=nz, nsteps=20, precision=precision, fspace=fspace, layers=lay)
    runs = []
    for medium3d in (False, True):
        with Solver(m, medium3d=medium3d) as s:
            assert s.info()["layered_medium"]
            s.run(20)
            s.sync()
            runs.append(everything(s))
    same(*runs)


def test_divisor_without_a_pair_equals_the_oracle():
    """A spacing above 2^20 has no quotient pair: every cell of the strips divides in FP64."""
    steps = 30
    m = configs.tiny_sw(nxT=36, nyT=11, nzT=22, h=1.5e6, nsteps=steps)
    oh, _ = Oracle(m, MIXED).step(steps)
    with Solver(m) as s:
        s.run(steps)
        s.sync()
        for f in range(4):
            np.testing.assert_array_equal(s.history(f), oh[:, f], err_msg=f"history field {f}")


# 120 items per SM of the half-step with the most: planes of one make 17.9 K interior items
# (separate launches), of eight 2.6 K (one launch); slip weakening alone has the wide fault tiles.
# 33 steps are a graph of 32 and one of 1, and one model stops inside the first.
@pytest.mark.parametrize("kchunk", [1, 8])
@pytest.mark.parametrize("law3", ["sw", "fvw"])
def test_batch_launches_equal_single_solves(kchunk, law3):
    third = (configs.tiny_sw if law3 == "sw" else configs.tiny_fvw)(nxT=129, nyT=49, nzT=85, nsteps=33)
    models = [configs.tiny_sw(seed=31, nxT=161, nyT=65, nzT=145, nsteps=33),
              configs.tiny_sw(seed=32, nxT=150, nyT=60, nzT=210, nsteps=17), third]
    for m in models:
        m["history_capacity"] = m["ntfd"]
    tiles = sum(-(-(m["nxt"] - 20) // 32) * -(-(m["nyt"] - 12) // 8) * -(-(m["nzt"] - 12) // kchunk) for m in models)
    assert (tiles > 120 * 148) == (kchunk == 1)
    b = Batch(int(sum(bytes_needed(m) for m in models) * 1.05) + (16 << 20), len(models))
    slots = [b.add(m) for m in models]
    b.set_tuning(kchunk, 0)
    b.run(33)
    b.sync()
    for m, slot in zip(models, slots):
        with Solver(m) as s:
            s.run(m["ntfd"])
            s.sync()
            ref, got = s.final(), b.final(slot)
            same({k: got[k] for k in ref}, ref)
            for f in range(s.nf):
                np.testing.assert_array_equal(b.history(slot, f, 0, m["ntfd"]), s.history(f))
    b.close()
