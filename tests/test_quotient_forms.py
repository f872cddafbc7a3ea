"""The PML quotients of divisors that have no pair with a non-negative low part.

A spacing such as 45.2 or 180.8 m has a signed pair only and 56.3 or 225.2 m none at all; such models take the
two-operation form with the sign put back, or the five-operation one, never FP64 division while
the spacing lies in [2^-20, 2^20].  Every form gives the oracle's bits on every path of a step."""
import ctypes as C

import numpy as np
import pytest

from fd3d_tsn_b200 import abi, configs
from fd3d_tsn_b200.batch import Batch
from fd3d_tsn_b200.slab import SlabSolver
from fd3d_tsn_b200.solver import Solver, lib
from oracle.oracle import MIXED, Oracle
from test_gpu_division import pml_divisors

PAIR, SIGNED, STEPS, EXACT = range(4)


def form(divisor, damping=False):
    f = C.c_int(-1)
    assert lib().fd3d_division_form(C.c_float(divisor), int(damping), C.byref(f)) == 0
    return f.value


def test_no_spacing_in_range_needs_fp64_division():
    spacings = [0.1 * k for k in range(1, 3001)] + [length / cells for length in (40e3, 50e3, 12345.0)
                                                    for cells in range(200, 900)]
    forms = np.array([form(h) for h in spacings])
    assert forms.max() == STEPS
    assert (forms == SIGNED).any() and (forms == STEPS).mean() < 0.01
    assert [form(h) for h in (45.0, 45.2, 40e3 / 650, 56.3, 225.2)] == [PAIR, SIGNED, SIGNED, STEPS, STEPS]
    assert [form(h) for h in (2.0 ** -20, 2.0 ** 20, 2.0 ** -21, 1.5e6, 0.0, -3.0)] == [PAIR, PAIR] + 4 * [EXACT]


def test_damping_divisors_take_a_pair_of_either_sign():
    forms = np.array([form(d, damping=True) for d in np.linspace(1.0, 2.0, 4001)])
    assert set(forms) <= {PAIR, STEPS} and (forms == STEPS).mean() < 0.01


def model(kind, steps=30):
    if kind != "damping":
        return configs.tiny_sw(nxT=36, nyT=11, nzT=22, h=kind, nsteps=steps)
    m = configs.tiny_sw(nxT=36, nyT=11, nzT=22, nsteps=steps)
    fact = m["pml_fact"]
    for k in range(100000):  # the first factor with a 1 + omega that has no pair
        m["pml_fact"] = fact * (1.0 + 1e-4 * k)
        if any(form(d, damping=True) == STEPS for d in pml_divisors(m)):
            return m
    raise AssertionError("no such factor")


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [180.8, 225.2, 1.5e6, "damping"])
def test_every_form_equals_the_oracle(kind):
    steps = 30
    m = model(kind, steps)
    oh, _ = Oracle(m, MIXED).step(steps)
    assert np.abs(oh[:, 0]).max() > 0.0

    def check(history):
        for f in range(4):
            np.testing.assert_array_equal(history(f), oh[:, f], err_msg=f"history field {f}")

    for profiled in (False, True):  # one launch per half-step, and separate launches
        with Solver(m) as s:
            s.set_profiling(profiled)
            s.run(steps)
            s.sync()
            check(s.history)
    with SlabSolver(m, nslabs=2) as s:
        s.run(steps)
        s.sync()
        check(s.history)


@pytest.mark.gpu
@pytest.mark.parametrize("kchunk", [1, 8])
def test_models_of_different_forms_in_one_batch(kchunk):
    """Planes of one make 17.9 K interior items of the large models, so the step takes its
    launches per region; planes of eight one launch per half-step."""
    steps = 12
    models = [model(200.0, steps), model(180.8, steps), model(225.2, steps), model(1.5e6, steps),
              configs.tiny_sw(seed=31, nxT=161, nyT=65, nzT=145, nsteps=steps),
              configs.tiny_sw(seed=32, nxT=150, nyT=60, nzT=210, nsteps=steps, h=112.6)]
    b = Batch(2 << 30, 8)
    b.set_tuning(kchunk, 0)
    slots = []
    for m in models:
        m["history_capacity"] = steps
        slots.append(b.add(m))
    b.run(steps)
    b.sync()
    for m, slot in zip(models, slots):
        oh, _ = Oracle(m, MIXED).step(steps)
        for f in range(4):
            np.testing.assert_array_equal(b.history(slot, f, 0, steps), oh[:, f], err_msg=f"h {m['dh']} field {f}")
    b.close()


@pytest.mark.gpu
def test_forms_match_ieee_on_every_dividend():
    divs = [45.2, 56.3, 112.6, 225.2, 1.83633673, 1.77408087, 11.3, 40e3 / 650]
    arr, bad, first = (C.c_float * len(divs))(*divs), (C.c_ulonglong * len(divs))(), (C.c_uint * len(divs))()
    rc = lib().fd3d_check_division(arr, len(divs), bad, first)
    assert rc == 0, abi.ERRORS.get(rc, rc)
    assert not any(bad), {d: (bad[k], hex(first[k])) for k, d in enumerate(divs) if bad[k]}
