"""Recoils on a warp's stack (GB300) are written by one lane and read by another, which may
then write the place anew: the members of a few cascades, each of which lives on one warp
or more, come out the same bit for bit however many idle lanes the warp waits for before it
pops, and with a stack so short that places are used over and over."""
import numpy as np
import pytest

from mytrim_gb300 import Engine, SimSpec
from mytrim_gb300 import workloads as W
from mytrim_gb300.engine import DATA_DIR

pytestmark = pytest.mark.gpu


def _members(precision, n, refill, stack):
    sim = SimSpec(**{**W.silver_into_silicon(n).__dict__, "E": 90e3})
    e = Engine(precision="fp32", seed=17)
    if precision == "surrogate":
        e.set_surrogate_params(np.load(DATA_DIR / "surrogate_params.npy"))
    e.configure(precision=precision, seed=17, refill_min_idle=refill, stack_capacity=stack)
    e.set_record_capacity(20000 * n)
    e.run([sim])
    rec = e.records()
    e.close()
    return np.sort(rec, order="key")


@pytest.mark.parametrize("precision", ["fp64", "fp32", "surrogate"])
@pytest.mark.parametrize("n", [1, 6])
def test_members_do_not_depend_on_the_refill(engine_lib, precision, n):
    want = _members(precision, n, 0, 0)
    assert len(want) > 500 * n
    for refill, stack in ((1, 0), (8, 0), (32, 0), (1, 3), (32, 40)):
        got = _members(precision, n, refill, stack)
        assert got.tobytes() == want.tobytes(), (refill, stack)
