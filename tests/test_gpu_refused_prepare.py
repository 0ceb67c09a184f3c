"""A prepare that refuses its simulations (GB300) has cleared the tables of the one before:
nothing can be launched, collected or read until the next good one, in every engine and at
sizes where the launch looks into them (runs that take new work at a pace, a histogram in
shared memory)."""
import numpy as np
import pytest

from mytrim_gb300 import Engine, SimSpec
from mytrim_gb300 import _ffi as F
from mytrim_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,n", [("fp32", 1), ("fp32", 20 * 152 * 8 * 4), ("fp64", 50)])
def test_refused_prepare_leaves_nothing_to_launch(engine_lib, precision, n):
    good = SimSpec(**{**W.cu_self_ion(n).__dict__, "E": 200.0})
    bad = SimSpec(**{**good.__dict__, "E": -1.0})
    e = Engine(precision=precision, seed=3)
    want = e.run([good])[0]
    e.prepare([good])
    with pytest.raises(F.EngineError):
        e.prepare([bad])
    with pytest.raises(F.EngineError, match="prepare"):
        e.launch()
    with pytest.raises(F.EngineError, match="launched"):
        e.collect()
    with pytest.raises(F.EngineError):
        e.primaries(0, 1)
    got = e.run([good])[0]
    assert got["collisions"] == want["collisions"] > 0
    assert np.array_equal(got["hist_vac"], want["hist_vac"])
    e.close()
