"""A prepare that refuses its simulations (GB300) has cleared the tables of the one before:
nothing can be launched or collected until the next good one, in every engine and at sizes
where the launch looks into them (a histogram in shared memory, runs that take new work at
a pace).  The member records of the run before stay readable."""
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
    if n < 100:
        e.set_record_capacity(10000)
    want = e.run([good])[0]
    records = len(e.records()) if n < 100 else 0
    with pytest.raises(F.EngineError):
        e.prepare([bad])
    with pytest.raises(F.EngineError, match="launched"):
        e.collect()
    if n < 100:
        assert len(e.records()) == records > 0
    e.prepare([good])
    with pytest.raises(F.EngineError):
        e.prepare([bad])
    with pytest.raises(F.EngineError, match="prepare"):
        e.launch()
    with pytest.raises(F.EngineError, match="launched"):
        e.collect()
    got = e.run([good])[0]
    assert got["collisions"] == want["collisions"] > 0
    assert np.array_equal(got["hist_vac"], want["hist_vac"])
    e.close()
