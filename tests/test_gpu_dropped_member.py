"""A member that starts outside the sample (GB300): sampleClusters has no material there, so
it is dropped at its first collision (trim.C:81-83).  Its record says one collision, the
one it was dropped at, and the tallies none, in every engine alike."""
import numpy as np
import pytest

from mytrim_gb300 import ElementSpec, Engine, LayerSpec, SimSpec
from mytrim_gb300 import _ffi as F
from mytrim_gb300.engine import DATA_DIR

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32", "surrogate"])
@pytest.mark.parametrize("n", [1, 100])
def test_dropped_member_record(engine_lib, precision, n):
    cu = LayerSpec(1e3, 8.96, [ElementSpec(29, 63.546, 1.0, 30.0, 3.0)])
    xe = LayerSpec(0.0, 3.0, [ElementSpec(54, 131.29, 1.0, 5.0, 2.0)])
    sim = SimSpec(layers=[cu, xe], Z=29, m=63.546, E=10e3, n_primaries=n, size=(1e3, 1e3, 1e3),
                  pos=(1100.0, 500.0, 500.0), bc=(F.BC_CUT, F.BC_PBC, F.BC_PBC), geometry="clusters",
                  cluster_hash=(4, 4, 4), clusters=np.array([[500.0, 500.0, 500.0, 60.0]]))
    e = Engine(precision="fp32", seed=5)
    if precision == "surrogate":
        e.set_surrogate_params(np.load(DATA_DIR / "surrogate_params.npy"))
    e.configure(precision=precision, seed=5)
    e.set_record_capacity(10 * n)
    tot = e.run([sim])[0]
    rec = e.records()
    e.close()
    assert len(rec) == n and tot["collisions"] == 0 and tot["members"] == n
    assert np.all(rec["ncoll"] == 1)
    assert np.all(rec["nvac"] == 0)
