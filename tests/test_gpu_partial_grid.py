"""A run whose grid is not resident as a whole (GB300): a long FP32 run of one block per SM
holds registers that a small FP64 or surrogate run's last blocks need.  Its idle warps
wait for recoils of warps that have started, not for blocks that have not: a cascade of
a few ms is over long before the FP32 run's is, and its tallies are those of a run that
has the GPU to itself.  (Warps that counted on the whole grid sat out their limit of 20 ms
first, every block in its turn.)"""
import numpy as np
import pytest

from mytrim_gb300 import Engine, SimSpec
from mytrim_gb300 import workloads as W
from mytrim_gb300.engine import DATA_DIR

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,E", [("fp64", 2e3), ("surrogate", 80e3)])
def test_small_run_beside_a_long_one(engine_lib, precision, E):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    long_run = SimSpec(**{**W.gold_deposition(4 * sms, voxels=0).__dict__, "E": 2e8})
    small = SimSpec(**{**W.silver_into_silicon(1).__dict__, "E": E})
    e = Engine(precision="fp32", seed=5)
    if precision == "surrogate":
        e.set_surrogate_params(np.load(DATA_DIR / "surrogate_params.npy"))
    e.configure(precision=precision, seed=5)
    want = e.run([small])[0]
    e.prepare([small])
    other = Engine(precision="fp32", seed=6)
    other.run([long_run])
    assert other.stats()["kernel_ms"] > 40.0
    other.prepare([long_run])
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    other.launch(a.cuda_stream)
    e.launch(b.cuda_stream)
    got = e.collect()[0]
    beside = not a.query()
    ms = e.stats()["kernel_ms"]
    other.collect()
    other.close()
    e.close()
    assert beside and ms < 15.0
    for k in ("members", "collisions", "vacancies"):
        assert got[k] == want[k]
    assert np.array_equal(got["hist_vac"], want["hist_vac"])
