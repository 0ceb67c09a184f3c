"""The autotuner's trials (GB300) run the kernel of the run they stand for, not the one that
their own number of primaries would get: a run of 10^7 takes new work without a pace, the
trial's 97,280 launched by themselves with one.  Seen in the collision loop's iterations,
of which a warp at a pace makes 2 % more (As 50 keV, 20 primaries per warp)."""
import pytest

from mytrim_gb300 import Engine
from mytrim_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_trials_take_the_runs_kernel(engine_lib):
    sim = W.arsenic_implant(10_000_000)
    trial = 20 * 152 * 8 * 4
    e = Engine(precision="fp32", seed=4)
    e.autotune([sim], trial_primaries=trial)
    tuned = e.stats()  # of the last trial, a stack of half the depth
    e.close()
    e = Engine(precision="fp32", seed=4)
    e.run([W.arsenic_implant(trial)])
    paced = e.stats()
    e.close()
    assert tuned["collisions"] == paced["collisions"]
    assert tuned["warp_steps"] < 0.99 * paced["warp_steps"]
