"""Recoils sent between warps (GB300): in a run of fewer primaries than warps nearly all
of a cascade is followed by warps that did not start it, so its whole-number tallies must
still be the oracle's on the same random streams, primary by primary -- also with stacks
so short that recoils pass through the overflow lists."""
import numpy as np
import pytest

import oracle_io
from mytrim_gb300 import Engine, SimSpec
from mytrim_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stack", [0, 4])
@pytest.mark.parametrize("n", [1, 5, 40])
def test_few_primaries_equal_oracle(oracle_built, engine_lib, n, stack):
    sim = SimSpec(**{**W.silver_into_silicon(n).__dict__, "E": 60e3})
    e = Engine(precision="fp64", seed=9, stack_capacity=stack)
    got = e.run([sim])[0]
    per = e.primaries(0, n)
    again = e.run([sim])[0]
    e.close()
    want = oracle_io.run(sim, seed=9, philox=True)
    for k in ("members", "collisions", "vacancies", "replacements", "interstitials"):
        assert got[k] == want[k] == again[k], k
    assert np.sum(per["vacancies"]) == want["vacancies"]
    assert np.array_equal(got["hist_vac"], again["hist_vac"])
    assert abs(got["Eel"] + got["Enuc"] - n * 60e3) <= 1e-9 * n * 60e3
