"""Recoils sent between warps with the network (GB300), which do so from 80 keV: in a run of
a few primaries most of a cascade is followed by warps that did not start it.  Collisions,
vacancies and final states, primary by primary, are those of the same primaries in a run
that fills the GPU (a trajectory depends on its key alone), with whole stacks and with
stacks so short that recoils pass through the overflow lists; in the lean variant, with
cluster samples (read through pointers), and with the event log, whose recoils are 64 bytes
instead of 48 and whose vacancy events are as many as the vacancies of each primary."""
import numpy as np
import pytest

from mytrim_gb300 import Engine, SimSpec
from mytrim_gb300 import _ffi as F
from mytrim_gb300 import workloads as W
from mytrim_gb300.engine import DATA_DIR

pytestmark = pytest.mark.gpu


def _run(kind, n, stack, first):
    sim = W.xenon_bubbles(n) if kind == "clusters" else W.silver_into_silicon(n)
    sim = SimSpec(**{**sim.__dict__, "E": 110e3})
    e = Engine(precision="fp32", seed=21)
    e.set_surrogate_params(np.load(DATA_DIR / "surrogate_params.npy"))
    e.configure(precision="surrogate", seed=21, stack_capacity=stack)
    if kind == "events":
        e.set_event_log([F.EV_VACANCY], capacity=5000 * n)
    tot = e.run([sim])[0]
    per = e.primaries(0, first)
    ev = e.events() if kind == "events" else None
    e.close()
    return tot, per, ev


@pytest.fixture(scope="module")
def full(engine_lib):
    return {kind: _run(kind, 8000, 0, 40) for kind in ("lean", "clusters", "events")}


@pytest.mark.parametrize("kind", ["lean", "clusters", "events"])
@pytest.mark.parametrize("stack", [0, 4])
@pytest.mark.parametrize("n", [1, 5, 40])
def test_few_primaries_equal_those_of_a_full_run(full, kind, stack, n):
    tot, per, ev = _run(kind, n, stack, n)
    want = full[kind][1]
    assert per["collisions"].min() > 1000
    for k in ("collisions", "vacancies", "state"):
        assert np.array_equal(per[k], want[k][:n]), k
    assert tot["vacancies"] == per["vacancies"].sum() and tot["collisions"] == per["collisions"].sum()
    if ev is not None:
        assert np.array_equal(np.bincount(ev["primary"].astype(np.int64), minlength=n), per["vacancies"])
