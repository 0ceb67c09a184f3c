"""The single-precision cascade kernel's variants (GB300).

A run of one simulation takes the variant that reads its constants as kernel parameters
and its material rows from shared memory; the same simulation among others takes the one
that reads them through pointers.  Both draw the same random numbers, do the same
arithmetic and count a displaced recoil when it starts, so every whole-number tally is
equal: for each feature level, followed and unfollowed recoils, and with stacks so small
that recoils pass through the overflow lists.
"""
import numpy as np
import pytest

from mytrim_gb300 import Engine, SimSpec, _ffi as F
from mytrim_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _arsenic(**k):
    return SimSpec(**{**W.arsenic_implant(300).__dict__, **k})


CASES = {
    "lean": _arsenic(),
    "unfollowed": _arsenic(primaries_only=True),
    "range": _arsenic(mode="range"),
    "generations": _arsenic(mode="primaries", max_generation=2),
    "evac": _arsenic(hist_evac_rows=14),
    "voxels": W.gold_deposition(20, voxels=8),
    "moliere": _arsenic(potential="moliere"),
    "clusters": W.xenon_bubbles(200),
}


def _whole(t):
    return {k: np.asarray(v).tolist() for k, v in t.items() if isinstance(v, (int, np.ndarray)) and k != "status"}


@pytest.mark.parametrize("stack", [0, 8])
@pytest.mark.parametrize("name", sorted(CASES))
def test_alone_equals_among_others(engine_lib, name, stack):
    e = Engine(precision="fp32", seed=11, stack_capacity=stack)
    alone = e.run([CASES[name]])[0]
    among = e.run([CASES[name], W.boron_implant(50)])[0]
    e.close()
    assert alone["members"] > 0
    assert _whole(alone) == _whole(among)


@pytest.mark.parametrize("name", ["lean", "clusters"])
def test_events_alone_equal_among_others(engine_lib, name):
    e = Engine(precision="fp32", seed=11)
    e.set_event_log(range(1, 8), 1 << 23)
    logs = []
    for sims in ([CASES[name]], [CASES[name], SimSpec(**{**W.boron_implant(5).__dict__, "first_primary": 10 ** 6})]):
        e.run(sims)
        ev = e.events()
        ev = ev[ev["sim"] == 0]
        logs.append(np.sort(ev, order=["key", "kind", "x", "y", "z", "E", "gen", "tag", "state"]))
    e.close()
    assert len(logs[0]) == len(logs[1]) > 0
    for f in logs[0].dtype.names:
        if f != "pad":
            assert np.array_equal(logs[0][f], logs[1][f]), f


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_batch_started_by_energy_equals_each_alone(engine_lib, precision):
    """A batch starts its simulations by falling energy; every simulation's primaries keep
    their own streams and tally slots, also beside one without primaries."""
    sims = [W.boron_implant(7), _arsenic(n_primaries=0), W.cu_self_ion(3, E=20e3), _arsenic(n_primaries=5),
            W.cu_self_ion(2, E=80e3), _arsenic(n_primaries=1)]
    e = Engine(precision=precision, seed=12)
    batch = e.run(sims)
    per = e.primaries(0, sum(s.n_primaries for s in sims))
    at = 0
    for i, s in enumerate(sims):
        lead = [_arsenic(n_primaries=0)] * i  # the streams are keyed by the simulation's number
        alone = e.run(lead + [s])[i]
        assert _whole(batch[i]) == _whole(alone), i
        assert per["vacancies"][at:at + s.n_primaries].sum() == alone["vacancies"]
        at += s.n_primaries
    e.close()
