"""Runs of one simulation with 12 to 64 primaries per warp take new work at a pace (GB300).
A primary's trajectory depends on its key alone: the first primaries of such a run, just
under and over the limit, in the lean, the member-record, the event and the cluster
variants, come out as in a small run, which takes work without a pace; so do those of ions that leave
the sample at once (warps out of work before the pace allows more).  Counts, states and
positions are equal; the energies are float sums handed over at other collisions, short enough for 1e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIRST = 2000
WARPS = 152 * 8 * 4


def _spec(kind, n):
    from mytrim_gb300 import ElementSpec, LayerSpec, SimSpec
    from mytrim_gb300 import _ffi as F
    cu = LayerSpec(1e7, 8.96, [ElementSpec(29, 63.546, 1.0, 30.0, 3.0)])
    kw = {}
    if kind == "leaves":
        kw = dict(bc=(F.BC_CUT, F.BC_PBC, F.BC_PBC), pos=(1.0, 0.0, 0.0), dir=(-1.0, 0.0, 0.0), size=(1e7, 1e3, 1e3))
    if kind == "clusters":
        cu = LayerSpec(1e3, 8.96, cu.elements)
        xe = LayerSpec(0.0, 3.0, [ElementSpec(54, 131.29, 1.0, 5.0, 2.0)])
        return SimSpec(layers=[cu, xe], Z=29, m=63.546, E=40e3, n_primaries=n, size=(1e3, 1e3, 1e3),
                       pos=(500.0, 500.0, 500.0), geometry="clusters", cluster_hash=(4, 4, 4),
                       clusters=np.array([[300.0, 500.0, 500.0, 60.0], [560.0, 500.0, 500.0, 40.0]]))
    return SimSpec(layers=[cu], Z=29, m=63.546, E=40e3, n_primaries=n, **kw)


def _run(kind, n):
    from mytrim_gb300 import Engine
    from mytrim_gb300 import _ffi as F
    e = Engine(precision="fp32", seed=33)
    if kind == "records":
        e.set_record_capacity(1000)
    if kind == "events":
        e.set_event_log([F.EV_LOST], capacity=100000)
    e.run([_spec(kind, n)])
    return e.primaries(0, FIRST)


@pytest.mark.parametrize("kind,n", [("lean", 12 * WARPS - 1), ("lean", 12 * WARPS), ("lean", 15 * WARPS + 77),
                                    ("records", 13 * WARPS), ("events", 13 * WARPS), ("clusters", 13 * WARPS),
                                    ("leaves", 12 * WARPS)])
def test_paced_runs_equal_small_ones(engine_lib, kind, n):
    got, want = _run(kind, n), _run(kind, FIRST)
    assert want["collisions"].sum() > 0
    for k in ("vacancies", "collisions", "state"):
        assert np.array_equal(got[k], want[k]), k
    rest = (want["state"] >= 1) & (want["state"] <= 3)  # positions are those of primaries at rest
    for k in ("x", "y", "z"):
        assert np.array_equal(got[k][rest], want[k][rest]), k
    for k in ("eel", "enuc"):
        np.testing.assert_allclose(got[k], want[k], rtol=1e-5, atol=1e-3, err_msg=k)
