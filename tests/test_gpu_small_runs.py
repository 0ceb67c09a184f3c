"""Runs of fewer primaries than resident warps are launched with fewer blocks (GB300).  A
primary's trajectory depends on its key alone, so each primary of a small run, at the sizes
where the number of blocks changes (a multiple of the SMs' warps of one block each) and at
the smallest, comes out as in a run that fills the GPU.  Counts and states are equal; the
per-primary energies are float sums handed over at other collisions, short enough for 1e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spec(n):
    from mytrim_gb300 import ElementSpec, LayerSpec, SimSpec
    cu = LayerSpec(1e7, 8.96, [ElementSpec(29, 63.546, 1.0, 30.0, 3.0)])
    return SimSpec(layers=[cu], Z=29, m=63.546, E=2000.0, n_primaries=n)


@pytest.fixture(scope="module")
def full(engine_lib):
    from mytrim_gb300 import Engine
    e = Engine(precision="fp32", seed=21)
    e.run([_spec(20000)])
    return e.primaries(0, 20000)


@pytest.mark.parametrize("n", [1, 3, 5, 607, 608, 609, 1216, 1217, 4256, 4257, 4864, 4865])
def test_small_runs_equal_the_full_one(full, n):
    from mytrim_gb300 import Engine
    e = Engine(precision="fp32", seed=21)
    e.run([_spec(n)])
    got = e.primaries(0, n)
    for k in ("vacancies", "collisions", "state"):
        assert np.array_equal(got[k], full[k][:n]), k
    for k in ("eel", "enuc"):
        np.testing.assert_allclose(got[k], full[k][:n], rtol=1e-5, err_msg=k)
    for k in ("x", "y", "z"):
        assert np.array_equal(got[k], full[k][:n]), k
