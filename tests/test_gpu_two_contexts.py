"""Two contexts in one process (GB300) whose runs stage tables of more than 48 KB in shared
memory: one context's prepare does not take from the other's kernel the shared memory that
it was prepared with."""
import pytest

from mytrim_gb300 import ElementSpec, Engine, LayerSpec, SimSpec

pytestmark = pytest.mark.gpu


def _stack(layers, elements):
    els = [(6 + 2 * k, 12.0 + 4.0 * k) for k in range(layers * elements)]
    return SimSpec(layers=[LayerSpec(100.0, 3.0, [ElementSpec(Z, m, 1.0, 25.0, 3.0) for Z, m in els[k::layers]])
                           for k in range(layers)],
                   Z=79, m=196.967, E=20e3, n_primaries=20)


@pytest.mark.parametrize("precision,large,small", [("fp64", (8, 1), (7, 1)), ("fp32", (8, 4), (7, 4))])
def test_prepare_beside_another_context(engine_lib, precision, large, small):
    a, b = Engine(precision=precision, seed=2), Engine(precision=precision, seed=2)
    want = a.run([_stack(*large)])[0]
    a.prepare([_stack(*large)])
    b.prepare([_stack(*small)])
    a.launch()
    b.launch()
    got, other = a.collect()[0], b.collect()[0]
    assert got["collisions"] == want["collisions"] > 0 and got["vacancies"] == want["vacancies"]
    assert other["collisions"] > 0
    a.close()
    b.close()
