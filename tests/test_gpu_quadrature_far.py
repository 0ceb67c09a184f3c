"""The scattering quadrature where the closest approach lies beyond the screening
function's table (GB300): reduced energies from 1e-10 down to 1e-40, turning points from
100 to 400 screening lengths, against the same 256-node rule in numpy.

Allowed: 1e-9 in sin^2(theta/2), as inside the table (the turning point is known to
1e-14, and the node nearest to it makes 1e-9 of one term in 128 of that)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PHI_C = np.array([0.18175, 0.50986, 0.28022, 0.028171])
PHI_D = np.array([3.1998, 0.94229, 0.4029, 0.20162])


def _phi(r):
    return np.exp(-r[..., None] * PHI_D) @ PHI_C


def _reference(eps, b):
    lo, hi = b.copy(), b + 1e3
    for _ in range(120):
        m = 0.5 * (lo + hi)
        up = m * m - _phi(m) * m / eps - b * b > 0
        hi, lo = np.where(up, m, hi), np.where(up, lo, m)
    r0 = 0.5 * (lo + hi)
    u = np.cos((2 * np.arange(1, 129) - 1) * np.pi / 512)[None, :]
    s = np.sqrt(1 - u * u)
    beta2 = ((b / r0) ** 2)[:, None]
    g = np.sqrt(1 - _phi(r0[:, None] / u) * u / (r0 * eps)[:, None] - beta2 * u * u)
    theta = np.pi - 2 * (b / r0) * (np.pi / 256) * (s / g).sum(1)
    return r0, np.sin(theta / 2) ** 2


@pytest.mark.parametrize("lo,hi", [(-18.0, -10.0), (-30.0, -18.0), (-40.0, -26.0)])
def test_turning_point_beyond_the_table(gpu_engine, lo, hi):
    rng = np.random.default_rng(23)
    n = 300
    eps, b = 10 ** rng.uniform(lo, hi, n), rng.uniform(0.0, 200.0, n)
    r0, want = _reference(eps, b)
    assert r0.max() > 160 and want.min() < 0.9
    s2, _ = gpu_engine.quadrature(eps, b)
    assert np.max(np.abs(s2 - want)) <= 1e-9
