"""The scattering quadrature (GB300), whose screening function comes from a table of
polynomials, against the same 256-node rule with numpy's exponentials: through the whole
training domain, and where the table ends (distances below 2^-6 and above 2^8).

Allowed: the distance of closest approach is found to 1e-14, and at the node nearest the
turning point, where g^2 is some 1e-5, that leaves 1e-9 of one term in 128: 1e-9 in
sin^2(theta/2).  (The time integral holds sqrt(r0^2 - b^2), which for far collisions says
nothing: a root known to 1e-16 leaves it 1e-8 of r0.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PHI_C = np.array([0.18175, 0.50986, 0.28022, 0.028171])
PHI_D = np.array([3.1998, 0.94229, 0.4029, 0.20162])


def _phi(r):
    return np.exp(-r[..., None] * PHI_D) @ PHI_C


def _reference(eps, b):
    lo, hi = b.copy(), 0.5 * (1 / eps + np.sqrt(1 / eps ** 2 + 4 * b * b)) * (1 + 1e-12)
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
    return np.sin(theta / 2) ** 2


@pytest.mark.parametrize("what", ["domain", "close", "far", "octaves"])
def test_quadrature_against_exponentials(gpu_engine, what):
    rng = np.random.default_rng(17)
    n = 500
    eps, b = 10 ** rng.uniform(-4, 4, n), 12 * np.sqrt(rng.uniform(0, 1, n))
    if what == "close":
        eps, b = 10 ** rng.uniform(1, 4, n), 10 ** rng.uniform(-4, -1.5, n)
    elif what == "far":
        eps, b = 10 ** rng.uniform(-4, -3, n), rng.uniform(100, 300, n)
    elif what == "octaves":
        b = 2.0 ** rng.integers(-6, 9, n) * (1 + rng.integers(-2, 3, n) * 2.0 ** -52)
        eps = np.full(n, 1e4)
    s2, _ = gpu_engine.quadrature(eps, b)
    assert np.max(np.abs(s2 - _reference(eps, b))) <= 1e-9
