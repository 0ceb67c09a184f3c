"""The quadrature's tables belong to a context's device (GB300): a context made after the
device's memory was given up (cudaDeviceReset ends only the process's own context; it
stands in for a second device here) integrates and trains as the first one did."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

CHILD = """
import ctypes
import numpy as np
from mytrim_gb300 import Engine
eps, b = np.array([1e-3, 0.1, 10.0, 3e-3]), np.array([0.5, 1.0, 0.1, 8.0])
got = []
for _ in range(2):
    e = Engine(precision="fp32")
    s2, tau = e.quadrature(eps, b)
    e.surrogate_train(n_train=1024, batch=512, epochs=1, qat_epochs=0, seed=3)
    got.append((s2, tau, e.surrogate_params()))
    e.close()
    assert ctypes.CDLL("libcudart.so.13").cudaDeviceReset() == 0
assert np.all(got[0][0] > 0)
for a, c in zip(*got):
    assert np.array_equal(a, c), (a, c)
print("same")
"""


def test_tables_follow_the_context(engine_lib):
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr[-500:]
