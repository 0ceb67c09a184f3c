"""The FP64 collision code's shorter routes, host build: the stopping that takes its
energy-independent parts from the tables equals the whole formula bit for bit, at all
energies and around the limits of each part (the cut reduced velocity, 25 and 1 keV/u)
for every pair of elements; the Newton loop's ratio test equals the rounded quotient's,
also within a few ulps of the threshold."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_stopping_and_ratio_shortcuts_are_exact(oracle_built):
    exe = ROOT / "oracle" / "_build" / "replay_host"
    tables = ROOT / "mytrim_gb300" / "data" / "stopping_tables.tsv"
    r = subprocess.run([str(exe), str(tables), "--stopcheck", "60"], capture_output=True, text=True)
    checked, bad = (int(v) for v in r.stdout.split())
    assert checked == 2 * 60 * 92 * 92
    assert bad == 0
    assert r.returncode == 0
