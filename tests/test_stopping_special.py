"""The FP64 stopping's shorter routes at energies that are no ordinary numbers (NaN, the
infinities, zeros, negative and subnormal ones), host build: the bits of the whole
formula, for hydrogen and every heavy ion in every element.  A NaN energy counts as
25 keV/u in the proton formula, as the reference's fmax has it (material.C:134-158)."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_stopping_at_special_energies(oracle_built):
    exe = ROOT / "oracle" / "_build" / "replay_host"
    tables = ROOT / "mytrim_gb300" / "data" / "stopping_tables.tsv"
    r = subprocess.run([str(exe), str(tables), "--stopspecial"], capture_output=True, text=True, check=True)
    assert r.stdout == ""
