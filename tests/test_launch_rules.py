"""The host's decisions about a launch, host build (oracle/_build/replay_host --rules)."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
QUEUE_FULL, NUMERIC, BUDGET, EVENTS_FULL, LOST_LETTER = 1, 2, 4, 16, 32


def _rules(*lines):
    exe = ROOT / "oracle" / "_build" / "replay_host"
    tables = ROOT / "mytrim_gb300" / "data" / "stopping_tables.tsv"
    r = subprocess.run([str(exe), str(tables), "--rules"], input="\n".join(lines) + "\n", capture_output=True,
                       text=True, check=True)
    return [int(v) for v in r.stdout.split()]


@pytest.mark.parametrize("others", [0, NUMERIC | BUDGET, EVENTS_FULL])
def test_which_runs_are_made_again(oracle_built, others):
    """A full overflow list: with larger ones.  Recoils lost between warps: as it was, the
    lists unchanged.  Nothing else, and neither more than three times."""
    no, same, larger = 0, 1, 2
    for attempt in range(5):
        again = attempt < 3
        want = [no, larger if again else no, same if again else no, larger if again else no]
        got = _rules(*(f"again {others | bits} {attempt}"
                       for bits in (0, QUEUE_FULL, LOST_LETTER, QUEUE_FULL | LOST_LETTER)))
        assert got == want
