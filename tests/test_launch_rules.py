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


def _pace(precision=1, primaries=100000, warps=4864, sims=1, members=1000.0):
    return _rules(f"pace {precision} {primaries} {warps} {sims} {members}")[0]


def test_pace_of_new_work(oracle_built):
    """12 to 64 primaries per warp in plain FP32 runs of one simulation."""
    assert _pace() == 15
    assert _pace(members=300.0) == 7 and _pace(members=200.0) == 0
    assert [_pace(primaries=4864 * k) for k in (11, 12, 63, 64)] == [0, 15, 15, 0]
    assert [_pace(precision=p) for p in (0, 1, 2)] == [0, 15, 0]
    assert [_pace(sims=n) for n in (1, 2)] == [15, 0]
