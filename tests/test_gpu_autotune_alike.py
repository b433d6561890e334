"""A purification whose two grids are the same launch is not timed against itself.

Up to 512 orbitals one wave of CTAs takes all tiles, so both of the tuner's grids are the same: the
first solve of a process then launches exactly what the second does (every other tuned kernel is
pinned, so that it is not timed either).
"""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

SCRIPT = r"""
import json, sys
sys.path.insert(0, %r)
from pm7b200 import api, geometry as G
z, x = G.water_cluster(int(sys.argv[1]), seed=2)
launches, ev = [], []
for k in range(2):
    before = api.launch_count()
    ev.append(api.run_pm7(z, x, want_matrices=0)["total_ev"])
    launches.append(api.launch_count() - before)
print(json.dumps({"launches": launches, "ev": ev, "tune": api.autotune_report()}))
"""


def _run(waters, force):
    env = dict(os.environ)
    env.pop("PM7_AUTOTUNE_CACHE", None)
    env["PM7_AUTOTUNE_FORCE"] = force
    p = subprocess.run([sys.executable, "-c", SCRIPT % str(ROOT / "pm7-rs_b200"), str(waters)], env=env, timeout=600,
                       capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-2000:]
    return json.loads(p.stdout.strip().splitlines()[-1])


@pytest.mark.parametrize("waters", [19, 42, 43, 85])  # 114, 252, 258 and 510 orbitals
def test_first_solve_launches_no_more_than_the_second(waters):
    tuned = {k.split("|")[1] for k in _run(waters, "")["tune"]}
    assert "sp2_square" in tuned
    r = _run(waters, ",".join(f"{k}=0" for k in sorted(tuned - {"sp2_square"})))
    assert r["launches"][0] == r["launches"][1]
    assert r["ev"][0] == r["ev"][1]
