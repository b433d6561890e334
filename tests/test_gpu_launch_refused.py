"""A cooperative launch that the runtime refuses is an error of the call, not a result.

A preloaded stand-in for `cudaLaunchCooperativeKernel` answers some launches with
cudaErrorCooperativeLaunchTooLarge without launching anything, and passes the others on: the
first or a later purification, the spectral bounds of the integer tensor-core path, the levels,
one of two grids while they are being timed. The refused call reports PM7_ERR_CUDA and the next
one works.
"""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent
PM7_ERR_CUDA = 9

FAKE = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
#include <stdlib.h>
struct dim3 { unsigned x, y, z; };
typedef int (*launch_fn)(const void *, struct dim3, struct dim3, void **, size_t, void *);
static int seen = 0;
static int setting(const char *name, int other) { const char *v = getenv(name); return v ? atoi(v) : other; }
int cudaLaunchCooperativeKernel(const void *fn, struct dim3 grid, struct dim3 block, void **args, size_t smem, void *st) {
  const int k = seen++, from = setting("REFUSE_FROM", 1 << 30);
  if (k >= from && k < from + setting("REFUSE_COUNT", 1 << 20)) return 720;
  if ((int)grid.x > setting("REFUSE_ABOVE", 1 << 30)) return 720;
  void *rt = dlopen("libcudart.so.12", RTLD_NOW | RTLD_NOLOAD);
  launch_fn real = rt ? (launch_fn)dlsym(rt, "cudaLaunchCooperativeKernel") : 0;
  return real ? real(fn, grid, block, args, smem, st) : 35;
}
"""

SCRIPT = r"""
import json, sys
sys.path.insert(0, %r)
from pm7b200 import api, geometry as G
out = []
for k in range(2):
    n = int(sys.argv[1])
    z, x = G.water_cluster(n, seed=2) if n > 0 else G.alkane(-n, seed=2)
    try:
        r = api.run_pm7(z, x, want_matrices=0) if n > 0 else api.run_pm7(z[:-1], x[:-1], multiplicity=2, want_matrices=0)
        out.append({"code": 0, "ev": r["total_ev"], "eps": list(r["mo_energies"])})
    except api.Pm7Error as e:
        out.append({"code": e.code})
print(json.dumps({"runs": out, "tune": api.autotune_report()}))
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    d = tmp_path_factory.mktemp("fake")
    (d / "fake.c").write_text(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", str(d / "fake.so"), str(d / "fake.c"), "-ldl"], check=True)
    return str(d / "fake.so")


def _run(size, fake=None, **env):
    e = dict(os.environ)
    for k in ("PM7_AUTOTUNE_CACHE", "PM7_AUTOTUNE_FORCE", "LD_PRELOAD"):
        e.pop(k, None)
    if fake:
        e["LD_PRELOAD"] = fake
    e.update(env)
    p = subprocess.run([sys.executable, "-c", SCRIPT % str(ROOT / "pm7-rs_b200"), str(size)], env=e, timeout=600,
                       capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-2000:]
    return json.loads(p.stdout.strip().splitlines()[-1])


# waters of 270 orbitals: purifications; of 780: bounds of the integer path; a radical of 61: levels alone
@pytest.mark.parametrize("size,first", [(45, 0), (45, 2), (130, 0), (130, 3), (-10, 0)])
def test_refused_launch_raises_and_the_next_call_works(fake, size, first):
    env = {"PM7_AUTOTUNE_FORCE": "sp2_square=0"}
    good = _run(size, **env)["runs"]
    got = _run(size, fake, REFUSE_FROM=str(first), REFUSE_COUNT="1", **env)["runs"]
    assert got[0] == {"code": PM7_ERR_CUDA}
    assert got[1] == good[0] == good[1]


def test_the_tuner_passes_over_a_refused_variant(fake):
    # 666 orbitals: 231 tiles, the larger grid takes every SM
    good = _run(111)
    got = _run(111, fake, REFUSE_ABOVE="147")
    assert got["runs"] == good["runs"]
    assert [v for k, v in got["tune"].items() if "|sp2_square|" in k] == [1]
