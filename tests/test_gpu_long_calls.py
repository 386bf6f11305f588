"""A long mp_step call on a small grid replays a graph of 64 steps from its second 64
on, also as a context's first call; short calls launch their kernels one by one the
first time.  Counted by a library that stands in front of cudaGraphLaunch in a child
process; the fields agree to the bit with the same steps launched in small calls."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

COUNTER = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
static int launches;
int graph_launches(void) { return launches; }
int cudaGraphLaunch(void *exec, void *stream) {
  static int (*real)(void *, void *);
  if (!real) {
    real = (int (*)(void *, void *))dlsym(RTLD_NEXT, "cudaGraphLaunch");
    if (!real) real = (int (*)(void *, void *))dlsym(dlopen("libcudart.so.12", RTLD_NOW), "cudaGraphLaunch");
  }
  ++launches;
  return real(exec, stream);
}
"""

CHILD = r"""
import ctypes, sys
import numpy as np
from mpulse_b200 import abi, runtime
from tests.cases import make_case, random_fields
count = ctypes.CDLL(sys.argv[1]).graph_launches
cfg = make_case("lin_vacuum_cpmlz", abi.MP_FP32)
init = random_fields(cfg, 9, smooth=True)


def run(calls):
    with runtime.Simulation(cfg) as g:
        for n, v in init.items():
            g.upload(n, v)
        before, out = count(), []
        for k in calls:
            g.step(k)
            out.append(count() - before)
            before = count()
        return out, g.time, {n: g.download(n) for n in abi.FIELD_NAMES}


long, t, a = run([2000])
short, u, b = run([50] * 40)
assert t == u == 2000
for n in a:
    np.testing.assert_array_equal(a[n], b[n], err_msg=n)
print(long[0], short[0], short[1:3])
"""


def test_first_long_call_replays_a_graph(tmp_path):
    src, lib = tmp_path / "count.c", tmp_path / "count.so"
    src.write_text(COUNTER)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", str(src), "-o", str(lib), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(lib), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD, str(lib)], cwd=ROOT, env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    # 2000 steps: 64 launched one by one, then 30 replays of 64, the last 16 one by one
    assert r.stdout.split() == ["30", "0", "[1,", "1]"], r.stdout
