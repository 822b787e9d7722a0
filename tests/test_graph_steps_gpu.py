"""bx_advance replays the graphs it captures: the CUDA calls of a call, counted
by a library loaded before the runtime, in a process of its own.  With n steps
per graph bx_advance(n) is one graph launch (and, where the stage kernel ends
the step, one kernel that sets the call's number of steps and time limit), a new
time limit builds no new graph there, and the state after any mix of replayed
and directly launched steps has the same bits."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
static int n[3];
int *bx_counts(void) { return n; }
/* the runtime, which the library under test has loaded by the first call */
#define NEXT(name) \
  static void *f; \
  if (!f) f = dlsym(dlopen("libcudart.so.12", RTLD_LAZY), name);
struct d3 { unsigned x, y, z; };
int cudaGraphLaunch(void *g, void *s) { NEXT("cudaGraphLaunch") n[0]++; return ((int (*)(void *, void *))f)(g, s); }
int cudaGraphInstantiate(void **e, void *g, unsigned long long q) {
  NEXT("cudaGraphInstantiate") n[1]++; return ((int (*)(void **, void *, unsigned long long))f)(e, g, q); }
int cudaLaunchKernel(const void *k, struct d3 a, struct d3 b, void **p, unsigned long m, void *s) {
  NEXT("cudaLaunchKernel") n[2]++;
  return ((int (*)(const void *, struct d3, struct d3, void **, unsigned long, void *))f)(k, a, b, p, m, s); }
int cudaLaunchKernelExC(const void *c, const void *k, void **p) {
  NEXT("cudaLaunchKernelExC") n[2]++; return ((int (*)(const void *, const void *, void **))f)(c, k, p); }
"""

CHILD = r"""
import ctypes, json, os, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
shim = ctypes.CDLL(sys.argv[2])
shim.bx_counts.restype = ctypes.POINTER(ctypes.c_int)
c = shim.bx_counts()
from batsrus_b200 import configs, initial
from batsrus_b200.explicit import ExplicitSolver
from batsrus_b200.grid import BlockGrid
from batsrus_b200.param import Scheme

def case(name):
    if name == "roe":
        return configs.uniform_3d_case(2, "Roe", "mc", 1.5, state="blast")[:3]
    if name == "3d":
        return configs.uniform_3d_case(2, "Linde", "mc3", 1.2, state="blast")[:3]
    g = BlockGrid.uniform(int(name[0]), (8, 8, 1) if name == "2d" else (8, 1, 1), (4, 3, 1) if name == "2d" else (7, 1, 1),
                          (0.0,) * 3, (1.0,) * 3, ("periodic",) * 6)
    s = Scheme(nOrder=2, nStage=2, typeFlux="Linde", typeLimiter="mc", limiterBeta=1.5, cfl=0.4, gamma=5.0 / 3.0,
               useDivbSource=name == "2d", useHalfStep=True)
    return g, s, initial.orszag_tang_3d(g)

out = {}
for name in ("3d", "2d", "1d", "roe"):
    g, s, st = case(name)
    x = ExplicitSolver(g, s)
    x.set_state(st)
    x.set_graph_steps(10)
    x.advance(11)  # one step, the capture, one graph
    r = []
    for k, limit in ((10, -1.0), (23, -1.0), (2, -1.0), (20, 1e30)):
        before = [c[i] for i in range(3)]
        x.advance(k, limit)
        r.append([c[i] - before[i] for i in range(3)])
    a, t = x.get_state(), x.time()
    y = ExplicitSolver(g, s)  # the library keeps one context: a new start
    y.set_state(st)
    y.set_graph_steps(1)
    y.advance(66)
    out[name] = dict(counts=r, same=bool(np.array_equal(a, y.get_state())) and list(t) == list(y.time()))
    y.close()
print(json.dumps(out))
"""


def test_calls_replay_whole_graphs(tmp_path):
    (tmp_path / "shim.c").write_text(SHIM)
    (tmp_path / "child.py").write_text(CHILD)
    so = str(tmp_path / "shim.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", so, str(tmp_path / "shim.c"), "-ldl"], check=True)
    r = subprocess.run([sys.executable, str(tmp_path / "child.py"), ROOT, so], capture_output=True, text=True,
                       env=dict(os.environ, LD_PRELOAD=so), timeout=300)
    assert r.returncode == 0, r.stderr
    out = json.loads(r.stdout.splitlines()[-1])
    for name, o in out.items():
        assert o["same"], name
        # [graph launches, graphs built, kernels launched]; Roe's steps are 2 stages and two kernels of bookkeeping
        k = 4 if name == "roe" else 2
        one = 0 if name == "roe" else 1
        assert o["counts"][0] == [1, 0, one], (name, o)
        assert o["counts"][1] == [2, 0, one + 3 * k], (name, o)
        assert o["counts"][2] == [0, 0, one + 2 * k], (name, o)
        if name != "roe":
            assert o["counts"][3] == [2, 0, one], (name, o)
