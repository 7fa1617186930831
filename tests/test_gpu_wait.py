"""A line kernel whose tile does not arrive gives up, leaves its outputs alone
and the host says so once; the context works on.

The tile is made not to arrive by tensor maps with boxes of half the lines, so
that fewer bytes come than the kernel waits for: a small library, loaded first,
takes the place of the function that encodes the maps.  It runs in a process of
its own."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SHIM = r"""
#include <dlfcn.h>
#include <cuda.h>
#include "st_internal.h"
extern "C" { int half = 0; void *lib = nullptr; void open_lib(const char *path) { lib = dlopen(path, RTLD_NOW | RTLD_NOLOAD); } }
namespace st {
int line_map(st_ctx *c, CUtensorMap *m, const void *p, bool f32, int dir, int nl, int box) {
    typedef int (*Map)(st_ctx *, CUtensorMap *, const void *, bool, int, int, int);
    const Map real = (Map)dlsym(lib, "_ZN2st8line_mapEP6st_ctxP14CUtensorMap_stPKvbiii");
    return real(c, m, p, f32, dir, half ? nl / 2 : nl, box);
}
}
"""

RUN = r"""
import ctypes, sys, time
sys.path.insert(0, sys.argv[2])
shim = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)
import torch
from shock_turbulence_b200 import Solver, StError, _lib
from shock_turbulence_b200.params import default_params
_lib.load()
shim.open_lib(_lib.LIB_PATH.encode())
half = ctypes.c_int.in_dll(shim, "half")

def case(grid, d, second):
    s = Solver(default_params(*grid))
    F = torch.randn(s.shape, dtype=torch.float64, device="cuda")
    new = lambda: [torch.full_like(F, 7.0) for _ in range(2)]
    def call(o):
        torch.cuda.synchronize()
        if second: getattr(s, f"D2FD{d}2_sym")(F, o[0], o[1], 1)
        else: getattr(s, f"DFD{d}_sym")(F, o[0], 1, 1.0)
    ref = new(); call(ref)
    out = new()
    half.value = 1
    t = time.time()
    try:
        call(out)
        raise SystemExit("no error reported")
    except StError as e:
        assert e.status == -3 and "wait" in str(e), e
    t = time.time() - t
    half.value = 0
    assert t < 20, t
    for o in out: assert bool((o == 7.0).all()), "stored"
    call(out)
    for o, r in zip(out, ref): assert torch.equal(o, r)

for args in (((64, 128, 128), "X", False), ((16, 64, 256), "Y", False), ((512, 64, 64), "X", True), ((32, 32, 64), "Z", True)):
    case(*args)
print("waits ran out")
"""


def test_wait_that_runs_out(tmp_path):
    src, so, run = tmp_path / "shim.cpp", tmp_path / "shim.so", tmp_path / "run.py"
    src.write_text(SHIM)
    run.write_text(RUN)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I/usr/local/cuda/include",
                           "-I" + os.path.join(ROOT, "shock_turbulence_b200", "csrc"), str(src), "-o", str(so), "-ldl"])
    r = subprocess.run([sys.executable, str(run), str(so), ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "waits ran out" in r.stdout, r.stdout + r.stderr
