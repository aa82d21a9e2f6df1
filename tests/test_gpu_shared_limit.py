"""Kernels that take more shared memory than the default raise their limit on the device
that they are launched on: the limit is a kernel's on one device, so it is raised again
after the process has moved to another.  With one GPU to run on, cudaGetDevice names
another device while the launches go to the one there is, and the calls that raise the
limit are counted.  GPU only."""
import os
import shutil
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))

COUNTER = """
#include <dlfcn.h>
static int calls = 0, device = 0;
extern "C" int limit_calls() { return calls; }
extern "C" void name_device(int d) { device = d; }
extern "C" int cudaGetDevice(int* d) {
  *d = device;
  return 0;
}
extern "C" int cudaFuncSetAttribute(const void* f, int attr, int value) {
  static auto real = (int (*)(const void*, int, int))dlsym(
      dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD), "cudaFuncSetAttribute");
  if (attr == 8) ++calls;  // cudaFuncAttributeMaxDynamicSharedMemorySize
  return real(f, attr, value);
}
"""

PROGRAM = """
import ctypes as C, sys
sys.path[:0] = [{tests!r}, {root!r}]
import topopt_gb300 as tg
from native import F, I, P, Grid, MgDims, ModalConsts, SumOut
lib, rt, count = tg.lib(), C.CDLL("libcudart.so.13"), C.CDLL({counter!r})
fine, coarse = (256, 128, 128), (128, 64, 64)

def zeros(n):
    p = P()
    assert rt.cudaMalloc(C.byref(p), C.c_size_t(n)) == 0
    assert rt.cudaMemset(p, 0, C.c_size_t(n)) == 0
    return p

g, cd = Grid(*fine), MgDims(*coarse)
ef, x, b, d, y = [zeros(4 * n) for n in (g.nv,) + 4 * (g.ndof,)]
act, mc, out = zeros(g.nnodes), ModalConsts(), SumOut()
for device in (0, 0, 1, 1, 0, 127, 128, 128):
    count.name_device(device)
    for mode in (0, 1, 2):
        n = count.limit_calls()
        lib["_ZN2tg14launch_fine_opIfEEviRKNS_4GridERKNS_11ModalConstsEPKT_PKhS9_S9_S9_S7_PS7_"
            "RKNS_6SumOutEP11CUstream_st"](I(mode), C.byref(g), C.byref(mc), ef, act, x, b, d,
                                           F(0.5), y, C.byref(out), None)
        fine_calls = count.limit_calls() - n
        lib["_ZN2tg12mg_level1_opEiRKNS_6MgDimsES2_RKNS_11ModalConstsEPKfPKhPKiSB_iS7_S7_S7_S7_fPf"
            "SC_P11CUstream_st"](I(mode), C.byref(MgDims(*fine)), C.byref(cd), C.byref(mc), ef, act,
                                 None, None, I(0), None, x, b, d, F(0.5), y, None, None)
        print(mode, fine_calls, count.limit_calls() - n - fine_calls)
assert rt.cudaDeviceSynchronize() == 0 and rt.cudaGetLastError() == 0
"""


def test_the_limit_is_raised_on_every_device(tg, tmp_path):
    src, counter = tmp_path / "counter.cpp", str(tmp_path / "counter.so")
    src.write_text(COUNTER)
    subprocess.run([shutil.which("g++"), "-shared", "-fPIC", "-o", counter, str(src), "-ldl"],
                   check=True)
    code = PROGRAM.format(tests=HERE, root=os.path.dirname(HERE), counter=counter)
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                          env=dict(os.environ, LD_PRELOAD=counter))
    assert done.returncode == 0, done.stderr
    rows = [[int(v) for v in line.split()] for line in done.stdout.splitlines()]
    # Devices 0, 0, 1, 1, 0, 127; beyond 128 of them, at every launch.
    assert rows == [[mode, n, n] for n in (1, 0, 1, 0, 0, 1, 1, 1) for mode in range(3)]
