"""A launch that the driver refuses is an error of the call that made it, whether
a step is launched directly, captured, or made of single calls.  The refusal is
made on the host: the child process runs with a stand-in for the runtime's launch
call that, when armed, returns cudaErrorLaunchOutOfResources instead of launching
(the last launch of a step, which moves the elements)."""
import os
import subprocess
import sys

import pytest

from geoflac_gb300 import build

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
static int armed = -1, pending = 0;
int refuse_count = 0;
void refuse_after(int n) { armed = n; }
int cudaLaunchKernelExC(const void *cfg, const void *f, void **args) {
    static int (*real)(const void *, const void *, void **);
    if (!real) real = (int (*)(const void *, const void *, void **))dlsym(RTLD_NEXT, "cudaLaunchKernelExC");
    ++refuse_count;
    if (armed == 0) { armed = -1; return pending = 701; }
    if (armed > 0) --armed;
    return real(cfg, f, args);
}
int cudaGetLastError(void) {
    static int (*real)(void);
    if (!real) real = (int (*)(void))dlsym(RTLD_NEXT, "cudaGetLastError");
    if (pending) { int e = pending; pending = 0; return e; }
    return real();
}
"""

CHILD = r"""
import ctypes as C, sys
from geoflac_gb300 import inpgen, new_state
from geoflac_gb300.capi import GfError
from geoflac_gb300.flac import Flac
mode, shim, path = sys.argv[1:4]
lib = C.CDLL(shim)
count = C.c_int.in_dll(lib, "refuse_count")
g = Flac(*new_state(inpgen.extension_60x20().write(path)), mode)
g.step(3)
n0 = count.value
g.step(1)                  # an ordinary step
n = count.value - n0
assert n >= 4, n
def refused(call):
    lib.refuse_after(n - 1)
    try:
        call()
    except GfError as e:
        lib.refuse_after(-1)
        return e.code == -1
    return False
# launched directly until the kind of step has come up sixteen times, then captured
for k in range(16):
    assert refused(lambda: g.step(1)), k
assert refused(g.flac)
for sync in (True, False):
    g.set_sync(sync)
    n = 1
    assert refused(g.fl_rheol), sync
g.set_sync(True)
try:
    g.step(1)
except GfError as e:
    assert e.code != -1, e
print("refusals reported")
"""


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_refused_launches_are_reported(tmp_path, mode):
    src, shim = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    cuda = build._cuda_lib_dir(build._nvcc())
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(shim), str(src), "-L" + cuda, "-Wl,--no-as-needed", "-lcudart",
                    "-Wl,-rpath," + cuda, "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(shim), PYTHONPATH=os.path.dirname(build.HERE))
    r = subprocess.run([sys.executable, "-c", CHILD, mode, str(shim), str(tmp_path / "m.inp")], env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "refusals reported" in r.stdout, r.stdout + r.stderr
