"""A mesh test whose launch the driver refuses is an error, not the last answer;
the next one answers as before.  (The refusal: see test_refused_launch_gpu.)"""
import os
import subprocess
import sys

import pytest

from geoflac_gb300 import build

from .test_refused_launch_gpu import SHIM

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes as C, sys
from geoflac_gb300 import inpgen, new_state
from geoflac_gb300.capi import GfError
from geoflac_gb300.flac import Flac
shim, path = sys.argv[1:3]
lib = C.CDLL(shim)
count = C.c_int.in_dll(lib, "refuse_count")
for nex, nez in ((60, 20), (160, 60)):   # one pass; an FP32 pass first
    g = Flac(*new_state(inpgen.two_phase_extension(nex, nez, 1e3 * nex, 1e5).write(path)), "fp64")
    n = count.value
    angle = g.itest_mesh()
    n = count.value - n
    assert n == (1 if nex * nez < 8192 else 2) and 0.0 < angle < 90.0, (n, angle)
    for k in range(n):
        lib.refuse_after(k)
        try:
            g.itest_mesh()
            raise SystemExit(f"launch {k} of {n}: no error")
        except GfError as e:
            assert e.code == -1, e
    lib.refuse_after(-1)
    assert g.itest_mesh() == angle
    g.close()
print("refusals reported")
"""


def test_refused_mesh_test_is_reported(tmp_path):
    src, shim = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    cuda = build._cuda_lib_dir(build._nvcc())
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(shim), str(src), "-L" + cuda, "-Wl,--no-as-needed", "-lcudart",
                    "-Wl,-rpath," + cuda, "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(shim), PYTHONPATH=os.path.dirname(build.HERE))
    r = subprocess.run([sys.executable, "-c", CHILD, str(shim), str(tmp_path / "m.inp")], env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "refusals reported" in r.stdout, r.stdout + r.stderr
