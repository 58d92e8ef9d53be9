"""FP64 fl_therm on meshes around the most nodes that run as one cluster of
16 CTAs (4096) and around the sizes where its CTAs take another warp: bit-exact
with the oracle's serial in-place update, as on the other sweep kernels."""
import pytest

from .test_therm64_gpu import test_fl_therm_equals_the_serial_update as check

pytestmark = pytest.mark.gpu


# nodes: 512 and 528 (a warp, two), 2048 and 2080 (four, five), 4095, 4096, 4160 (no cluster), 9801
@pytest.mark.parametrize("nex,nez", [(15, 31), (15, 32), (31, 63), (31, 64), (62, 64), (63, 63), (64, 63), (98, 98)])
def test_cluster_sweeps_equal_the_serial_update(workdir, nex, nez):
    check(workdir, nex, nez)
