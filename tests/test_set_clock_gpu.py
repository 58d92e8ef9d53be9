"""gf_set_clock writes the clock's scalars and nothing else of the device clock:
a stop code that a call before it left, or that a batch sets right after it, is
reported."""
import ctypes as C

import pytest

from geoflac_gb300 import capi, inpgen
from geoflac_gb300.batch import Batch
from geoflac_gb300.capi import GfError
from geoflac_gb300.flac import Flac, new_state

pytestmark = pytest.mark.gpu


def _model(workdir, tag, mode):
    return Flac(*new_state(inpgen.extension_60x20().write(str(workdir / f"clock_{tag}.inp"))), mode)


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_a_stop_code_survives(workdir, mode):
    g = _model(workdir, mode, mode)
    g.step(3)
    k = capi.GfClock.from_buffer_copy(g.clock)
    capi.check(g.lib.gf_get_clock(g.ctx, C.byref(k)), "gf_get_clock")
    k.time, k.dt, k.vel_max = 1234.5, k.dt * 0.5, 0.25
    g.download(capi.F_VEL)
    g.state["vel"][5, 7] = 1e6  # one step of this folds an element: stop 40
    g.upload(capi.F_VEL)
    g.set_sync(False)
    g.fl_move()
    for _ in range(3):
        capi.check(g.lib.gf_set_clock(g.ctx, C.byref(k)), "gf_set_clock")
    with pytest.raises(GfError) as e:
        g.status()
    assert e.value.code == 40
    got = capi.GfClock()
    capi.check(g.lib.gf_get_clock(g.ctx, C.byref(got)), "gf_get_clock")
    for f in ("time", "dt", "dtavg", "dt_elastic", "dt_maxwell", "dtmax_therm", "frac", "vel_max", "dlmin", "nloop"):
        assert getattr(got, f) == getattr(k, f), f
    g.close()


def test_an_injection_right_after(workdir):
    torch = pytest.importorskip("torch")
    g = _model(workdir, "inject", "mixed")
    b = Batch([g])
    grid = torch.empty((1, 16, 16, 9), dtype=torch.float32, device="cuda")
    b.sample(grid, 16, 16)
    torch.cuda.synchronize()
    fold = grid.clone()
    fold[:, ::2, :, 8] += 5e4  # every other row of points above its upper neighbours
    torch.cuda.synchronize()
    for _ in range(100):
        capi.check(g.lib.gf_set_clock(g.ctx, C.byref(g.clock)), "gf_set_clock")
        with pytest.raises(GfError) as e:
            b.inject(fold, 16, 16)
        assert e.value.code == 41
    b.inject(grid, 16, 16)
    b.close()
    g.close()
