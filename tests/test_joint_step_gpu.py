"""Mixed path: a step whose thermal update shares launches with fl_rheol,
fl_node and fl_move (gf_step) against the same step as separate subroutine
calls, over the forms that decide which parts are joined: mesh sizes around
a block, the bottom condition that reads coordinates, a fixed mesh, surface
diffusion between fl_move's parts.

The two are the same device code in differently compiled kernels, so FP32
fields may differ by contraction; after 12 steps they agree at rounding
level, as the ensemble's kernels do: coordinates and temperatures 1e-10,
stresses and velocities 1e-5 of the field's largest value, plastic strain
1e-6, integer fields exact."""
import ctypes as C

import numpy as np
import pytest

from geoflac_gb300 import capi, inpgen
from geoflac_gb300.flac import Flac, new_state

from ._util import FLOAT_FIELDS, INT_FIELDS
from .test_batch_gpu import TOL

pytestmark = pytest.mark.gpu


def _model(path, nex, nez, **kw):
    m = inpgen.two_phase_extension(nex, nez, 5e3 * nex, 5e3 * nez)
    for k, v in kw.items():
        setattr(m, k, v)
    return m.write(path)


def _mixed(path, movegrid):
    p, c, s = new_state(path)
    p.movegrid = movegrid
    return Flac(p, c, s, "mixed")


def _by_calls(g):
    p, k = g.params, g.clock
    g.fl_therm()
    if k.nloop % p.ifreq_rmasses == 0:
        g.change_phase()
    g.fl_rheol()
    g.fl_node()
    g.fl_move()
    if k.nloop % p.ifreq_rmasses == 0:
        g.rmasses()
    if k.nloop % p.ifreq_imasses == 0:
        g.dt_mass()
    g.download(0)
    k.nloop += 1
    k.time += k.dt
    capi.check(g.lib.gf_set_clock(g.ctx, C.byref(k)), "gf_set_clock")


@pytest.mark.parametrize("nex,nez,kw", [
    (60, 20, {}),
    (15, 15, {}),   # 225 elements, 256 nodes: one block
    (16, 16, {}),   # 256 elements, 289 nodes: a block of elements, more of nodes
    (33, 7, {}),
    (200, 60, {}),
    (60, 20, dict(itemp_bc=2, bot_bc=20.0)),
    (60, 20, dict(movegrid=0)),
    (60, 20, dict(topo_kappa=1e-6)),
], ids=lambda v: "_".join(v) if isinstance(v, dict) else str(v))
def test_joint_step_matches_separate_calls(workdir, nex, nez, kw):
    kw = dict(kw)
    move = kw.pop("movegrid", 1)
    path = _model(str(workdir / f"joint_{nex}_{nez}_{'_'.join(kw)}.inp"), nex, nez, **kw)
    a, b = _mixed(path, move), _mixed(path, move)
    a.step(12)
    for _ in range(12):
        _by_calls(b)
    a.download()
    b.download()
    for f in FLOAT_FIELDS + ("temp0",):
        x, y = np.asarray(a.state[f], dtype=np.float64), np.asarray(b.state[f], dtype=np.float64)
        scale = max(float(np.abs(y).max()), 1e-300)
        d = float(np.abs(x - y).max()) / scale
        assert d <= TOL.get(f, 1e-5), f"{f} differs by {d:.3e} of its largest value"
    for f in INT_FIELDS:
        assert np.array_equal(a.state[f], b.state[f]), f
    assert a.clock.nloop == b.clock.nloop and a.clock.nsrate == b.clock.nsrate
    assert a.clock.time == pytest.approx(b.clock.time, rel=1e-6)
    a.close()
    b.close()
