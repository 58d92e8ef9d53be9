"""A batch follows what its members' own calls did between two batch calls:
parameters that change the schedule of a step (against a batch that captures
nothing), parameters kept in the members' device records, and marker counts
(against a batch created after the change).  Everything to the last bit."""
import ctypes as C

import numpy as np
import pytest

from geoflac_gb300 import capi, inpgen
from geoflac_gb300.batch import Batch
from geoflac_gb300.flac import Flac, new_state

from ._util import FLOAT_FIELDS, INT_FIELDS

pytestmark = pytest.mark.gpu


def _members(workdir, tag, n=3):
    return [Flac(*new_state(inpgen.ensemble_member(k, scale=(20, 8, 60, 20))[0].write(
        str(workdir / f"follow_{tag}_{k}.inp"))), "mixed") for k in range(n)]


def _batch(members, graph_steps):
    b = Batch(members)
    b.set_config(threads=256, items_per_thread=2, ctas_per_sm=1, graph_steps=graph_steps)
    return b


def _same(a, b):
    for x, y in zip(a, b):
        x.download()
        y.download()
        for f in FLOAT_FIELDS + INT_FIELDS:
            assert np.array_equal(x.state[f], y.state[f]), f
        assert x.clock.time == y.clock.time and x.clock.dt == y.clock.dt


@pytest.mark.parametrize("change", [dict(istress_therm=1), dict(itemp_bc=2, bot_bc=0.03)])
def test_captured_steps_follow_the_schedule(workdir, change):
    """30 steps one by one (their ordinary kind is captured after eight), then
    the thermal stress, or the flux condition, is switched on and off again."""
    runs = []
    for g in (0, 1):
        ms = _members(workdir, f"{g}_{'_'.join(change)}")
        b = _batch(ms, g)
        b.step(30)
        for m in ms:
            old = {k: getattr(m.params, k) for k in change}
            for k, v in change.items():
                setattr(m.params, k, v)
            m.set_params()
        b.step(7)
        for m in ms:
            for k, v in old.items():
                setattr(m.params, k, v)
            m.set_params()
        b.step(7)
        runs.append(ms)
        b.close()
    _same(*runs)


@pytest.mark.parametrize("graph_steps", [0, 1])
def test_records_follow_the_parameters(workdir, graph_steps):
    """a member whose mesh is held from now on, and the sampled heights' reference"""
    torch = pytest.importorskip("torch")
    ms = _members(workdir, f"rec{graph_steps}")
    b = _batch(ms, graph_steps)
    b.step(30)
    grid = torch.empty((2, 3, 16, 16, 9), dtype=torch.float32, device="cuda")
    b.sample(grid[0], 16, 16)
    held = ms[1]
    before = held.download(capi.F_CORD)["cord"].copy()
    held.params.movegrid = 0
    held.params.z0 += 1000.0
    held.set_params()
    b.sample(grid[1], 16, 16)
    torch.cuda.synchronize()
    lower = (grid[0, ..., 8] - grid[1, ..., 8]).cpu().numpy()
    assert np.abs(lower[1] - 1000.0).max() < 1e-2 and not lower[0].any() and not lower[2].any()
    b.step(3)
    assert np.array_equal(held.download(capi.F_CORD)["cord"], before)
    b.close()


@pytest.mark.parametrize("graph_steps", [0, 1])
def test_marker_tiles_follow_the_marker_count(workdir, graph_steps):
    """Two states whose deep mantle is marked as serpentine (phase 9, mantle
    again where it is hot): one batch is made while the context counts half the
    markers, the other when it counts all."""
    runs = []
    for late in (False, True):
        p, c, s = new_state(inpgen.convergence_60x15().write(str(workdir / f"follow_m{graph_steps}{late}.inp")))
        s["mark_phase"][s["mark_phase"] == 4] = 9
        g = Flac(p, c, s, "mixed")
        n = g.clock.nmarkers
        k = capi.GfClock.from_buffer_copy(g.clock)
        k.nmarkers = n // 2
        b = None
        if not late:
            capi.check(g.lib.gf_set_clock(g.ctx, C.byref(k)), "gf_set_clock")
            b = _batch([g], graph_steps)
            k.nmarkers = n
            capi.check(g.lib.gf_set_clock(g.ctx, C.byref(k)), "gf_set_clock")
        else:
            b = _batch([g], graph_steps)
        b.step(12)
        runs.append([g])
        b.close()
    _same(*runs)
    ph = runs[0][0].state["mark_phase"]
    assert (ph[n // 2:n] == 4).any()
