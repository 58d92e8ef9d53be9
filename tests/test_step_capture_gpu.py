"""gf_step runs a kind of step directly until it has come up often enough to be
captured: before, at and past that point, and across a change of parameters
(which drops what was captured), the states equal those of single gf_flac calls
to the last bit, and the node-force terms of a replayed step are not taken for
current ones."""
import numpy as np
import pytest

from geoflac_gb300 import inpgen, new_state
from geoflac_gb300.batch import Batch
from geoflac_gb300.flac import Flac

from ._util import FLOAT_FIELDS, INT_FIELDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("steps", [(15,), (16,), (17, 3), (60, 1, 45)])
def test_steps_equal_single_calls(workdir, mode, steps):
    path = inpgen.extension_60x20().write(str(workdir / f"cap_{mode}_{sum(steps)}.inp"))
    a, b = (Flac(*new_state(path), mode) for _ in range(2))
    for k, n in enumerate(steps):
        a.step(n)
        for _ in range(n):
            b.flac()
        if k == 0:
            for g in (a, b):
                g.params.ifreq_visc = 7
                g.set_params()
    for g in (a, b):  # a fl_node between steps: from the stresses and the mesh as they are
        g.fl_node()
        g.download()
    for f in FLOAT_FIELDS + INT_FIELDS:
        assert np.array_equal(a.state[f], b.state[f]), f
    assert a.clock.time == b.clock.time and a.clock.dt == b.clock.dt
    a.close()
    b.close()


@pytest.mark.parametrize("chunk", [1, 2, 10])
def test_batch_chunks_equal_direct_launches(workdir, chunk):
    """graph_steps > 0 (launched directly at first, then captured) against
    direct launches throughout: 100 steps, so that every chunk is replayed."""
    states = []
    for g in (0, chunk):
        ms = [Flac(*new_state(inpgen.ensemble_member(k, scale=(20, 8, 60, 20))[0].write(
            str(workdir / f"capb_{chunk}_{g}_{k}.inp"))), "mixed") for k in range(3)]
        b = Batch(ms)
        b.set_config(threads=256, items_per_thread=2, ctas_per_sm=1, graph_steps=g)
        b.step(100)
        for m in ms:
            m.download()
        states.append(ms)
        b.close()
    for x, y in zip(*states):
        for f in FLOAT_FIELDS + INT_FIELDS:
            assert np.array_equal(x.state[f], y.state[f]), f
        assert x.clock.time == y.clock.time
