"""Ensemble tiles: a batch with fewer elements than the chip holds threads at
the configured depth is cut finer than configured.  Above that size (2048
threads on each SM, 152 SMs: 622,592 elements at depth 2) depths 1, 2 and 3
(cut to 2) run as different tilings of one kernel, so the states agree to the
last bit; the configuration read back is the one that was set."""
import numpy as np
import pytest

from geoflac_gb300 import inpgen
from geoflac_gb300.batch import Batch
from geoflac_gb300.flac import Flac, clone, new_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nex,nez", [(1013, 631), (60, 20)])  # 639,203 and 1,200 elements
def test_tile_depths_agree(workdir, nex, nez):
    path = inpgen.two_phase_extension(nex, nez, 1e3 * nex, 1e3 * max(nez, 100)).write(str(workdir / f"tiles_{nex}.inp"))
    p, c, s = new_state(path)
    ref = None
    for depth in (1, 2, 3):
        g = Flac(*clone(p, c, s), "mixed")
        b = Batch([g])
        b.set_config(threads=256, items_per_thread=depth, ctas_per_sm=1, graph_steps=0)
        b.step(2)
        assert b.config()["items_per_thread"] == depth
        g.download()
        got = {f: np.copy(g.state[f]) for f in ("cord", "vel", "temp", "stress0", "aps")}
        if ref is None:
            ref = got
        for f in got:
            assert np.array_equal(got[f], ref[f]), f"depth {depth}: {f}"
        b.close()
        g.close()
