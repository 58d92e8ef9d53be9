"""Batch calls and the members' own calls, each on streams of their own, take
effect in the order they are made: member calls that only enqueue, then a sample,
a residual or an injection; a sample or a backup, then further member calls.
Against the same sequence with a wait after every call, to the last bit."""
import numpy as np
import pytest

from geoflac_gb300 import capi, inpgen
from geoflac_gb300.batch import Batch
from geoflac_gb300.flac import Flac, new_state

pytestmark = pytest.mark.gpu
H, W = 64, 256


@pytest.mark.parametrize("nex,nez", [(60, 20), (700, 210)])
def test_calls_take_effect_in_order(workdir, nex, nez):
    torch = pytest.importorskip("torch")
    path = inpgen.two_phase_extension(nex, nez, 1e3 * nex, 1e3 * max(nez, 100)).write(str(workdir / f"order_{nex}.inp"))
    runs = []
    for wait in (True, False):
        g = Flac(*new_state(path), "mixed")
        b = Batch([g])
        if not wait:
            g.set_sync(False)
        out, grids = [], torch.zeros((6, 1, H, W, 9), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()

        def then():
            if wait:
                torch.cuda.synchronize()

        def member():
            for call in (g.fl_therm, g.fl_rheol, g.fl_node, g.fl_move):
                call()
                then()

        for k in range(3):
            member()
            b.sample(grids[k], H, W)
            then()
        b.backup()
        then()
        member()
        b.sample(grids[3], H, W)
        then()
        member()
        out.append(b.force_residual())
        member()
        b.restore([0])
        b.sample(grids[4], H, W)
        then()
        member()
        torch.cuda.synchronize()
        b.inject(grids[2], H, W)
        b.sample(grids[5], H, W)
        then()
        g.step(3)
        g.status()
        g.download()
        torch.cuda.synchronize()
        runs.append((out, grids.cpu().numpy(), {f: g.state[f].copy() for f in ("cord", "vel", "temp", "stress0", "aps")}))
        b.close()
        g.close()
    (ra, ga, sa), (rb, gb, sb) = runs
    assert np.array_equal(ga, gb)
    assert np.allclose(ra, rb, rtol=1e-12, atol=0.0)  # (sums by atomics)
    for f in sa:
        assert np.array_equal(sa[f], sb[f]), f
