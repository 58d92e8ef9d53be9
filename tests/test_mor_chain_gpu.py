"""diff_topo's MOR columns, done 256 at a time where every erupted height lies
below its element's height and walked in order otherwise, against the oracle's
serial loop: column counts around a chunk, gaps between active columns, and
heights above one and above several elements (rows turned into oceanic crust).
One fl_move; integer fields exact, floating-point fields to the tolerance of the
other comparisons of the magma sub-model (1e-10 of the field's largest value)."""
import numpy as np
import pytest

from geoflac_gb300 import inpgen, new_state
from geoflac_gb300.flac import Flac
from oracle.oracle import Oracle

from ._util import oracle_state
from .test_magma_gpu import _compare

pytestmark = pytest.mark.gpu


def _state(workdir, nex, kind, make):
    m = inpgen.magma_arc(nex, 15)
    p, c, s = make(m.write(str(workdir / f"mor_{nex}_{kind}_{make.__module__.split('.')[-1]}.inp")))
    rng = np.random.default_rng(nex)
    f = s["fmagma2"]
    on = np.ones(nex, bool) if kind != "gaps" else rng.random(nex) < 0.5
    f[2:6, on] = rng.uniform(0.001, 0.01, (4, int(on.sum())))
    s["fmelt"][4, ::3] = 0.02
    # erupted heights of a hundred metres or so (dt is 0.6e9 to 1.7e9 s); rows are 20 km high
    p.prod_magma2 = 0.02 / (0.04 * 1e9)
    if kind == "erupts":
        f[2:6, nex // 2] *= 250.0                     # above its element's height
        f[2:6, min(nex // 2 + 3, nex - 3)] *= 600.0  # above several
    return p, c, s


# nx - 3 = nex - 2 columns (the widest-spaced mesh would fold under an eruption)
@pytest.mark.parametrize("nex,kind", [(n, k) for n in (5, 257, 258, 259, 300) for k in ("all", "gaps", "erupts")
                                      if n > 5 or k != "erupts"])
def test_mor_columns_match_the_serial_loop(workdir, nex, kind):
    p, c, s = _state(workdir, nex, kind, new_state)
    orc = Oracle(*_state(workdir, nex, kind, oracle_state))
    orc.finish_setflac()
    gpu = Flac(p, c, s, "fp64")
    z0 = np.copy(orc.s["cord"][0, :, 1])
    orc.fl_move()
    gpu.fl_move()
    assert np.abs(orc.s["cord"][0, :, 1] - z0).max() > 1.0
    _compare(gpu, orc, f"{kind} {nex}")
    gpu.close()
