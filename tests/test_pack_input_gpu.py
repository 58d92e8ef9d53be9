"""gf_fno_pack_input writes to any BF16 address: outputs that are not 16-byte
aligned hold the values of aligned ones, and nothing is written beside them."""
import numpy as np
import pytest

from geoflac_gb300.fno import Fno, FnoConfig, _p

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,H,W", [(1, 1, 1), (3, 7, 37), (2, 16, 32)])
@pytest.mark.parametrize("off", [1, 2, 4, 7, 8])
def test_output_addresses(n, H, W, off):
    torch = pytest.importorskip("torch")
    lib = Fno(FnoConfig(H=64, W=128, m1=8, m2=8, layers=1), seed=0).lib
    g = torch.Generator().manual_seed(off)
    raw, prm = torch.randn(n, H, W, 9, generator=g).cuda(), torch.randn(n, 4, generator=g).cuda()
    stats = torch.rand(26, generator=g).add_(0.5).cuda()
    size = n * H * W * 16
    whole = torch.full((size + 64,), 7.0, dtype=torch.bfloat16, device="cuda")
    out = [torch.empty(size, dtype=torch.bfloat16, device="cuda"), whole[off:off + size]]
    for o in out:
        assert lib.gf_fno_pack_input(_p(raw), _p(prm), _p(stats), _p(o), n, H, W, torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(out[0], out[1])
    assert (whole[:off] == 7.0).all() and (whole[off + size:] == 7.0).all()
    st = stats.cpu().numpy()
    got = out[0].view(n, H, W, 16).float().cpu().numpy()
    want = (raw.cpu().numpy() - st[:9]) / st[9:18]
    assert np.abs(got[..., :9] - want).max() <= 2.0 ** -8 * np.abs(want).max()
