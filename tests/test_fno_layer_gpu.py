"""The fused kernels of the surrogate's forward pass against the layer-by-layer
products: the same sums in the same order and the same BF16 roundings, so the
outputs and everything kept for the backward pass are the same bits; and the
same forward against the FP64 reference (3e-2, the tolerance of the
layer-by-layer path).  The gradients of the fused backward pass are those of the
products bit for bit too."""
import numpy as np
import pytest

from geoflac_gb300.fno import Fno, FnoConfig, init_params
from oracle import fno_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,m1,m2,B,cin", [(128, 384, 24, 24, 1, 16), (128, 384, 24, 24, 5, 16), (128, 256, 16, 8, 2, 32),
                                             (64, 128, 8, 32, 3, 64), (64, 384, 32, 16, 131, 16)])
def test_fused_forward_equals_the_products(H, W, m1, m2, B, cin):
    torch = pytest.importorskip("torch")
    cfg = FnoConfig(H=H, W=W, m1=m1, m2=m2, cin=cin, layers=3)
    p = {k: (v * (30.0 if k.startswith("R") else 1.0)).astype(np.float32) for k, v in init_params(cfg, seed=3).items()}
    net = Fno(cfg, params=p)
    assert net.fused
    x = torch.randn(B, H, W, cin, generator=torch.Generator().manual_seed(B + W)).to(torch.bfloat16).cuda()
    got = {}
    for fused in (False, True):
        net.fused = fused
        out = net.forward(x)
        assert torch.equal(out, net.forward(x, train=True))
        sv = net.saved
        got[fused] = [out, sv["zp"], sv["h"], sv["vL"], *sv["v"], *sv["z"], *[u[0] for u in sv["spec"]]]
    assert net.lib.gf_gemm_error() == 0
    for a, b in zip(got[False], got[True]):
        assert torch.equal(a.reshape(-1), b.reshape(-1))
    if B <= 2:
        ref = fno_ref.forward_fft(cfg, p, x.float().cpu().numpy())
        assert np.linalg.norm(out.cpu().numpy() - ref) <= 3e-2 * np.linalg.norm(ref)


@pytest.mark.parametrize("H,W,m1,m2,B,cin", [(128, 384, 24, 24, 8, 16), (128, 256, 16, 8, 16, 32), (64, 128, 8, 32, 24, 64),
                                             (64, 384, 32, 16, 136, 16)])
def test_fused_backward_equals_the_products(H, W, m1, m2, B, cin):
    torch = pytest.importorskip("torch")
    cfg = FnoConfig(H=H, W=W, m1=m1, m2=m2, cin=cin, layers=3)
    p = {k: (v * (30.0 if k.startswith("R") else 1.0)).astype(np.float32) for k, v in init_params(cfg, seed=4).items()}
    net = Fno(cfg, params=p)
    g = torch.Generator().manual_seed(B + W)
    x = torch.randn(B, H, W, cin, generator=g).to(torch.bfloat16).cuda()
    y = torch.randn(B, H, W, cfg.cout, generator=g).cuda()
    got = []
    for fused in (False, True):
        net.fused = fused
        out = net.forward(x, train=True)
        _, dout = net.loss_grad(out, y)
        got.append({k: v.clone() for k, v in net.backward(dout).items()})
    assert net.lib.gf_gemm_error() == 0
    for k in got[0]:
        assert torch.equal(got[0][k], got[1][k]), k
