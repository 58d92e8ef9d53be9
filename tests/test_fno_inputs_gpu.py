"""What the surrogate's network takes as its input: tensors whose sizes or
strides are not those of [B, H, W, cin] rows are refused by both forward paths,
and a view of wider rows gives the outputs of its copy."""
import pytest

from geoflac_gb300.fno import Fno, FnoConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fused", [True, False])
def test_sizes_and_strides(fused):
    torch = pytest.importorskip("torch")
    cfg = FnoConfig(H=64, W=128, m1=8, m2=8, layers=2)
    net = Fno(cfg, seed=1)
    net.fused = net.fused and fused
    assert net.fused == fused
    wide = torch.randn(2, 64, 128, 32, generator=torch.Generator().manual_seed(2)).to(torch.bfloat16).cuda()
    x = wide[..., :16].contiguous()
    for bad in (x[:, :, :127], x[:, :32], x[..., :8], wide, x.transpose(1, 2), x[:1].expand(2, -1, -1, -1)):
        with pytest.raises(RuntimeError):
            net.forward(bad)
    assert torch.equal(net.forward(wide[..., :16]), net.forward(x))
    assert torch.equal(net.forward(wide[..., ::2]), net.forward(wide[..., ::2].contiguous()))
    assert torch.equal(net.forward(wide[..., :16], train=True), net.forward(x))
    assert torch.equal(net.saved["x"].view(x.shape), x)
