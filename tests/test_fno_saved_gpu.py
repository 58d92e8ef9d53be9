"""A training pass belongs to the weights it was made with: changing them between
forward and backward (by an optimiser step, or in place) leaves the gradients as
they are, on both paths."""
import pytest

from geoflac_gb300.fno import Fno, FnoConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("change", ["adam", "scale"])
@pytest.mark.parametrize("B,fused", [(8, True), (16, True), (8, False)])
def test_weights_may_change_in_between(change, B, fused):
    torch = pytest.importorskip("torch")
    cfg = FnoConfig(H=64, W=128, m1=8, m2=8, layers=2)
    g = torch.Generator().manual_seed(7)
    x = torch.randn(B, 64, 128, 16, generator=g).to(torch.bfloat16).cuda()
    y = torch.randn(B, 64, 128, 16, generator=g).cuda()
    grads = []
    for moved in (False, True):
        net = Fno(cfg, seed=3)
        assert net.fused
        net.fused = fused
        for k, v in net.p.items():
            if k.startswith("R"):
                v *= 30.0
        _, dout = net.loss_grad(net.forward(x, train=True), y)
        net.backward(dout)  # (gradients for the optimiser)
        out = net.forward(x, train=True)
        _, dout = net.loss_grad(out, y)
        if moved:
            if change == "adam":
                net.adam(lr=1e-1)
            else:
                for v in net.p.values():
                    v *= -2.0
        grads.append({k: v.clone() for k, v in net.backward(dout).items()})
    for k in grads[0]:
        assert torch.equal(grads[0][k], grads[1][k]), k
