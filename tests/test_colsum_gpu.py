"""Column sums share no scratch: sums issued in turn on several streams equal
those issued one after another, with the caller's scratch and with the call's
own, and so do the gradients of two networks trained side by side."""
import ctypes as C

import pytest

from geoflac_gb300 import capi
from geoflac_gb300.fno import Fno, FnoConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("own", [True, False])
@pytest.mark.parametrize("layout,rows,cols", [(0, 4096, 64), (0, 100001, 256), (1, 50000, 16), (2, 49152, 128), (0, 4095, 7)])
def test_sums_on_several_streams(own, layout, rows, cols):
    torch = pytest.importorskip("torch")
    lib = capi.load_library()
    g = torch.Generator().manual_seed(rows)
    xs = [torch.randn(rows, cols, generator=g).cuda().to(torch.bfloat16 if layout == 1 else torch.float32) for _ in range(4)]
    parts = [torch.empty(1024 * cols, device="cuda") for _ in xs]
    streams = [torch.cuda.Stream() for _ in xs]
    names = ("gf_fno_colsum", "gf_fno_colsum_bf16", "gf_fno_colsum_blocked")

    def call(x, part, out, stream):
        tail = (C.c_void_p(out.data_ptr()), C.c_longlong(rows), cols, 0, C.c_void_p(stream.cuda_stream))
        if own:
            return getattr(lib, names[layout])(C.c_void_p(x.data_ptr()), *tail)
        return lib.gf_fno_colsum_with(C.c_void_p(x.data_ptr()), layout, C.c_void_p(part.data_ptr()), *tail)

    def run(wait):
        outs = [torch.empty(20, cols, device="cuda") for _ in xs]
        torch.cuda.synchronize()
        for k in range(20):
            for x, part, out, s in zip(xs, parts, outs, streams):
                assert call(x, part, out[k], s) == 0
                if wait:
                    s.synchronize()
        torch.cuda.synchronize()
        return outs

    for x, a, b in zip(xs, run(True), run(False)):
        assert torch.equal(a, b)
        # two stages of at most rows / 1024 / (256 / cols) additions in FP32 per thread
        rows_of = x.double().view(rows // 32, cols // 8, 32, 8).transpose(1, 2).reshape(rows, cols) if layout == 2 else x.double()
        bound = 2.0 ** -24 * (rows / 64 + 1200) * rows_of.abs().sum(0)
        assert ((a[0].double() - rows_of.sum(0)).abs() <= bound).all()


def test_two_networks_side_by_side():
    torch = pytest.importorskip("torch")
    cfg = FnoConfig(H=64, W=128, m1=8, m2=8, layers=2)
    g = torch.Generator().manual_seed(5)
    data = [(torch.randn(8, 64, 128, 16, generator=g).to(torch.bfloat16).cuda(), torch.randn(8, 64, 128, 16, generator=g).cuda())
            for _ in range(2)]
    torch.cuda.synchronize()

    def train(streams, together):
        nets, grads = [], [[], []]
        for k, s in enumerate(streams):
            with torch.cuda.stream(s):
                nets.append(Fno(cfg, seed=k))
        torch.cuda.synchronize()
        for it in range(6):
            for k, s in enumerate(streams):
                with torch.cuda.stream(s):
                    x, y = data[k]
                    _, dout = nets[k].loss_grad(nets[k].forward(x, train=True), y)
                    grads[k].append({n: v.clone() for n, v in nets[k].backward(dout).items()})
                    nets[k].adam(lr=1e-3)
                if not together:
                    torch.cuda.synchronize()
        torch.cuda.synchronize()
        return grads

    alone = train([torch.cuda.current_stream()] * 2, False)
    both = train([torch.cuda.Stream(), torch.cuda.Stream()], True)
    for a, b in zip(alone, both):
        for x, y in zip(a, b):
            for n in x:
                assert torch.equal(x[n], y[n]), n
