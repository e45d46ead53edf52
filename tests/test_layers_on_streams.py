"""Two layers that share one Buffer, each with its own streams: their backwards run at the same time and neither takes tiles of
the other's weight gradients.  Weight gradients are sums in a fixed order, so they repeat bit by bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def test_backwards_on_independent_streams(native):
    from streamep_b200.models.moe_layer import make_buffer
    from streamep_b200.stream_moe import make_streams, stream_moe_func
    T, H, I, E, K = 4096, 512, 256, 4, 2       # 24 to 96 claimed units a layer: both grids fit the GPU together
    buf = make_buffer(None, T, H, K, E, layers_in_flight=2)
    g = torch.Generator(device="cpu").manual_seed(7)
    rnd = lambda *shape: torch.randn(*shape, generator=g).to(torch.bfloat16).to(DEV)   # noqa: E731
    layers = []
    for _ in range(2):
        idx = torch.rand(T, E, generator=g).topk(K, dim=1).indices.to(DEV)
        layers.append(dict(x=rnd(T, H), idx=idx, w=torch.rand(T, K, generator=g).to(DEV), dy=rnd(T, H), streams=make_streams(),
                           caller=torch.cuda.Stream(), w1=(rnd(E, 2 * I, H) * 0.05).requires_grad_(True),
                           w2=(rnd(E, H, I) * 0.05).requires_grad_(True)))

    def forward(s):
        return stream_moe_func(buf, s["x"], s["idx"], s["w"], None, s["w1"], s["w2"], streams=s["streams"], num_experts=E)

    want = []
    for s in layers:
        want.append(torch.autograd.grad(forward(s), (s["w1"], s["w2"]), s["dy"]))
        torch.cuda.synchronize()
    for _ in range(4):
        outs = []
        for s in layers:
            with torch.cuda.stream(s["caller"]):
                outs.append(forward(s))
        torch.cuda.synchronize()
        got = []
        for s, out in zip(layers, outs):
            with torch.cuda.stream(s["caller"]):
                torch.cuda._sleep(2_000_000)       # both backwards are queued before either starts
                got.append(torch.autograd.grad(out, (s["w1"], s["w2"]), s["dy"]))
        torch.cuda.synchronize()
        buf.check_status()
        for a, b in zip(got, want):
            assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
