"""The single-rank layer under CUDA graph capture (its kernels overlap their set-up with the kernel before them): replays on new
inputs give what a plain call gives."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,K", [(16, 8, 6), (3000, 4, 4)])      # counted inside the placing kernel, and by a launch of its own
def test_layer_in_a_graph(native, T, E, K):
    from streamep_b200.models.moe_layer import make_buffer
    from streamep_b200.stream_moe import make_streams, stream_moe_func
    H, I, dev = 256, 128, "cuda"
    g = torch.Generator(device="cpu").manual_seed(T)
    w1 = (torch.randn(E, 2 * I, H, generator=g) * 0.05).to(torch.bfloat16).to(dev)
    w2 = (torch.randn(E, H, I, generator=g) * 0.05).to(torch.bfloat16).to(dev)
    new = lambda: (torch.randn(T, H, generator=g).to(torch.bfloat16).to(dev), torch.rand(T, E, generator=g).topk(K, dim=1).indices.to(dev),
                   torch.rand(T, K, generator=g).to(dev))      # noqa: E731
    buf, streams = make_buffer(None, T, H, K, E, capacity_factor=2.0), make_streams()
    x, idx, w = new()

    def layer(*a):
        with torch.no_grad():
            return stream_moe_func(buf, *a, None, w1, w2, streams=streams, num_experts=E)
    layer(x, idx, w)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = layer(x, idx, w)
    for _ in range(3):
        x2, idx2, w2_ = new()
        x.copy_(x2), idx.copy_(idx2), w.copy_(w2_)
        graph.replay()
        torch.cuda.synchronize()
        want = layer(x2, idx2, w2_)
        torch.cuda.synchronize()
        # K bf16 additions per element, in an order that differs from run to run
        torch.testing.assert_close(out.float(), want.float(), atol=K * 2.0 ** -8 * float(want.abs().max()), rtol=0)
    buf.check_status()
