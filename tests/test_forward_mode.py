"""Forward-mode tangents are refused by the single-rank layer, with and without gradients enabled."""
import pytest
import torch
import torch.autograd.forward_ad as fwad

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(T, H, I, E, K, seed):
    g = torch.Generator(device="cpu").manual_seed(seed)
    x, dy = (torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV) for _ in range(2))
    idx = torch.rand(T, E, generator=g).topk(K, dim=1).indices.to(DEV)
    w = torch.rand(T, K, generator=g).to(DEV)
    w1 = (torch.randn(E, 2 * I, H, generator=g) * 0.05).to(torch.bfloat16).to(DEV)
    w2 = (torch.randn(E, H, I, generator=g) * 0.05).to(torch.bfloat16).to(DEV)
    return x, dy, idx, w, w1, w2


@pytest.mark.parametrize("grad_mode", [True, False])
def test_forward_mode_is_refused(native, grad_mode):
    from streamep_b200.models.moe_layer import make_buffer
    from streamep_b200.stream_moe import make_streams, stream_moe_func
    x, dy, idx, w, w1, w2 = _inputs(64, 128, 64, 4, 2, 0)
    buf = make_buffer(None, 64, 128, 2, 4)
    with fwad.dual_level(), torch.set_grad_enabled(grad_mode), pytest.raises((RuntimeError, NotImplementedError)):
        stream_moe_func(buf, fwad.make_dual(x, dy), idx, w, None, w1, w2, streams=make_streams(), num_experts=4)
    torch.cuda.synchronize()
