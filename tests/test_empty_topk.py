"""A layer call without any expert per token (top-0): zeros out, zero gradients, as for a call whose pairs are all skipped."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("level", [0, 2])
def test_layer_without_experts_per_token(native, fused, level):
    from streamep_b200.models.moe_layer import make_buffer
    from streamep_b200.stream_moe import make_streams, stream_moe_func
    T, H, I, E = 70, 128, 64, 4
    buf = make_buffer(None, T, H, 1, E)
    x, w1, w2 = (torch.randn(*s, device=DEV).to(torch.bfloat16).requires_grad_(True) for s in ((T, H), (E, 2 * I, H), (E, H, I)))
    w = torch.empty(T, 0, device=DEV, requires_grad=True)
    out = stream_moe_func(buf, x, torch.empty(T, 0, dtype=torch.int64, device=DEV), w, None, w1, w2, streams=make_streams(), num_experts=E,
                          activation_checkpoint_level=level, fused=fused)
    grads = torch.autograd.grad(out, (x, w, w1, w2), torch.ones_like(out))
    torch.cuda.synchronize()
    buf.check_status()
    assert out.shape == (T, H) and not out.any()
    for g, t in zip(grads, (x, w, w1, w2)):
        assert g.shape == t.shape and not g.any()
