"""Expert weights beyond half of the L2, whose row tiles are walked in higher bands: full bands, a partial last band and a
band higher than the call, against the fp32 oracle (bf16 tolerances of the layer tests)."""
import pytest
import torch

from streamep_b200.models.reference import check_close, moe_reference_grads

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("T,H,I", [(9000, 4096, 4352), (700, 4096, 4352), (5000, 8456, 4104)])
def test_layer_with_large_experts(native, T, H, I):
    from streamep_b200.models.moe_layer import make_buffer
    from streamep_b200.stream_moe import make_streams, stream_moe_func
    E, K = 2, 1
    assert 2 * (2 * I) * H > 64 << 20
    g = torch.Generator(device="cuda").manual_seed(T)
    new = lambda *shape, std=1.0: torch.empty(shape, dtype=torch.bfloat16, device=DEV).normal_(0.0, std, generator=g)  # noqa: E731
    x, dy, w1, w2 = new(T, H), new(T, H), new(E, 2 * I, H, std=0.02), new(E, H, I, std=0.02)
    idx = torch.randint(0, E, (T, K), generator=g, device=DEV)
    w = torch.rand(T, K, generator=g, device=DEV)
    leaves = [t.clone().requires_grad_(True) for t in (x, w, w1, w2)]
    buf = make_buffer(None, T, H, K, E, imbalance=2.0)
    out = stream_moe_func(buf, leaves[0], idx, leaves[1], None, leaves[2], leaves[3], streams=make_streams(), num_experts=E)
    grads = torch.autograd.grad(out, leaves, dy)
    torch.cuda.synchronize()
    buf.check_status()
    want_out, *want = moe_reference_grads(x, idx, w, w1, w2, dy)
    for name, got, ref, tol in zip(("out", "dx", "dtopk_weights", "dW1", "dW2"), (out, *grads), (want_out, *want),
                                   (2e-2, 2e-2, 2e-2, 3e-2, 3e-2)):
        check_close(name, got, ref, atol=tol * float(ref.abs().max()), rtol=tol)
