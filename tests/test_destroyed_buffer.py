"""A backward after ``Buffer.destroy()`` is refused on the host: the autograd node holds the native runtime, whose status block
and tile counters are freed by then."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("capacity", [False, True])
def test_backward_after_destroy_is_refused(native, capacity):
    from streamep_b200.models.moe_layer import make_buffer
    from streamep_b200.stream_moe import make_streams, stream_moe_func
    T, H, I, E, K = 64, 128, 64, 4, 2
    buf = make_buffer(None, T, H, K, E, capacity_factor=2.0 if capacity else None)
    runtime = buf.runtime
    x = torch.randn(T, H, device=DEV).to(torch.bfloat16).requires_grad_(True)
    idx = torch.rand(T, E, device=DEV).topk(K, dim=1).indices
    w1, w2 = (torch.randn(E, a, b, device=DEV).to(torch.bfloat16) for a, b in ((2 * I, H), (H, I)))
    out = stream_moe_func(buf, x, idx, torch.ones(T, K, device=DEV), None, w1, w2, streams=make_streams(), num_experts=E)
    buf.explicitly_destroy = True
    buf.destroy()
    launches = runtime.launch_count()
    with pytest.raises(RuntimeError, match="destroyed"):
        out.backward(torch.ones_like(out))
    assert runtime.launch_count() == launches
    for call in (lambda: runtime.poll_status(True), runtime.barrier, runtime.mark_local_phase,
                 lambda: runtime.alloc_symmetric([8], torch.int32, True)):
        with pytest.raises(ValueError, match="destroyed"):
            call()
    torch.cuda.synchronize()
