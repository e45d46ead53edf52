"""With NVTX ranges on, a single-rank layer launches the kernels it launches without them: a profile shows the product."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("grad", [True, False])
def test_nvtx_ranges_do_not_change_the_kernels(native, monkeypatch, grad):
    from torch.profiler import ProfilerActivity, profile

    from streamep_b200.models.moe_layer import make_buffer
    from streamep_b200.stream_moe import make_streams, stream_moe, stream_moe_func
    T, H, I, E, K = 300, 512, 256, 4, 2        # few tiles: default widths are narrowed
    buf, streams = make_buffer(None, T, H, K, E), make_streams()
    g = torch.Generator(device="cpu").manual_seed(1)
    x = torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV)
    idx = torch.rand(T, E, generator=g).topk(K, dim=1).indices.to(DEV)
    w = torch.rand(T, K, generator=g).to(DEV)
    w1, w2 = ((torch.randn(E, a, b, generator=g) * 0.05).to(torch.bfloat16).to(DEV).requires_grad_(True) for a, b in ((2 * I, H), (H, I)))
    runs = []
    for nvtx in (False, True):
        monkeypatch.setattr(stream_moe, "_NVTX_ENABLED", nvtx)
        for _ in range(2):                     # (the first round warms the profiler up)
            launches = buf.runtime.launch_count()
            with profile(activities=[ProfilerActivity.CUDA]) as prof, torch.set_grad_enabled(grad):
                out = stream_moe_func(buf, x, idx, w, None, w1, w2, streams=streams, num_experts=E)
                grads = torch.autograd.grad(out, (w1, w2), torch.ones_like(out)) if grad else ()
                torch.cuda.synchronize()
            launches = buf.runtime.launch_count() - launches
        kernels = sorted(ev.name for ev in prof.events() if "sep::" in ev.name)
        runs.append((launches, kernels, grads))
    assert runs[0][1] and runs[0][:2] == runs[1][:2]
    for a, b in zip(runs[0][2], runs[1][2]):
        assert torch.equal(a, b)
