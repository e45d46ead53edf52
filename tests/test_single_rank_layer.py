"""The single-rank layer's own dispatch (counting sort + row copies) at the edges of its two forms: one token, one
expert, the largest call that counts inside the placing kernel and the smallest one that does not, many experts, rows
that end inside a copy piece, skipped pairs, no valid pair at all; and a capacity-mode layout that does not fit."""
import pytest
import torch

from streamep_b200.errors import StreamEPOverflow
from streamep_b200.models.reference import check_close, moe_reference_grads

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _run(T, H, I, E, K, seed, skip, level=0, capacity_factor=None):
    from streamep_b200.models.moe_layer import make_buffer
    from streamep_b200.stream_moe import make_streams, stream_moe_func
    g = torch.Generator(device="cpu").manual_seed(seed)
    x, dy = (torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV) for _ in range(2))
    idx = torch.rand(T, E, generator=g).topk(K, dim=1).indices
    idx = torch.where(torch.rand(T, K, generator=g) < skip, torch.full_like(idx, -1), idx).to(DEV)
    w = torch.rand(T, K, generator=g).to(DEV)
    w1 = (torch.randn(E, 2 * I, H, generator=g) * 0.05).to(torch.bfloat16).to(DEV)
    w2 = (torch.randn(E, H, I, generator=g) * 0.05).to(torch.bfloat16).to(DEV)
    buf = make_buffer(None, T, H, K, E, capacity_factor=capacity_factor)
    leaves = [t.clone().requires_grad_(True) for t in (x, w, w1, w2)]
    args = (buf, leaves[0], idx, leaves[1], None, leaves[2], leaves[3])
    out = stream_moe_func(*args, streams=make_streams(), num_experts=E, activation_checkpoint_level=level)
    grads = torch.autograd.grad(out, leaves, dy)
    with torch.no_grad():
        plain = stream_moe_func(*args, streams=make_streams(), num_experts=E)
    torch.cuda.synchronize()
    want = moe_reference_grads(x, idx, w, w1, w2, dy) if bool((idx >= 0).any()) else [torch.zeros_like(t) for t in (x, *leaves)]
    return buf, out, grads, plain, want


@pytest.mark.parametrize("T,H,I,E,K,skip,level", [
    (1, 256, 128, 8, 2, 0.0, 0),
    (300, 256, 128, 1, 1, 0.0, 2),
    (4096, 64, 64, 3, 2, 0.1, 0),        # 8192 pairs: counted inside the placing kernel
    (2731, 64, 64, 5, 3, 0.1, 1),        # 8193 pairs: one more than that
    (700, 2056, 72, 40, 13, 0.3, 2),     # row of 257 16-byte pieces, count matrix over many experts
    (64, 128, 64, 300, 32, 0.0, 0),
    (130, 128, 64, 8, 4, 1.0, 0),        # no valid pair
])
def test_single_rank_layer(native, T, H, I, E, K, skip, level):
    buf, out, grads, plain, (want_out, *want) = _run(T, H, I, E, K, T + E, skip, level)
    buf.check_status()
    # out and dx are sums of K rows, added one by one in bf16: every addition rounds by at most 2^-9 of the partial sum, which
    # the largest result bounds (statistically; inputs are N(0, 1)), so K * 2^-9 once that exceeds the layer tolerance
    sums = max(2e-2, K * 2.0 ** -9)
    for name, got, ref, tol in zip(("out", "dx", "dtopk_weights", "dW1", "dW2", "out without gradients"), (out, *grads, plain),
                                   (want_out, *want, want_out), (sums, sums, 2e-2, 3e-2, 3e-2, sums)):
        check_close(name, got, ref, atol=tol * max(float(ref.abs().max()), 1e-6), rtol=tol)


def test_single_rank_capacity_overflow_runs_empty(native):
    buf, out, grads, _, _ = _run(2000, 128, 64, 4, 2, 3, 0.0, capacity_factor=0.5)
    assert float(out.detach().abs().max()) == 0.0 and all(float(g.abs().max()) == 0.0 for g in grads)
    assert buf.overflow_info()["count"] == 2
    with pytest.raises(StreamEPOverflow, match="capacity overflow"):
        buf.check_status()
