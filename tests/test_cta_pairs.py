"""The layer on CTA pairs (256-row UMMA units): experts with even and odd tile counts, full and one-row last tiles, an
expert without rows, widths that end in a narrow tile, against the fp32 oracle (bf16 tolerances of the layer tests)."""
import re
from contextlib import nullcontext

import pytest
import torch

from streamep_b200.models.reference import check_close, moe_reference_grads

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(rows, K, H, I, seed):
    E = len(rows)
    g = torch.Generator(device="cpu").manual_seed(seed)
    pairs = torch.repeat_interleave(torch.arange(E), torch.tensor(rows))
    pairs = pairs[torch.randperm(pairs.numel(), generator=g)]
    T = -(-pairs.numel() // K)
    idx = torch.full((T * K,), -1, dtype=torch.int64)
    idx[:pairs.numel()] = pairs
    idx = idx.view(T, K).to(DEV)
    w = torch.rand(T, K, generator=g).to(DEV)
    x, dy = (torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV) for _ in range(2))
    w1 = (torch.randn(E, 2 * I, H, generator=g) * 0.05).to(torch.bfloat16).to(DEV)
    w2 = (torch.randn(E, H, I, generator=g) * 0.05).to(torch.bfloat16).to(DEV)
    return idx, w, x, dy, w1, w2


WIDE = dict(tile_n_a=256, tile_n_y=256, tile_n_y_bwd=256, tile_n_a_bwd=256, tile_n_dW1=256, tile_n_dW2=256)


@pytest.mark.parametrize("rows,K,H,I,level,capacity", [
    ([256, 512], 1, 256, 128, 0, False),                # full pairs only; one narrow (128-column) output tile
    ([1281, 1408, 2049], 1, 1216, 192, 1, False),       # odd tile counts, one-row last tiles, narrow last column tiles
    ([1537, 0, 1000, 1664], 2, 1288, 520, 2, False),    # empty expert, widths that are no multiple of 32 or 64, odd dW row tiles
    ([1300, 1290, 1410, 1203], 3, 576, 256, 0, True),   # live counts in device memory
    ([4096, 2560, 3073], 2, 1024, 704, 0, True),        # several units per CTA pair
])
def test_layer_on_cta_pairs(native, rows, K, H, I, level, capacity):
    from torch.profiler import ProfilerActivity, profile

    from streamep_b200.models.moe_layer import make_buffer
    from streamep_b200.stream_moe import TileConfig, make_streams, stream_moe_func
    idx, w, x, dy, w1, w2 = _inputs(rows, K, H, I, seed=sum(rows))
    E, T = len(rows), x.shape[0]
    buf = make_buffer(None, T, H, K, E, imbalance=2.0, capacity_factor=1.5 if capacity else None)
    streams = make_streams()
    leaves = [t.clone().requires_grad_(True) for t in (x, w, w1, w2)]
    want_out, *want = moe_reference_grads(x, idx, w, w1, w2, dy)
    for profiled in (False, True, True):
        with profile(activities=[ProfilerActivity.CUDA]) if profiled else nullcontext() as prof:
            # (widths given: a call with few tiles would take narrower ones, which are no pairs)
            out = stream_moe_func(buf, leaves[0], idx, leaves[1], None, leaves[2], leaves[3], streams=streams, num_experts=E,
                                  tile_config=TileConfig(**WIDE), activation_checkpoint_level=level)
            grads = torch.autograd.grad(out, leaves, dy)
            torch.cuda.synchronize()
        buf.check_status()
        for name, got, ref, tol in zip(("out", "dx", "dtopk_weights", "dW1", "dW2"), (out, *grads), (want_out, *want),
                                       (2e-2, 2e-2, 2e-2, 3e-2, 3e-2)):
            check_close(name, got, ref, atol=tol * float(ref.abs().max()), rtol=tol)
    # every GEMM ran on pairs of CTAs (the last template argument), the recomputed pre-activation and the weight gradients too
    gemms = sorted(re.search(r"grouped_gemm_kernel<([^>]*)>", ev.name).group(1) for ev in prof.events() if "grouped_gemm_kernel" in ev.name)
    assert len(gemms) == (5 if level == 0 else 6) and all(re.fullmatch(r"\D*256,.*,\D*2", g) for g in gemms), gemms
