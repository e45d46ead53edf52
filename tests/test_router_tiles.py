"""The tensor-core router in each of its tiles: one token, tiles of 16, 64 and 128 tokens, the hidden dimension whole and split over
2 and 8 CTAs, one to four blocks of 128 experts (the tile is capped where the logits of more would not fit), ragged ends."""
import pytest
import torch

from streamep_b200.ops import grouped_gemm as gg

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("T,H,E,K,R,plan", [
    (1, 256, 8, 2, 1, (16, 2, 8)),
    (70, 7168, 512, 8, 8, (16, 8, 3)),
    (3000, 512, 40, 6, 8, (64, 2, 8)),
    (8192 + 5, 2048, 64, 6, 8, (64, 1, 8)),
    (9601, 264, 256, 8, 4, (128, 1, 4)),
    (12001, 136, 384, 4, 2, (64, 1, 3)),
    (5000, 256, 512, 32, 1, (64, 1, 3)),
])
def test_router_tile(native, T, H, E, K, R, plan):
    rt = gg.default_runtime()
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert tuple(rt.router_plan(T, H, E)) == plan
    g = torch.Generator(device="cpu").manual_seed(T)
    x = torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV)
    wg = (torch.randn(E, H, generator=g) * 0.1).to(torch.bfloat16).to(DEV)
    idx, w, in_rank, probs = gg.router_topk(x, wg, K, num_ranks=R, return_probs=True)
    torch.cuda.synchronize()
    assert rt.poll_status(True) == ""
    logits = x.double() @ wg.double().t()
    want = torch.softmax(logits, -1)
    # fp32 sums of H <= 7168 exact products and __expf: a logit of up to ~40 is off by a few 1e-5, and so, relatively, is exp of it
    torch.testing.assert_close(probs.double(), want, rtol=2e-4, atol=1e-7)
    top, order = want.topk(min(K + 1, E), -1)
    clear = torch.ones(T, dtype=torch.bool, device=DEV) if K == E else (top[:, K - 1] / top[:, K] > 1 + 1e-3)
    assert clear.float().mean() > 0.9           # (tokens whose last choice is a near-tie may choose either)
    dense = torch.zeros(T, E, dtype=torch.float64, device=DEV).scatter_(1, idx, w.double())
    rdense = torch.zeros(T, E, dtype=torch.float64, device=DEV).scatter_(1, order[:, :K], top[:, :K] / top[:, :K].sum(-1, keepdim=True))
    torch.testing.assert_close(dense[clear], rdense[clear], rtol=4e-4, atol=1e-7)
    want_rank = torch.zeros(T, R, dtype=torch.bool, device=DEV).scatter_(1, idx // (E // R), True)
    assert torch.equal(in_rank, want_rank)
