"""The weight-gradient scheduler's queue on CTA pairs, whose second CTA gets a copy of every entry and reports back: enough units a pair
for the queue to come round many times, runs of experts without rows longer than it, one k-block, a last tile of 40 columns; single CTAs
in the same shape.  Which instance ran shows in the CTAs that issue products (the first of a pair); values against fp32 matmuls."""
import pytest
import torch

from streamep_b200.ops import grouped_gemm as gg

pytestmark = pytest.mark.gpu
DEV = "cuda"

LONG_RUNS = [0] * 20 + [65, 1] + [0] * 12 + [640] + [0] * 9


@pytest.mark.parametrize("rows,M,N,pairs,num_sms", [
    (LONG_RUNS, 1024, 296, True, 4),                      # 344 units a pair
    (([0] * 5 + [70, 0, 1, 200, 0]) * 6, 1024, 512, True, None),      # about 13 units a pair, on every SM
    (LONG_RUNS, 256, 296, False, 4),
])
@pytest.mark.parametrize("dynamic", [True, False])
def test_dw_queue_comes_round(native, rows, M, N, pairs, num_sms, dynamic):
    from streamep_b200.models.moe_layer import make_buffer
    buf = make_buffer(None, 64, 64, 1, 8)
    g = torch.Generator(device="cpu").manual_seed(sum(rows))
    first = torch.tensor([0] + [-(-n // 128) for n in rows]).cumsum(0)
    a, b, a2, b2 = (torch.randn(int(first[-1]) * 128, c, generator=g).to(torch.bfloat16) for c in (M, N, N, M))
    for e, n in enumerate(rows):               # padding rows: zeros where the caller says so, otherwise whatever is there
        for t in (a, b, a2, b2):
            t[int(first[e]) * 128 + n:int(first[e + 1]) * 128] = 0.0 if pairs else float("inf")
    a, b, a2, b2 = (t.to(DEV) for t in (a, b, a2, b2))
    off, freq = first.int().to(DEV), torch.tensor(rows, dtype=torch.int32, device=DEV)
    for timed in (False, True):                # (the claim counter is back at zero for the second one)
        stamps = buf.runtime.set_kernel_timing(timed)
        got = gg.grouped_gemm_dw(a, b, off, freq, lhs2=a2, rhs2=b2, tile_n=256, num_sms=num_sms, dynamic_tiles=dynamic,
                                 padding_is_zero=pairs, buffer=buf)
        torch.cuda.synchronize()
        buf.check_status()
        for out, x, y in ((got[0], a, b), (got[1], a2, b2)):
            for e, n in enumerate(rows):
                s = slice(int(first[e]) * 128, int(first[e]) * 128 + n)
                # one bf16 rounding of an fp32 sum of n products
                torch.testing.assert_close(out[e].float(), x[s].float().t() @ y[s].float(), rtol=2.0 ** -8, atol=max(n, 1) * 2.0 ** -16)
    launch = stamps[0].cpu()
    buf.runtime.set_kernel_timing(False)
    issued = (launch[:, 8] > 0)[launch[:, 0] > 0]          # of a CTA that ran: its thread that issues products had a tile loop
    assert issued.numel() >= 4 and issued.numel() % 2 == 0
    assert issued.tolist() == [not pairs or i % 2 == 0 for i in range(issued.numel())]
