"""The weight-gradient GEMM's scheduler and stores at their edges: more empty experts in a row than its queue holds, units of one k-block,
more units than CTAs and fewer, and output widths that end inside a 64-column store, against fp32 matmuls."""
import pytest
import torch

from streamep_b200.ops import grouped_gemm as gg

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rows,M,N,tile_n,pairs,num_sms", [
    ([0] * 20 + [65, 1] + [0] * 12 + [640] + [0] * 9, 256, 296, 256, True, 4),     # last tile of 40 columns
    ([700, 0, 64, 129], 512, 136, 256, True, None),                               # fewer units than CTAs
    ([0] * 17 + [130] + [0] * 9 + [1, 63], 200, 328, 256, False, 3),              # single CTAs, partial row tiles
    ([300, 0, 0, 257], 384, 104, 128, False, 2),
])
@pytest.mark.parametrize("dynamic", [True, False])
def test_dw_units(native, rows, M, N, tile_n, pairs, num_sms, dynamic):
    from streamep_b200.models.moe_layer import make_buffer
    buf = make_buffer(None, 64, 64, 1, 8)
    g = torch.Generator(device="cpu").manual_seed(sum(rows))
    tiles = [-(-n // 128) for n in rows]
    first = torch.tensor([0] + tiles).cumsum(0)
    a, b, a2, b2 = (torch.randn(int(first[-1]) * 128, c, generator=g).to(torch.bfloat16) for c in (M, N, N, M))
    for e, n in enumerate(rows):               # padding rows: zeros where the caller says so, otherwise whatever is there
        for t in (a, b, a2, b2):
            t[int(first[e]) * 128 + n:int(first[e + 1]) * 128] = 0.0 if pairs else float("inf")
    a, b, a2, b2 = (t.to(DEV) for t in (a, b, a2, b2))
    off, freq = first.int().to(DEV), torch.tensor(rows, dtype=torch.int32, device=DEV)
    for _ in range(2):                         # (the claim counter is back at zero)
        got = gg.grouped_gemm_dw(a, b, off, freq, lhs2=a2, rhs2=b2, tile_n=tile_n, num_sms=num_sms, dynamic_tiles=dynamic,
                                 padding_is_zero=pairs, buffer=buf)
        torch.cuda.synchronize()
        buf.check_status()
        for out, x, y in ((got[0], a, b), (got[1], a2, b2)):
            for e, n in enumerate(rows):
                s = slice(int(first[e]) * 128, int(first[e]) * 128 + n)
                want = x[s].float().t() @ y[s].float()
                # one bf16 rounding of an fp32 sum of n products
                torch.testing.assert_close(out[e].float(), want, rtol=2.0 ** -8, atol=max(n, 1) * 2.0 ** -16)
