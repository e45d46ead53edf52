"""What several ranks run on CTA pairs: the pushes fused into GEMM-A and GEMM-Y_bwd, the scatter into other ranks' landing rows, the
return of dL/dweight and the paired weight gradients, with the ranks emulated on one GPU, against the fp32 oracle."""
from types import SimpleNamespace

import pytest
import torch

from test_layer_local import _check, _make
from streamep_b200.models.reference import check_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,tokens,H,I,E,K,level,capacity,push_ctas", [
    (2, 1000, 512, 256, 4, 2, 0, False, 0),                  # every CTA pushes and multiplies
    (2, [1500, 901], 504, 264, 4, 2, 1, False, 5),           # odd tile counts, ragged widths; an odd number of push-only CTAs
    (4, [1100, 700, 0, 1300], 512, 256, 4, 2, 2, False, 28), # one expert a rank, a rank without tokens, the pool built again
    (2, 1000, 512, 256, 4, 2, 0, True, 28),                  # live counts in device memory, fixed landing rows
])
def test_fused_ranks_on_cta_pairs(native, R, tokens, H, I, E, K, level, capacity, push_ctas):
    from streamep_b200 import LocalWorld
    from streamep_b200.stream_moe import TileConfig, _resolve_tile_config, moe_backward, moe_forward
    EL = E // R
    w1, w2, xs, idxs, ws, dys = _make(R, tokens, H, I, E, K, seed=21, sentinel_p=0.03)
    world = LocalWorld(R, arena_bytes=256 << 20)
    for b in world.buffers:
        b.runtime.set_push_ctas(push_ctas)
    if capacity:
        world.enable_capacity_mode(tokens, H, K, E, capacity_factor=1.6)
    streams = world.make_streams()
    cfg = _resolve_tile_config(TileConfig(tile_n_a=256, tile_n_y=256, tile_n_y_bwd=256, tile_n_a_bwd=256, tile_n_dW1=256, tile_n_dW2=256), I, H)

    def rank_fn(r, buf):
        ctx = SimpleNamespace()
        w1l, w2l = w1[r * EL:(r + 1) * EL].contiguous(), w2[r * EL:(r + 1) * EL].contiguous()
        out = moe_forward(ctx, streams, buf, xs[r], idxs[r], ws[r], None, w1l, w2l, E, cfg, level, True)
        assert ctx.handle._dispatch_out.num_pairs > 0        # the GEMMs over row tiles run on pairs
        return out, moe_backward(ctx, dys[r])

    # the weight gradients run on pairs where at most 15 % of the slots for 128-row tiles of 2 * I and H would stay empty
    tiles, units = -(-2 * I // 128) + -(-H // 128), -(-2 * I // 256) + -(-H // 256)
    assert 2 * units <= 1.15 * tiles
    for _ in range(2):
        res = world.run(rank_fn)
        torch.cuda.synchronize()
        world.check_status()
        acc = [None, None]
        for r in range(R):
            if xs[r].shape[0]:
                _check(r, res[r][0], res[r][1], xs[r], idxs[r], ws[r], dys[r], w1, w2, EL, acc)
        for i, name in ((2, "dW1"), (3, "dW2")):
            got, want = torch.cat([res[r][1][i] for r in range(R)]), acc[i - 2]
            check_close(name, got, want, atol=3e-2 * float(want.abs().max()), rtol=3e-2)
        del res
