"""The bulk-copy push of a single rank on more blocks than the GPU holds, next to a GEMM that waits for its rows on every SM, and twice
along one handle: the blocks that run first have to finish the whole push and leave its counters at zero."""
import pytest
import torch

from streamep_b200.ops import grouped_gemm as gg

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("T,H,K,skip", [
    (3000, 1024, 4, 0.1),     # whole tokens a chunk
    (1500, 8200, 3, 0.1),     # rows in two pieces
    (1, 1024, 2, 0.0),        # one chunk, all other blocks find nothing
])
def test_bulk_push_with_more_blocks_than_sms(native, T, H, K, skip):
    from streamep_b200.models.moe_layer import make_buffer
    I, E = 128, 8
    g = torch.Generator(device="cpu").manual_seed(T + H)
    x, dy = (torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV) for _ in range(2))
    idx = torch.rand(T, E, generator=g).topk(K, dim=1).indices
    idx = torch.where(torch.rand(T, K, generator=g) < skip, torch.full_like(idx, -1), idx).to(DEV)
    w = torch.rand(T, K, generator=g).to(DEV)
    w1 = (torch.randn(E, 2 * I, H, generator=g) * 0.05).to(torch.bfloat16).to(DEV)
    buf = make_buffer(None, T, H, K, E, timeout_ms=5000)
    config = native.Config(2 * torch.cuda.get_device_properties(0).multi_processor_count + 6, 24, 256, 6, 128)
    comm, comp = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):
        with torch.cuda.stream(comm):
            pool, h, ready = buf.dispatch(x, idx, w, None, E, config=config)
        ready.wait_on(comp.cuda_stream, torch.cuda.current_device())
        buf.wait_dispatch_main_started(comp)
        with torch.cuda.stream(comp):
            post, _ = gg.streaming_moe_a(pool, w1, h.tile_id_to_expert, pool_arrival_count=h.pool_arrival_count,
                                         pool_arrival_target=h.pool_arrival_target, tile_n=128, buffer=buf)
        torch.cuda.synchronize()
        buf.check_status()
        assert torch.equal(h.pool_arrival_count, h.pool_arrival_target)
        live = h.pool_recv_token >= 0
        src, k = h.pool_src[live][:, 1].long(), h.pool_k_slot[live].long()
        assert int(live.sum()) == int((idx >= 0).sum()) and torch.equal(pool[live], x[src])
        assert torch.equal(h.pool_topk_weight[live], w[src, k])
        # the rows as they were when the GEMM's gates opened: its results against those of a second run on the finished pool
        again, _ = gg.streaming_moe_a(pool, w1, h.tile_id_to_expert, tile_n=128, buffer=buf)
        assert torch.equal(post[live], again[live])
        with torch.cuda.stream(comm):
            for _ in range(2):
                grads, count, _ = buf.dispatch_grads(h, dy, config=config)
        torch.cuda.synchronize()
        buf.check_status()
        assert torch.equal(grads[live], dy[src]) and torch.equal(count, h.pool_arrival_target)
