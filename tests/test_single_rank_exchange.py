"""The stand-alone exchange of one rank at the edges of its kernels: rows that end inside a copy piece, more pairs per token
than a chunk holds, skipped pairs and tokens, one token, no valid pair; every value against the routing itself (rows are
moved, so the comparison is exact)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("T,H,E,K,skip", [
    (1, 8, 1, 1, 0.0),
    (333, 2056, 8, 3, 0.2),          # row of 257 16-byte pieces
    (1000, 1024, 12, 5, 0.1),        # row of exactly one piece of the combine, half a piece of the push
    (700, 520, 40, 20, 0.5),         # more pairs per token than a chunk
    (64, 128, 64, 32, 0.0),          # a lane per pair
    (50, 64, 4, 2, 1.0),             # nothing is sent
])
def test_single_rank_exchange(native, T, H, E, K, skip):
    from streamep_b200.models.moe_layer import make_buffer
    from streamep_b200.ops.grouped_gemm import compress_pool_to_recv, reexpand_recv_to_pool
    g = torch.Generator(device="cpu").manual_seed(T + H)
    x, dy = (torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV) for _ in range(2))
    idx = torch.rand(T, E, generator=g).topk(K, dim=1).indices
    idx = torch.where(torch.rand(T, K, generator=g) < skip, torch.full_like(idx, -1), idx).to(DEV)
    w = torch.rand(T, K, generator=g).to(DEV)
    buf = make_buffer(None, T, H, K, E)
    valid = idx >= 0
    sent = valid.any(dim=1).nonzero().flatten()
    for _ in range(2):                       # a second pass finds what the first one left behind
        pool, h, _ = buf.dispatch(x, idx, w, None, E)
        grad_pool, count, _ = buf.dispatch_grads(h, dy)
        torch.cuda.synchronize()
        buf.check_status()
        assert h.num_recv_tokens == sent.numel() and torch.equal(h.pool_arrival_count, h.pool_arrival_target)
        assert torch.equal(count, h.pool_arrival_target)
        if sent.numel() == 0:
            continue
        slots = h.recv_token_to_slots.long()
        assert torch.equal(slots >= 0, valid[sent])
        assert torch.equal(h.k_local_total.long(), valid[sent].sum(dim=1)) and torch.equal(h.k_local_remaining, h.k_local_total)
        tok = sent.view(-1, 1).expand(-1, K)[valid[sent]]
        k = torch.arange(K, device=DEV).expand(sent.numel(), K)[valid[sent]]
        s = slots[slots >= 0]
        assert s.unique().numel() == s.numel()
        assert torch.equal(pool[s], x[tok]) and torch.equal(grad_pool[s], dy[tok])
        assert torch.equal(h.pool_topk_weight[s], w[tok, k]) and torch.equal(h.pool_k_slot[s].long(), k)
        assert torch.equal(sent[h.pool_recv_token[s].long()], tok) and torch.equal(h.pool_src[s, 1].long(), tok)
        assert torch.equal(h.tile_id_to_expert[s // 128].long(), idx[tok, k])
        rows = compress_pool_to_recv(pool, h.pool_recv_token, h.num_recv_tokens, buffer=buf)
        assert torch.equal(rows, x[sent])
        again = reexpand_recv_to_pool(rows, h.pool_recv_token, pool.shape[0], buffer=buf)
        assert torch.equal(again[s], x[tok]) and float(again[h.pool_recv_token < 0].float().abs().sum()) == 0.0
        out_rows = buf.alloc_symmetric([sent.numel(), H], torch.bfloat16)
        out_rows.copy_(dy[sent])
        h.y_done_per_token.fill_(1)
        out, _ = buf.combine(out_rows, h, combine_seq=1)
        slot_grads = torch.rand(pool.shape[0], device=DEV)
        dx, dw = buf.combine_grads(out_rows, h, slot_grads, torch.ones(sent.numel(), dtype=torch.int64, device=DEV), dispatch_seq=1)
        torch.cuda.synchronize()
        buf.check_status()
        want = torch.zeros_like(dy)
        want[sent] = dy[sent]
        assert torch.equal(out, want) and torch.equal(dx, want)
        want_dw = torch.zeros_like(w)
        want_dw[tok, k] = slot_grads[s]
        assert torch.equal(dw, want_dw)
