"""The bulk-copy push reads rows from 16-byte boundaries: contiguous rows that start elsewhere (a view of a flat buffer at an odd element)
are copied to one first, forward and backward, and give what aligned rows give."""
import pytest
import torch

from streamep_b200.ops import grouped_gemm as gg

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rows(T, H, seed, shift):
    flat = torch.empty(T * H + 8, dtype=torch.bfloat16, device=DEV)
    t = flat[shift:shift + T * H].view(T, H)
    t.copy_(torch.randn(T, H, generator=torch.Generator(device="cpu").manual_seed(seed)).to(torch.bfloat16))
    assert t.is_contiguous() and (t.data_ptr() % 16 == 0) == (shift % 8 == 0)
    return t


@pytest.mark.parametrize("T,H", [(150, 1032), (3, 8200)])       # chunks of seven tokens, rows in two pieces
def test_bulk_push_of_unaligned_rows(native, T, H):
    from streamep_b200.models.moe_layer import make_buffer
    E, K = 4, 2
    idx = torch.rand(T, E, generator=torch.Generator(device="cpu").manual_seed(3)).topk(K, dim=1).indices.to(DEV)
    w = torch.ones(T, K, device=DEV)

    def run(shift):
        buf = make_buffer(None, T, H, K, E)
        pool, h, _ = buf.dispatch(_rows(T, H, 5, shift), idx, w, None, E)
        grads, _, _ = buf.dispatch_grads(h, _rows(T, H, 6, shift))
        got = [gg.compress_pool_to_recv(p, h.pool_recv_token, T, buffer=buf) for p in (pool, grads)]
        torch.cuda.synchronize()
        buf.check_status()
        return got

    want = [_rows(T, H, seed, 0) for seed in (5, 6)]
    for shift in (3, 0):
        assert all(torch.equal(a, b) for a, b in zip(run(shift), want))
