"""Contiguous inputs that do not start on a 16-byte boundary (views of a flat buffer at an odd element) give what aligned copies of
them give; places that cannot be copied (a GEMM's scatter destination, rows combined in place) are refused on the host."""
import pytest
import torch

from streamep_b200.ops import grouped_gemm as gg

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rows(T, H, seed, shift=0):
    g = torch.Generator(device="cpu").manual_seed(seed)
    flat = torch.empty(T * H + 8, dtype=torch.bfloat16, device=DEV)
    t = flat[shift:shift + T * H].view(T, H)
    t.copy_(torch.randn(T, H, generator=g).to(torch.bfloat16))
    assert t.is_contiguous() and (t.data_ptr() % 16 == 0) == (shift % 8 == 0)
    return t


def _routing(T, E, K):
    return torch.rand(T, E, generator=torch.Generator(device="cpu").manual_seed(3)).topk(K, dim=1).indices.to(DEV)


@pytest.mark.parametrize("level", [0, 2])
def test_layer(native, level):
    from streamep_b200.models.moe_layer import make_buffer
    from streamep_b200.stream_moe import make_streams, stream_moe_func
    T, H, I, E, K = 200, 136, 64, 4, 2
    buf, streams, idx = make_buffer(None, T, H, K, E), make_streams(), _routing(T, E, K)
    g = torch.Generator(device="cpu").manual_seed(1)
    w1, w2 = ((torch.randn(E, a, b, generator=g) * 0.05).to(torch.bfloat16).to(DEV).requires_grad_(True) for a, b in ((2 * I, H), (H, I)))
    w = torch.ones(T, K, device=DEV)

    def run(shift):
        x = _rows(T, H, 2, shift).requires_grad_(True)
        out = stream_moe_func(buf, x, idx, w, None, w1, w2, streams=streams, num_experts=E, activation_checkpoint_level=level)
        # the gradient of `out` arrives as a view at element `shift` of the concatenation's gradient
        both = torch.cat([out.new_zeros(shift), out.flatten()])
        scale = torch.cat([out.new_zeros(shift), _rows(T, H, 4).flatten()])
        grads = torch.autograd.grad((both * scale).sum(), (x, w1, w2))
        torch.cuda.synchronize()
        return (out,) + grads

    for a, b in zip(run(1), run(0)):
        torch.testing.assert_close(a.float(), b.float(), rtol=0, atol=2e-2 * float(b.detach().abs().max()))    # (bf16 sums in any order)


def test_exchange_and_pool_rows(native):
    from streamep_b200.models.moe_layer import make_buffer
    T, H, E, K = 150, 136, 4, 2
    idx, w = _routing(T, E, K), torch.ones(T, K, device=DEV)

    def run(shift):
        buf = make_buffer(None, T, H, K, E)
        pool, h, _ = buf.dispatch(_rows(T, H, 5, shift), idx, w, None, E)
        rows = gg.compress_pool_to_recv(pool, h.pool_recv_token, T, buffer=buf)
        grad_pool, _, _ = buf.dispatch_grads(h, _rows(T, H, 6, shift))
        grads = gg.compress_pool_to_recv(_copy(grad_pool, shift), h.pool_recv_token, T, buffer=buf)
        back = gg.reexpand_recv_to_pool(_copy(rows, shift), h.pool_recv_token, h.TK_padded, buffer=buf)
        h.y_done_per_token.fill_(1)
        out, _ = buf.combine(_rows(T, H, 7, shift), h, combine_seq=1)
        torch.cuda.synchronize()
        buf.check_status()
        return rows, grads, back, out

    for a, b in zip(run(3), run(0)):
        assert torch.equal(a, b)


def _copy(t, shift):
    flat = t.new_empty(t.numel() + 8)
    out = flat[shift:shift + t.numel()].view(t.shape)
    return out.copy_(t)


@pytest.mark.parametrize("tensor_cores", [True, False])
def test_router(native, tensor_cores):
    rt = gg.default_runtime()
    rt.set_router_on_tensor_cores(tensor_cores)
    try:
        a, b = (gg.router_topk(_rows(100, 256, 8, s), _rows(16, 256, 9, s), 4) for s in (1, 0))
    finally:
        rt.set_router_on_tensor_cores(True)
    assert all(torch.equal(u, v) for u, v in zip(a, b))


def test_places_that_cannot_be_moved_are_refused(native):
    from streamep_b200.models.moe_layer import make_buffer
    T, H, I, E, K = 128, 64, 64, 1, 1
    buf = make_buffer(None, T, H, K, E)
    tile, token = torch.zeros(1, dtype=torch.int32, device=DEV), torch.arange(128, dtype=torch.int32, device=DEV)
    w = torch.ones(128, device=DEV)
    with pytest.raises(ValueError, match="16-byte"):
        gg.streaming_moe_y(_rows(128, I, 1), _rows(H, I, 2).view(1, H, I), tile, w, token, o=_rows(128, H, 3, 1), buffer=buf)
    with pytest.raises(ValueError, match="16-byte"):
        gg.streaming_moe_y_bwd(_rows(128, H, 1), _rows(H, I, 2).view(1, H, I), _rows(128, 2 * I, 3, 1), tile, w, token, buffer=buf)
    _, h, _ = buf.dispatch(_rows(T, H, 5), torch.zeros(T, 1, dtype=torch.int64, device=DEV), torch.ones(T, 1, device=DEV), None, E)
    arena = buf.alloc_symmetric([T * H + 8], torch.bfloat16)
    with pytest.raises(ValueError, match="16-byte"):
        buf.combine(arena[1:1 + T * H].view(T, H), h, combine_seq=1)
    torch.cuda.synchronize()
