"""The combine of one rank takes a row in pieces of 32 lanes x 4 vectors while every piece finds a warp of its own, and x 8 beyond: the rule
(CPU), and the values on both sides of its line, at row ends inside and on the edge of a piece (rows are moved: exact)."""
import pytest
import torch

from streamep_b200 import _ext

CASES = [
    (1, 8, 2, 4),
    (64, 1024, 2, 4),        # one piece a row, exactly as many as warps (2 blocks x 32)
    (65, 1024, 2, 8),        # one more: half of a wide piece
    (32, 2048, 2, 4),        # two pieces a row
    (33, 2048, 2, 8),        # exactly one wide piece
    (40, 2056, 2, 8),        # ... and one vector more
    (21, 2056, 2, 4),        # three pieces, the last of one vector
    (1000, 7168, 80, 8),     # the default number of blocks
    (300, 7168, 80, 4),
]


@pytest.mark.parametrize("T,H,blocks,vectors", CASES)
def test_combine_piece_rule(T, H, blocks, vectors):
    assert _ext.load().combine_piece_vectors(T, H, blocks) == vectors


@pytest.mark.gpu
@pytest.mark.parametrize("T,H,blocks,vectors", CASES)
def test_combine_piece_values(native, T, H, blocks, vectors):
    from streamep_b200.models.moe_layer import make_buffer
    g = torch.Generator(device="cpu").manual_seed(T + H)
    E, K = 8, 2
    x, rows = (torch.randn(T, H, generator=g).to(torch.bfloat16).cuda() for _ in range(2))
    idx = torch.rand(T, E, generator=g).topk(K, dim=1).indices.cuda()
    w = torch.rand(T, K, generator=g).cuda()
    buf = make_buffer(None, T, H, K, E)
    _, h, _ = buf.dispatch(x, idx, w, None, E)
    sym = buf.alloc_symmetric([T, H], torch.bfloat16)
    sym.copy_(rows)
    h.y_done_per_token.fill_(1)
    for _ in range(2):
        out, _ = buf.combine(sym, h, combine_seq=1, config=native.Config(blocks, 24, 256, 6, 128))
        torch.cuda.synchronize()
        buf.check_status()
        assert torch.equal(out, rows)
