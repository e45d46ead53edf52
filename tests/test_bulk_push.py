"""The stand-alone push through the bulk-copy engine at its edges: the shortest row it takes, chunks of several tokens with a partial last
one, a lane per pair, rows longer than a shared-memory slot, one token, tokens without pairs; every value as in the exchange's test."""
import pytest

import test_single_rank_exchange as exchange

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,H,E,K,skip", [
    (1, 1024, 4, 2, 0.0),
    (1003, 1024, 12, 3, 0.3),        # 8 tokens of 3 pairs a chunk, 3 in the last one
    (517, 1032, 40, 32, 0.2),        # a lane for every pair of one token
    (300, 8200, 8, 2, 0.1),          # rows of 16400 bytes: a second piece of 16 bytes
    (2000, 8192, 8, 4, 0.0),         # rows of exactly one slot, more chunks than warps
    (90, 1536, 4, 2, 1.0),           # nothing is sent
])
def test_bulk_push(native, T, H, E, K, skip):
    exchange.test_single_rank_exchange(native, T, H, E, K, skip)
