"""Widths on the edges of the single-rank exchange's kernels: the widest row that the register push takes, the narrowest of the bulk push,
exactly one and one more than one piece of the combine; every value as in the exchange's test."""
import pytest

import test_single_rank_exchange as exchange

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,H,E,K,skip", [
    (700, 1016, 12, 5, 0.1),         # register push: 127 of a warp's 128 vectors
    (50, 1016, 40, 20, 0.3),         # ... and more pairs per token than a chunk
    (700, 1024, 12, 5, 0.1),         # bulk push
    (600, 2048, 12, 5, 0.1),         # a row of exactly one piece of the combine (32 lanes of 8 vectors)
    (333, 2056, 8, 3, 0.2),          # ... and one vector more
])
def test_exchange_edges(native, T, H, E, K, skip):
    exchange.test_single_rank_exchange(native, T, H, E, K, skip)
