"""The tile widths a single-rank layer picks on 148 SMs (CPU; negative = 256 on CTA pairs), at shapes on both sides of the rule."""
import pytest

from streamep_b200 import _ext
from streamep_b200.stream_moe import TileConfig, _resolve_tile_config
from streamep_b200.stream_moe.stream_moe import _native_config


@pytest.mark.parametrize("T,H,I,E,K,want", [
    (512, 2048, 1408, 8, 6, [-256] * 5),                       # 2 to 4 narrow rounds for 2 to 3 of pairs
    (683, 2048, 1408, 8, 6, [-256] * 5),
    (1777, 1000, 520, 12, 3, [-256, -256, 128, -256, -256]),   # (ffn 520: the default width is 128)
    (8192, 2048, 1408, 8, 6, [-256] * 5),
    (16, 2048, 1408, 8, 6, [256, 128, 128, 128, -256]),        # no pairs: one round of 88 or 64 wide tiles
    (384, 2048, 1408, 8, 6, [256, 128, 256, 128, -256]),       # ... 4, 3, 2, 3 narrow rounds for 2, 2, 1, 2
    (256, 2048, 1408, 8, 6, [128, 256, 256, 256, -256]),       # ... 3 for 2, and 2 for 1
    (512, 256, 128, 4, 2, [128, 128, 128, 128, -256]),         # every width in one round
    (1200, 256, 128, 4, 2, [128, 128, 128, 128, -256]),        # ... of pairs
])
def test_layer_widths(T, H, I, E, K, want):
    cfg = _resolve_tile_config(None, I, H)
    assert _ext.load().layer_widths(T, H, I, E, K, 148, _native_config(cfg, True)) == want


def test_given_widths_are_kept():
    cfg = _resolve_tile_config(TileConfig(tile_n_a=128, tile_n_y=256, tile_n_y_bwd=128, tile_n_a_bwd=256, tile_n_dW1=128, tile_n_dW2=128), 1408, 2048)
    assert _ext.load().layer_widths(16, 2048, 1408, 8, 6, 148, _native_config(cfg, False)) == [128, 256, 128, 256, 128]
