"""Which tiles the products of a token block take (csrc/seq_tiles.h)."""
import pytest

from tile_forms import NARROW, PAIR, WIDE, form, waves


@pytest.mark.parametrize("gated", [False, True])
def test_no_form_that_takes_the_chip_longer(gated):
    """A wide tile takes no less time than a narrow one, and a pair's as long as a wide one."""
    for tokens in (65, 128, 129, 256, 257, 300, 517, 900, 1280, 1501, 2048, 4000, 6001):
        for features in list(range(64, 9000, 64)) + [65, 1000, 2050, 4099, 32000, 151936]:
            narrow, wide, pair = waves(gated, tokens, features)
            for blocks in (1, 8, 16, 32, 48, 64, 88):
                f = form(gated, tokens, features, blocks)
                assert f != PAIR or (1 < pair <= wide)
                assert f == NARROW or wide <= 0.8 * narrow
                assert f != NARROW or wide > 0.55 * narrow


@pytest.mark.parametrize("gated,tokens,features,blocks,want", [
    (False, 2048, 8192, 32, PAIR), (False, 2048, 2048, 32, WIDE), (False, 520, 3072, 32, NARROW), (False, 100, 32000, 32, NARROW),
    (False, 900, 4736, 64, WIDE), (True, 900, 2368, 88, WIDE),  # an odd number of feature tiles: pairs would take a wave more
    (False, 2048, 2560, 32, PAIR), (False, 2048, 3072, 8, WIDE), (False, 2048, 6144, 16, PAIR),
    (True, 6001, 4096, 32, WIDE), (True, 6001, 4096, 64, PAIR), (True, 2048, 1536, 16, NARROW), (True, 2048, 1536, 32, PAIR)])
def test_measured_shapes(gated, tokens, features, blocks, want):
    assert form(gated, tokens, features, blocks) == want
