"""The widths of the backward launch's tiles where it is a single round (``csrc/loss_bwd.cu``: ``plan_tiles``): as narrow as lets all tiles
run at once, a band's as equal as multiples of 16 channels can be."""
import pytest

from scalingcontrasts_b200._ext import available, native

pytestmark = pytest.mark.skipif(not available(), reason="the native extension is not built")


@pytest.mark.parametrize("ends", [[48, 96, 192, 384, 768], [16, 208, 576, 832], [1024], [16], [64, 128, 192, 256, 320, 384, 448, 512],
                                  [16, 32, 64, 128, 256, 512, 1024, 2048], [4096]])
@pytest.mark.parametrize("rows", [128, 512, 1024, 1152, 2048, 2944, 3072, 18816])
@pytest.mark.parametrize("split", [1, 2])
def test_one_round_takes_the_narrowest_width_that_fits(ends, rows, split):
    tiles, ctas = native().backward_plan(rows, ends, split, 148)
    widths = [end - begin for begin, end in zip([0] + ends[:-1], ends)]
    row_blocks = rows // 128
    if sum(-(-w // 256) for w in widths) * row_blocks * split > 148:
        return  # not a single round
    assert ctas == len(tiles) * row_blocks and ctas * split <= 148 and len(tiles) <= 32
    chosen = next(w for w in range(32, 257, 16)
                  if sum(-(-b // w) for b in widths) * row_blocks * split <= 148 and sum(-(-b // w) for b in widths) <= 32)
    for band, width in enumerate(widths):
        mine = sorted((t[1], t[2]) for t in tiles if t[0] == band)
        assert len(mine) <= -(-width // chosen) and sum(w for _, w in mine) == width
        assert all(w <= chosen and w % 16 == 0 for _, w in mine)
        assert max(w for _, w in mine) - min(w for _, w in mine[:-1] or mine) == 0  # all but the last are alike
