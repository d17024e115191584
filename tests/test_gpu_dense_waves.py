"""Dense products on CTA pairs with the tile widths that plan_pair_waves chooses on 74 pairs: two waves of 144 columns (a box of 16 behind two of 64), one wave of 176 (a box
of 48) and of 208 on 1024 rows, two waves of 208 on 1000, and a ragged last column tile behind each."""
import pytest

import test_gpu_pair_tiles as tiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,J,R,rank", [(2048, 2560, 200, 0), (2048, 2560, 128, 16), (1000, 3104, 128, 0), (1024, 3600, 72, 0), (1000, 7680, 64, 0)])
def test_waves_of_narrower_tiles(M, J, R, rank):
    tiles.test_dense_tile_widths(M, J, R, rank)
