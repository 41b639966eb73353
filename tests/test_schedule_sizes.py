"""gray_schedule_words holds all that the scheduled forward lays out in it, without a GPU: the header, an
estimate, five words of work order and a frontier per block tile, and the super-tiles' coarse frontiers.
(A buffer that is too small loses the frontiers or the whole schedule without an error.)"""
import pytest

from gray_gb300 import batch

HEADER, ESTIMATE, ORDER, SUPER, SUPER_WORDS = 64, 1, 5, 4, 1 + 255 * 8


def _ceil(a, b):
    return -(-a // b)


@pytest.mark.parametrize("tile", [(8, 16), (16, 8)])
@pytest.mark.parametrize("size", [(1, 1), (7, 5), (8, 16), (9, 17), (16, 8), (17, 9), (64, 1), (1, 64), (640, 480),
                                  (1001, 333), (1600, 1040), (1920, 1080), (3840, 2160), (7680, 4320)])
def test_schedule_holds_every_part(gray_lib, tile, size):
    frontier = int(batch._bind().gray_frontier_words())
    words = gray_lib.gray_schedule_words(*size)
    for w, h in {size, (max(1, size[0] - 1), size[1]), (size[0], max(1, size[1] // 2)), (1, 1)}:
        tx, ty = _ceil(w, tile[0]), _ceil(h, tile[1])
        need = HEADER + tx * ty * (ESTIMATE + ORDER + frontier) + _ceil(tx, SUPER) * _ceil(ty, SUPER) * SUPER_WORDS
        assert words >= need, (w, h)
