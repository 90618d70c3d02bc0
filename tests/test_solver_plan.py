"""How a job's tiles are split over the GPU (host code, no GPU needed): which of them stay on the
chip, and that every group fits the blocks there are and covers its tile."""
import ctypes as C

import numpy as np
import pytest

from cuphu_b200._lib import check, lib

SMS = 148


def solver_plan(shapes, precision=0, sms=SMS):
    """Per tile: on the chip, blocks of its group, rows and columns of a region in items; and the
    number of blocks launched."""
    n = len(shapes)
    out = np.zeros((n, 4), np.int32)
    r, c = (np.ascontiguousarray([s[k] for s in shapes], dtype=np.int32) for k in (0, 1))
    ip = C.POINTER(C.c_int)
    nblk = lib().cuphu_test_solver_plan(r.ctypes.data_as(ip), c.ctypes.data_as(ip), n, sms,
                                        precision, out.ctypes.data_as(ip))
    check(min(nblk, 0))
    return out, nblk


def _jobs():
    rng = np.random.default_rng(5)
    yield [(1, 1), (1, 40000), (70, 1), (967, 967)]
    for _ in range(40):
        lo, hi = sorted(np.exp(rng.uniform(np.log(1), np.log(2600), 2)))
        yield [tuple(int(v) for v in np.exp(rng.uniform(np.log(lo), np.log(hi + 1), 2)))
               for _ in range(int(rng.integers(1, 20)))]


@pytest.mark.parametrize("sms", [SMS, 40])
def test_groups_cover_their_tiles(sms):
    for shapes in _jobs():
        for precision in (0, 1):
            got, nblk = solver_plan(shapes, precision, sms)
            assert 0 <= nblk <= sms
            for (nr, nc), (on, blocks, a, b) in zip(shapes, got):
                rows, cols = -(-nr // 16), -(-nc // 64)
                # what is kept on the chip depends on the tile alone
                assert on == solver_plan([(nr, nc)], precision, sms)[0][0, 0]
                if not on:
                    assert blocks == 0
                elif precision:
                    assert rows * cols <= 8 * min(sms, 128) and blocks <= nblk
                else:
                    assert 1 <= a * b <= 16 and b <= 4
                    assert blocks == -(-rows // a) * -(-cols // b) <= nblk


def test_tiles_beyond_the_chip_are_streamed():
    on = [t[0] for t in solver_plan([(1536, 1536), (1700, 1600), (5, 38000), (60, 50)])[0]]
    assert on == [1, 0, 0, 1]
    on = [t[0] for t in solver_plan([(1024, 1024), (1, 64 * 1025), (901, 1250), (90, 75)], 1)[0]]
    assert on == [1, 0, 0, 1]
