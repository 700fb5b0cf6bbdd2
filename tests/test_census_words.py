"""The census kernel's four-pixel words: the byte comparison inside a word for
every pair of bytes (CPU), and the descriptors at the edges of the words, tiles
and windows, with every alignment of a row's first word, against the oracle (GPU)."""
import numpy as np
import pytest

import oracle
import vx_sgm


def test_byte_comparison_inside_a_word():
    # A word holds the pair of interest in one byte and extreme neighbours in the others.
    n, c = (v.astype(np.uint32).ravel() for v in np.meshgrid(np.arange(256), np.arange(256)))
    for at in range(4):
        for rest_n, rest_c in ((0, 0), (0, 255), (255, 0), (255, 255), (127, 128), (128, 127)):
            spread = lambda v, rest: sum(np.uint32(rest << 8 * i) for i in range(4) if i != at) | (v << np.uint32(8 * at))
            wn, wc = spread(n, rest_n), spread(c, rest_c)
            d = (wn | np.uint32(0x80808080)) - (wc & np.uint32(0x7F7F7F7F))
            lt = (~wn & wc) | (~(wn ^ wc) & ~d)
            assert np.array_equal(lt >> np.uint32(8 * at + 7) & 1, n < c)


@pytest.mark.gpu
@pytest.mark.parametrize("rx,ry", [(0, 1), (1, 0), (1, 1), (2, 2), (3, 2), (3, 3), (4, 3), (5, 2), (15, 0), (0, 31), (31, 0), (2, 6)])
def test_descriptors_at_every_edge(gpu_ctx, sgm, rx, ry):
    cfg = vx_sgm.SGMStereoConfig(num_disparities=8, census_radius_x=rx, census_radius_y=ry, num_paths=2)
    rng = np.random.default_rng(100 * rx + ry)
    for w, h in ((1, 5), (3, 2), (4, 33), (31, 3), (34, 35), (65, 4), (130, 70), (207, 40)):
        L, R = (rng.integers(0, 256, (h, w), dtype=np.uint8) for _ in range(2))
        tl, tr = gpu_ctx.texture_gray8(L, w, h), gpu_ctx.texture_gray8(R, w, h)
        cl, cr, _, _ = sgm.debug_dump(gpu_ctx, tl, tr, cfg)
        assert np.array_equal(cl, oracle.census(L, rx, ry)) and np.array_equal(cr, oracle.census(R, rx, ry)), (w, h)
