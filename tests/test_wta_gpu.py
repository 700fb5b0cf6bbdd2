"""The WTA row loop and the cost kernel's split rows against the oracle at the edges of its strips, lanes and carry:
every lanes-a-pixel variant with and without pads, each path count, byte and wide
slabs, values that wrap, rows shorter than a warp's pixels. Integers (and the
subpixel step, correctly rounded), so results are equal."""
import pytest

import oracle
import vx_sgm
from gpu_helpers import assert_disparity_equal, cfg_pair, run_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("paths", [2, 4, 8])
@pytest.mark.parametrize("p1,p2", [(10, 120), (10, 400), (126, 120)])   # byte slabs, wide slabs, many escapes
@pytest.mark.parametrize("nd", [1, 16, 17, 32, 33, 64, 65, 100, 128, 129, 192, 256])
def test_rows_of_every_width_class(gpu_ctx, sgm, nd, p1, p2, paths):
    pairs, cfgs, ocfgs = [], [], []
    for i, (w, h) in enumerate([(1, 3), (7, 2), (16, 5), (33, 4), (130, 9), (401, 3)]):
        L, R, _ = vx_sgm.synth_pair(i % 3, w, h, 0, max(1, min(nd, w) - 2), 31 * nd + w)
        c, o = cfg_pair(num_disparities=nd, p1=p1, p2=p2, census_radius_x=2, census_radius_y=2, num_paths=paths, lr_check=i != 4)
        pairs.append((L, R))
        cfgs.append(c)
        ocfgs.append(o)
    for (L, R), o, got in zip(pairs, ocfgs, run_batch(gpu_ctx, sgm, pairs, cfgs)):
        d, di, _ = oracle.sgm(L, R, o)
        assert_disparity_equal(got, (d, di), what=f"{L.shape} D={nd} {paths} paths")


@pytest.mark.parametrize("nd", [16, 33, 64, 128, 192, 256])
@pytest.mark.parametrize("w", [127, 128, 257, 1030])
def test_cost_passes_split_over_ctas(gpu_ctx, sgm, nd, w):
    """A row's passes in several CTAs (synchronous, few rows) and rows of unequal passes in one
    batch, where a row's CTAs take its passes in turn: 1 to 9 passes a row."""
    pairs, cfgs, ocfgs = [], [], []
    for i, (wi, d) in enumerate([(w, nd), (1030, 128)]):
        L, R, _ = vx_sgm.synth_pair(i, wi, 5, 0, max(1, min(d, wi) - 2), 7 * nd + w)
        c, o = cfg_pair(num_disparities=d, census_radius_x=2, census_radius_y=2, num_paths=4, lr_check=True)
        pairs.append((L, R))
        cfgs.append(c)
        ocfgs.append(o)
    for n in (1, 2):
        for (L, R), o, got in zip(pairs[:n], ocfgs, run_batch(gpu_ctx, sgm, pairs[:n], cfgs[:n])):
            d, di, _ = oracle.sgm(L, R, o)
            assert_disparity_equal(got, (d, di), what=f"{L.shape} D={nd} {n} pairs")
