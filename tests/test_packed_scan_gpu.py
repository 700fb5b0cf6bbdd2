"""The packed across-lanes scan kernels against the oracle on every lane geometry
(with and without pads), in both kinds, with byte and wide slabs, with values
that wrap, and as classes of one mixed batch with a shadow pool. Integers, so
results are equal."""
import numpy as np
import pytest

import oracle
import vx_sgm
from gpu_helpers import assert_disparity_equal, cfg_pair, run_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["scan8", "scan16", "scan32"])
@pytest.mark.parametrize("nd,p1,p2,rx,ry", [
    (16, 10, 120, 2, 2), (32, 10, 120, 2, 2), (48, 10, 120, 2, 2), (64, 0, 120, 4, 3), (96, 15, 300, 2, 2),
    (128, 3, 120, 4, 3), (192, 10, 120, 4, 3), (256, 7, 90, 2, 2),                   # lanes a power of two
    (1, 10, 120, 2, 2), (15, 10, 300, 2, 2), (20, 2, 120, 4, 3), (80, 10, 120, 2, 2), (100, 3, 120, 4, 3),
    (112, 15, 300, 4, 3), (144, 10, 120, 2, 2), (200, 0, 2000, 4, 3), (250, 10, 120, 2, 2),   # pads
    (16, 3690, 400, 2, 2), (256, 126, 120, 4, 3),                                    # the largest P1 of the packed form
])
def test_every_path_of_every_geometry(gpu_ctx, sgm, monkeypatch, form, nd, p1, p2, rx, ry):
    monkeypatch.setenv("VX_SGM_AGG_FORM", form)
    w, h = 71, 23
    L, R, _ = vx_sgm.synth_pair(nd % 3, w, h, 0, max(1, min(nd - 2, w - 2)), nd * 100 + p1)
    cfg, _ = cfg_pair(num_disparities=nd, p1=p1, p2=p2, census_radius_x=rx, census_radius_y=ry, num_paths=8)
    tl, tr = gpu_ctx.texture_gray8(L, w, h), gpu_ctx.texture_gray8(R, w, h)
    _, _, got, _ = sgm.debug_dump(gpu_ctx, tl, tr, cfg)
    cl, cr = oracle.census(L, rx, ry), oracle.census(R, rx, ry)
    for k in range(8):
        want = oracle.path_costs(cl, cr, nd, p1, p2, *oracle.path_dir(k))
        bad = np.argwhere(got[k] != want)
        assert bad.size == 0, f"path {k} differs at {bad[:4]}"


@pytest.mark.parametrize("form", ["scan8", "scan16"])
@pytest.mark.parametrize("pool", ["", "40"])
def test_classes_of_a_mixed_batch(gpu_ctx, sgm, monkeypatch, form, pool):
    """Seven geometries in one batch: seven launches that overlap, escapes in shadow
    pools (synchronous batches), one of them forced to overflow and be recomputed."""
    monkeypatch.setenv("VX_SGM_AGG_FORM", form)
    if pool:
        monkeypatch.setenv("VX_SGM_SHADOW_POOL", pool)
    pairs, cfgs, ocfgs = [], [], []
    for i, nd in enumerate([64, 192, 33, 128, 256, 100, 16, 64, 48]):
        w, h = 60 + 37 * i, 30 + 11 * ((i * 5) % 7)
        L, R, _ = vx_sgm.synth_pair(i % 3, w, h, 0, max(1, min(nd, w) - 3), 700 + i)
        c, o = cfg_pair(num_disparities=nd, census_radius_x=2 + i % 3, census_radius_y=2, num_paths=[8, 4, 2][i % 3],
                        p2=300 if i == 5 else 120, lr_check=bool(i % 2))
        pairs.append((L, R))
        cfgs.append(c)
        ocfgs.append(o)
    for (L, R), o, got in zip(pairs, ocfgs, run_batch(gpu_ctx, sgm, pairs, cfgs)):
        d, di, _ = oracle.sgm(L, R, o)
        assert_disparity_equal(got, (d, di), what=f"{form} D={o.num_disparities}")
