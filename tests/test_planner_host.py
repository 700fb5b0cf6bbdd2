"""Which kernels the planner sends a call to, from the launches of the library's host side alone."""
import json

import pytest

from host_gpu import host_gpu  # noqa: F401


def batch(g, sizes, paths=8, census=2, **penalties):
    """(left, right, out, configs) of pairs (w, h, D)."""
    vx = g.vx
    img = lambda w, h, f: vx.Texture.create(g.ctx, w, h, f)
    left, right = ([img(w, h, vx.FORMAT_U8) for w, h, _ in sizes] for _ in range(2))
    out = [img(w, h, vx.FORMAT_F32) for w, h, _ in sizes]
    return left, right, out, [vx.SGMStereoConfig(num_disparities=d, num_paths=paths, census_radius_x=census,
                                                 census_radius_y=census, **penalties) for _, _, d in sizes]


def aggregation(g, sgm, b):
    """The form that a batch runs: pairs, single, scan or packed."""
    g.log()
    sgm.compute_batch(g.ctx, *b)
    names = {n.split("<")[0] for n in g.launches()} - {"census_kernel", "cost_kernel", "wta_kernel"}
    return names


LARGE = [(640, 480, 256)] * 16          # 1728 units of 64 scanlines


def test_a_tuning_is_of_its_penalties(host_gpu, tmp_path):  # noqa: F811
    g = host_gpu
    small, large = batch(g, LARGE, p1=10, p2=120), batch(g, LARGE, p1=127, p2=120)    # 127: the packed range ends
    plain = g.vx.SGMStereo(g.ctx)
    want_small, want_large = aggregation(g, plain, small), aggregation(g, plain, large)
    assert want_small == {"packed_kernel"} and want_large != want_small
    tuned = g.vx.SGMStereo(g.ctx)
    unit = tuned.autotune_batch(g.ctx, *small, iterations=1)[2]
    tuned.tuning_save(str(tmp_path / "t.json"))
    entry, = json.load(open(tmp_path / "t.json"))["entries"]
    assert entry["packed"] == 1 and entry["unit_scanlines"] == unit
    loaded = g.vx.SGMStereo(g.ctx)
    loaded.tuning_load(str(tmp_path / "t.json"))
    # A scan entry of small penalties, and one of a file without the field, which is of all.
    entry.update(unit_scanlines=1, warpgroups=1)
    scan, old = g.vx.SGMStereo(g.ctx), g.vx.SGMStereo(g.ctx)
    json.dump({"version": 1, "entries": [entry]}, open(tmp_path / "scan.json", "w"))
    scan.tuning_load(str(tmp_path / "scan.json"))
    del entry["packed"]
    entry["unit_scanlines"] = 64
    json.dump({"version": 1, "entries": [entry]}, open(tmp_path / "old.json", "w"))
    old.tuning_load(str(tmp_path / "old.json"))
    for sgm in (tuned, loaded, scan):
        assert aggregation(g, sgm, large) == want_large
    assert aggregation(g, scan, small) == want_small
    assert aggregation(g, old, small) == aggregation(g, old, large) == want_large


@pytest.mark.parametrize("form,unit", [("scan", 1), ("scan8", 1), ("scan16", 1), ("scan32", 1), ("pairs", 64), ("single", 32)])
def test_a_tuning_under_a_forced_form_is_of_that_form(host_gpu, monkeypatch, form, unit):  # noqa: F811
    g = host_gpu
    monkeypatch.setenv("VX_SGM_AGG_FORM", form)
    assert g.vx.SGMStereo(g.ctx).autotune_batch(g.ctx, *batch(g, [(64, 48, 64)]), iterations=1)[2] == unit


# Measured on B200, us of aggregation: packed scan / scanline pairs.
@pytest.mark.parametrize("n,w,h,d,p2,form", [
    (16, 1280, 720, 144, 120, "pairs"),      # 13997 / 9063: 9 lanes of 16
    (16, 1280, 720, 80, 120, "pairs"),       # 6775 / 5128
    (32, 640, 480, 100, 120, "pairs"),       # 4639 / 4185
    (32, 640, 480, 40, 120, "pairs"),        # 2206 / 1977
    (16, 1280, 720, 208, 120, "packed"),     # 14564 / 15289
    (32, 640, 480, 8, 120, "packed"),        # 563 / 880
    (32, 640, 480, 64, 120, "packed"),       # 1892 / 2552
    (8, 2048, 1536, 256, 120, "packed"),     # 19347 / 25833
    (32, 640, 480, 64, 300, "pairs"),        # wide slabs: 5214 / 3529
    (16, 640, 480, 128, 300, "pairs"),       # 5015 / 3928
    (16, 1280, 720, 144, 300, "pairs"),      # 24509 / 12258
    (8, 2048, 1536, 256, 300, "pairs"),      # 50992 / 45727
    (16, 1920, 1080, 192, 300, "packed"),    # 34272 / 47732: 24 disparities a lane
    (12, 1280, 720, 192, 300, "packed"),     # 11450 / 17625
    (16, 1280, 720, 208, 300, "packed"),     # 24799 / 29179
    (2, 2048, 1536, 256, 300, "packed"),     # 12831 / 18271: few units
    (1, 640, 480, 100, 120, "packed"),
])
def test_large_batches_run_the_faster_form(host_gpu, n, w, h, d, p2, form):  # noqa: F811
    got, = aggregation(host_gpu, host_gpu.vx.SGMStereo(host_gpu.ctx), batch(host_gpu, [(w, h, d)] * n, p1=10, p2=p2))
    assert got == {"packed": "packed_kernel", "pairs": "aggregate_kernel"}[form]


@pytest.mark.parametrize("n,form", [(1, "scan"), (8, "scan"), (40, "pairs")])
def test_penalties_beyond_the_packed_range_keep_their_forms(host_gpu, n, form):  # noqa: F811
    got, = aggregation(host_gpu, host_gpu.vx.SGMStereo(host_gpu.ctx),
                       batch(host_gpu, [(640, 480, 128)] * n, p1=700, p2=3000))
    assert got == {"scan": "scan_kernel", "pairs": "aggregate_kernel"}[form]


# Measured on B200, us of the WTA: 16 warps a row / the choice.
@pytest.mark.parametrize("n,w,h,d,paths,warps", [
    (1000, 32, 32, 32, 4, {1}),              # 567 / 62
    (600, 100, 100, 128, 8, {1, 2}),         # 1715 / 969
    (100, 32, 32, 16, 2, {1}),               # 53 / 10
    (30, 640, 480, 64, 4, {2, 4}),           # 500 / 407
    (1, 640, 480, 64, 4, {8, 10, 16}),       # lone pairs: by the rounds of CTAs
    (1, 1280, 720, 64, 8, {8}),
    (8, 2048, 1536, 256, 8, {6, 8, 12}),     # wide rows do not care
])
def test_narrow_rows_take_few_warps(host_gpu, n, w, h, d, paths, warps):  # noqa: F811
    g = host_gpu
    b = batch(g, [(w, h, d)] * n, paths=paths)
    g.log()
    g.vx.SGMStereo(g.ctx).compute_batch(g.ctx, *b)
    wta, = [line.split() for line in g.log() if line.startswith("launch") and "wta_kernel" in line]
    assert int(wta[wta.index("block") + 1]) // 32 in warps
