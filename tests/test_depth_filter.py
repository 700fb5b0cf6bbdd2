"""Depth-map post-filters (vx-vision DepthFilter: median, bilateral).

CPU: the oracle restatement (oracle/depth_oracle.cpp) equals the reference
shader's own outputs (tests/golden/depth_filter_cases.npz, made by
tests/golden/make_depth_golden.py from shaders/DepthFilter.metal compiled as
C++); the reference's own test assertions hold on the oracle.
GPU: the CUDA filters through the C ABI against the same fixtures — the median
bit-exact, the bilateral within 1e-5 relative (its range weights come from CUDA's
__expf intrinsic, the fixtures' from the host's expf) — and against the oracle on SGM
disparity maps."""
import json
import os

import numpy as np
import pytest

import oracle
import vx_sgm
from host_gpu import host_gpu  # noqa: F401

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "depth_filter_cases.npz")
BILATERAL_RTOL = 1e-5


def _cases():
    z = np.load(GOLDEN)
    meta = json.loads(bytes(z["meta"]).decode())
    maps = {k.split("/", 1)[1]: z[k] for k in z.files if k.startswith("map/")}
    return [(m, maps[m["map"]], z[f"out/{m['id']}"]) for m in meta]


def _run_oracle(m, depth):
    if m["kind"] == "median":
        return oracle.depth_median(depth, m["radius"])
    return oracle.depth_bilateral(depth, m["radius"], m["sigma_spatial"], m["sigma_depth"])


def _same_bits(a, b):
    return np.array_equal(np.asarray(a, np.float32).view(np.uint32), np.asarray(b, np.float32).view(np.uint32))


def test_oracle_equals_reference_fixtures():
    cases = _cases()
    assert len(cases) >= 60
    for m, depth, want in cases:
        got = _run_oracle(m, depth)
        assert _same_bits(got, want), m


def test_reference_assertions_on_oracle():
    """vx-vision/tests/test_kernels.rs:840-901, on the oracle."""
    w = h = 32
    edge = np.where(np.arange(w * h).reshape(h, w) % w < w // 2, 1.0, 5.0).astype(np.float32)
    r = oracle.depth_bilateral(edge, 2, 3.0, 0.1)
    assert abs(r[h // 2, w // 4] - 1.0) < 0.5 and abs(r[h // 2, 3 * w // 4] - 5.0) < 0.5
    noisy = np.full((h, w), 2.0, np.float32)
    noisy.flat[100] = 99.0
    noisy.flat[200] = 0.5
    assert abs(oracle.depth_median(noisy, 1).flat[100] - 2.0) < 1.0


def test_median_excludes_invalid_and_takes_upper_middle():
    d = np.array([[-1, 3, 1], [2, -1, 4], [-1, -1, 5]], np.float32)
    # centre window (r = 1, clamped) holds the valid values 3 1 2 4 5 -> sorted 1 2 3 4 5 -> index 2
    assert oracle.depth_median(d, 1)[1, 1] == 3.0
    d2 = np.array([[1, 2], [3, 4]], np.float32)
    # r = 1 window of (0, 0), clamped: 1 1 2 1 1 2 3 3 4 -> count 9, index 4 -> 2
    assert oracle.depth_median(d2, 1)[0, 0] == 2.0
    assert oracle.depth_median(np.full((3, 3), -1, np.float32), 1).max() == 0.0


@pytest.mark.gpu
def test_cuda_filters_match_reference_fixtures(gpu_ctx):
    filt = vx_sgm.DepthFilter(gpu_ctx)
    for m, depth, want in _cases():
        h, w = depth.shape
        tin = gpu_ctx.texture_r32float(depth, w, h)
        tout = gpu_ctx.texture_output_r32float(w, h)
        if m["kind"] == "median":
            filt.apply_median(gpu_ctx, tin, tout, vx_sgm.DepthMedianConfig(m["radius"]))
            assert _same_bits(tout.read_r32float(), want), m
        else:
            filt.apply_bilateral(gpu_ctx, tin, tout, vx_sgm.DepthFilterConfig(
                m["radius"], m["sigma_spatial"], m["sigma_depth"]))
            got = tout.read_r32float()
            np.testing.assert_allclose(got, want, rtol=BILATERAL_RTOL, atol=0, err_msg=str(m))
    filt.close()


@pytest.mark.gpu
def test_cuda_median_on_sgm_output_large(gpu_ctx, sgm):
    """The demo chain: SGM with the LR check (invalid = -1), then the median filter; the
    filtered map equals the oracle's median of the same map, bit for bit."""
    w, h = 640, 480
    L, R, _ = vx_sgm.synth_pair(vx_sgm.SCENE_PLANES, w, h, 4, 60, 77)
    cfg = vx_sgm.SGMStereoConfig(num_disparities=64, census_radius_x=2, census_radius_y=2,
                                 num_paths=4, lr_check=True)
    tl, tr = gpu_ctx.texture_gray8(L, w, h), gpu_ctx.texture_gray8(R, w, h)
    disp = gpu_ctx.texture_output_r32float(w, h)
    sgm.compute_disparity(gpu_ctx, tl, tr, disp, cfg)
    d = disp.read_r32float()
    assert (d < 0).any()
    filt = vx_sgm.DepthFilter(gpu_ctx)
    out = gpu_ctx.texture_output_r32float(w, h)
    for r in (1, 2, 3):
        filt.apply_median(gpu_ctx, disp, out, vx_sgm.DepthMedianConfig(r))
        assert _same_bits(out.read_r32float(), oracle.depth_median(d, r)), r
    filt.apply_bilateral(gpu_ctx, disp, out, vx_sgm.DepthFilterConfig())
    np.testing.assert_allclose(out.read_r32float(), oracle.depth_bilateral(d, 3, 5.0, 0.05),
                               rtol=BILATERAL_RTOL, atol=0)
    filt.close()


@pytest.mark.gpu
def test_cuda_filter_argument_checks(gpu_ctx):
    filt = vx_sgm.DepthFilter(gpu_ctx)
    a = gpu_ctx.texture_output_r32float(16, 8)
    b = gpu_ctx.texture_output_r32float(16, 9)
    with pytest.raises(vx_sgm.VxError) as e:
        filt.apply_median(gpu_ctx, a, b)
    assert e.value.status == 5  # size mismatch
    c = gpu_ctx.texture_output_r32float(16, 8)
    for bad in (-1, 6):
        with pytest.raises(vx_sgm.VxError) as e:
            filt.apply_median(gpu_ctx, a, c, vx_sgm.DepthMedianConfig(bad))
        assert e.value.status == 6
    with pytest.raises(vx_sgm.VxError):
        filt.apply_bilateral(gpu_ctx, a, c, vx_sgm.DepthFilterConfig(3, 0.0, 0.05))
    with pytest.raises(vx_sgm.VxError):
        filt.apply_median(gpu_ctx, a, a)  # in place
    filt.close()


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(1, 1), (2, 3), (63, 5), (64, 8), (65, 9), (127, 4), (130, 17)])
def test_cuda_median_tile_edges(gpu_ctx, w, h):
    """Every radius around the tile size (64 outputs by 4 or 8 rows, two a thread), with few, many
    and no valid values, +inf among them, in aligned textures and in a plane of odd pitch."""
    import torch
    rng = np.random.default_rng(w * 100 + h)
    filt = vx_sgm.DepthFilter(gpu_ctx)
    for invalid in (0.0, 0.3, 0.9, 1.0):
        d = rng.choice(np.array([1.5, 2.0, 3.25, 80.0, np.inf], np.float32), (h, w)) * rng.integers(1, 9, (h, w))
        d = np.where(rng.random((h, w)) < invalid, rng.choice([-1.0, 0.0, np.nan, -np.inf], (h, w)), d).astype(np.float32)
        tin, tout = gpu_ctx.texture_r32float(d, w, h), gpu_ctx.texture_output_r32float(w, h)
        pitch = 4 * (w + 1)
        buf = torch.zeros(pitch * h + 4, dtype=torch.uint8, device="cuda")
        odd = vx_sgm.Texture.wrap_device(gpu_ctx, buf.data_ptr() + 4, pitch, w, h, vx_sgm.FORMAT_F32)
        torch.cuda.synchronize()
        for r in range(6):
            want = oracle.depth_median(d, r)
            for out in (tout, odd):
                filt.apply_median(gpu_ctx, tin, out, vx_sgm.DepthMedianConfig(r))
                assert _same_bits(out.read_r32float(), want), (invalid, r)
        odd.close()
    filt.close()


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(1, 1), (3, 2), (127, 7), (128, 8), (129, 9), (261, 17)])
def test_cuda_bilateral_tile_edges(gpu_ctx, w, h):
    """Every instantiated radius and the first beyond them around the tile size (128 x 8 outputs, four a
    thread), with invalid values, infinities, NaN and extreme sigmas, in an aligned texture and in a plane of
    odd pitch: within the filter's tolerance of the oracle, NaN and infinity where it has them."""
    import torch
    rng = np.random.default_rng(w * 10 + h)
    filt = vx_sgm.DepthFilter(gpu_ctx)
    pitch = 4 * (w + 1)
    buf = torch.zeros(pitch * h + 4, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    odd = vx_sgm.Texture.wrap_device(gpu_ctx, buf.data_ptr() + 4, pitch, w, h, vx_sgm.FORMAT_F32)
    even = gpu_ctx.texture_output_r32float(w, h)
    for special in (False, True):
        d = (1.0 + 4.0 * rng.random((h, w))).astype(np.float32)
        d[rng.random((h, w)) < 0.3] = -1.0
        if special:
            d[rng.random((h, w)) < 0.02] = np.nan
            d[rng.random((h, w)) < 0.02] = np.inf
        tin = gpu_ctx.texture_r32float(d, w, h)
        for r in (0, 1, 2, 3, 4, 5, 6, 7, 8, 9):
            for ss, sd in ((5.0, 0.05), (0.3, 2.0), (1e4, 1e6)):
                want = oracle.depth_bilateral(d, r, ss, sd)
                for out in (even, odd):
                    filt.apply_bilateral(gpu_ctx, tin, out, vx_sgm.DepthFilterConfig(r, ss, sd))
                    np.testing.assert_allclose(out.read_r32float(), want, rtol=BILATERAL_RTOL, atol=0,
                                               err_msg=f"r={r} ss={ss} sd={sd} special={special}")
    odd.close()
    filt.close()


@pytest.mark.gpu
@pytest.mark.parametrize("invalid", [-np.inf, -3.4e38, -1.0, -0.0, 0.0])
def test_cuda_bilateral_skips_every_invalid_value(gpu_ctx, invalid):
    """Any value <= 0 is left out, whatever its size (an SGM config may name any invalid value): a map of 2
    with one such pixel stays 2 around it, and mixed with valid values the result is the oracle's."""
    w, h = 21, 13
    filt = vx_sgm.DepthFilter(gpu_ctx)
    flat = np.full((h, w), 2.0, np.float32)
    flat[6, 10] = invalid
    rng = np.random.default_rng(5)
    mixed = np.where(rng.random((h, w)) < 0.3, invalid, 1.0 + 4.0 * rng.random((h, w))).astype(np.float32)
    out = gpu_ctx.texture_output_r32float(w, h)
    for r in range(10):                      # 1..8 have a kernel each, 0 and 9 the general one
        filt.apply_bilateral(gpu_ctx, gpu_ctx.texture_r32float(flat, w, h), out, vx_sgm.DepthFilterConfig(r, 5.0, 0.05))
        want = np.full((h, w), 2.0, np.float32)
        want[6, 10] = 0.0
        np.testing.assert_allclose(out.read_r32float(), want, rtol=BILATERAL_RTOL, atol=0, err_msg=f"r={r}")
        filt.apply_bilateral(gpu_ctx, gpu_ctx.texture_r32float(mixed, w, h), out, vx_sgm.DepthFilterConfig(r, 5.0, 2.0))
        np.testing.assert_allclose(out.read_r32float(), oracle.depth_bilateral(mixed, r, 5.0, 2.0),
                                   rtol=BILATERAL_RTOL, atol=0, err_msg=f"r={r}")
    filt.close()


@pytest.mark.parametrize("rows,launches", [(8 * 65535, 2), (4 * 65535, 1), (4 * 65535 + 1, 2), (8 * 65535 + 1, None)])
def test_tall_maps_are_taken_at_every_radius(host_gpu, rows, launches):  # noqa: F811
    """Up to 524280 rows at every radius; the launches of the radii with tiles of 4 rows."""
    g = host_gpu
    a, b = (g.vx.Texture.create(g.ctx, 1, rows, g.vx.FORMAT_F32) for _ in range(2))
    filt = g.vx.DepthFilter(g.ctx)
    for r in range(6):
        g.log()
        if launches is None:
            with pytest.raises(g.vx.VxError):
                filt.apply_median(g.ctx, a, b, g.vx.DepthMedianConfig(r))
        else:
            filt.apply_median(g.ctx, a, b, g.vx.DepthMedianConfig(r))
            assert len(g.launches()) == (launches if r >= 3 else 1), r


@pytest.mark.gpu
@pytest.mark.parametrize("r", [2, 3, 5])
def test_cuda_median_of_a_tall_map(gpu_ctx, r):
    """More rows than one grid of 4-row tiles has: the seam of the two launches and the last rows."""
    w, h, tail = 3, 4 * 65535 + 9, 60
    rng = np.random.default_rng(r)
    d = np.where(rng.random((h, w)) < 0.3, -1.0, 1.0 + rng.random((h, w))).astype(np.float32)
    filt = vx_sgm.DepthFilter(gpu_ctx)
    out = gpu_ctx.texture_output_r32float(w, h)
    filt.apply_median(gpu_ctx, gpu_ctx.texture_r32float(d, w, h), out, vx_sgm.DepthMedianConfig(r))
    got = out.read_r32float()
    assert _same_bits(got[-tail + r:], oracle.depth_median(d[-tail:], r)[r:])
    assert _same_bits(got[:tail - r], oracle.depth_median(d[:tail], r)[:-r])
    filt.close()
