"""Which memory of a destroyed image a context keeps as it is: only what no work can be using. The
others go through cudaFree themselves, since nothing promises that another wait covers them."""
import numpy as np
import pytest

from host_gpu import host_gpu  # noqa: F401

W, H = 64, 48
STREAM = 0x500


def texture(g, fmt=None):
    return g.vx.Texture.create(g.ctx, W, H, g.vx.FORMAT_F32 if fmt is None else fmt)


def calls(g, t):
    """Uses of an F32 image: (name, call with a stream or None)."""
    out = texture(g)
    f = g.vx.DepthFilter(g.ctx)
    a = np.zeros((H, W), np.float32)
    return {"none": lambda s: None, "upload": lambda s: t.upload(a, stream=s), "download": lambda s: t.download(a, stream=s),
            "median in": lambda s: f.apply_median(g.ctx, t, out, stream=s),
            "median out": lambda s: f.apply_median(g.ctx, out, t, stream=s),
            "bilateral": lambda s: f.apply_bilateral(g.ctx, t, out, stream=s)}


def freed(g):
    return [line.split()[1] for line in g.log() if line.startswith("free")]


def address(line):
    return line.split()[1]


USES = ["none", "upload", "download", "median in", "median out", "bilateral", "disparity", "batch", "depth"]


def use(g, t, name, stream):
    if name in ("disparity", "batch", "depth"):
        sgm = g.vx.SGMStereo(g.ctx)
        left, right = (texture(g, g.vx.FORMAT_U8) for _ in range(2))
        cfg = g.vx.SGMStereoConfig(num_disparities=16)
        if name == "disparity":
            sgm.compute_disparity(g.ctx, left, right, t, cfg, stream=stream)
        elif name == "batch":
            sgm.compute_batch(g.ctx, [left], [right], [t], [cfg], stream=stream)
        else:
            k = g.vx.CameraIntrinsics(1.0, 1.0, 1.0, 1.0, W, H)
            sgm.compute(g.ctx, left, right, cfg, k, 1.0, depth_out=t).texture.close()
    else:
        calls(g, t)[name](stream)


@pytest.mark.parametrize("name", USES)
def test_an_image_of_synchronous_calls_leaves_its_memory_as_it_is(host_gpu, name):  # noqa: F811
    g = host_gpu
    t = texture(g)
    use(g, t, name, None)
    g.log()
    t.close()
    assert not g.log()                       # no call to the device: neither a wait nor a free
    before = g.vx.memory_allocation_count()
    texture(g).close()
    assert g.vx.memory_allocation_count() == before


@pytest.mark.parametrize("name", USES[1:-1] + ["pointer"])
def test_memory_that_work_may_still_use_is_freed_itself(host_gpu, name):  # noqa: F811
    g = host_gpu
    t = texture(g)
    if name == "pointer":
        ptr = t.device_ptr
    else:
        use(g, t, name, STREAM)
        ptr = None
    g.log()
    before = g.vx.memory_allocation_count()
    t.close()
    log = [line for line in g.log() if not line.startswith("launch")]
    assert [line.split()[0] for line in log] == ["free", "mallocpitch"], log
    assert ptr is None or int(address(log[0]), 16) == ptr
    assert log[1].endswith("mode 2")         # relaxed: no capture of this thread sees it
    assert g.vx.memory_allocation_count() == before + 1


def test_an_image_of_a_failed_call_is_freed_itself(host_gpu):  # noqa: F811
    g = host_gpu
    t, bad = texture(g), texture(g, g.vx.FORMAT_U8)
    with pytest.raises(g.vx.VxError):
        g.vx.SGMStereo(g.ctx).compute_disparity(g.ctx, bad, t, t, g.vx.SGMStereoConfig(num_disparities=16))
    g.log()
    t.close()
    assert len(freed(g)) == 1


def test_nothing_is_kept_after_the_context(host_gpu):  # noqa: F811
    g = host_gpu
    ctx = g.vx.Context(0)
    kept, late, busy = (g.vx.Texture.create(ctx, W, H, g.vx.FORMAT_F32) for _ in range(3))
    busy.device_ptr
    kept.close()
    g.log()
    ctx.close()
    assert len(freed(g)) == 1
    late.close()
    busy.close()
    log = g.log()
    assert [line.split()[0] for line in log] == ["free", "free"], log


def test_every_image_allocation_is_counted(host_gpu):  # noqa: F811
    g = host_gpu
    texture(g).close()                        # something to give back
    before = g.vx.memory_allocation_count()
    g.fail(pitch=1)
    g.log()
    t = g.vx.Texture.create(g.ctx, W, H + 1, g.vx.FORMAT_F32)     # fails, gives back, succeeds
    assert freed(g)
    assert g.vx.memory_allocation_count() == before + 2
    t.close()
    g.fail(pitch=2)
    with pytest.raises(g.vx.VxError):
        g.vx.Texture.create(g.ctx, W, H + 2, g.vx.FORMAT_F32)
    g.fail()


@pytest.mark.parametrize("name", ["disparity", "batch", "graph", "autotune", "matcher", "frames", "cloud", "server"])
def test_kept_memory_is_given_back_where_other_allocations_fail(host_gpu, name):  # noqa: F811
    """The first allocation of the call fails: the kept blocks go, and the call succeeds."""
    g = host_gpu
    vx = g.vx
    ctx = vx.Context(0)
    sgm, m, dc = vx.SGMStereo(ctx), vx.StereoMatcher(ctx), vx.DepthToCloud(ctx)
    l, r, o, spare, d = (vx.Texture.create(ctx, W, H, f) for f in (vx.FORMAT_U8,) * 2 + (vx.FORMAT_F32,) * 3)
    cfg = vx.SGMStereoConfig(num_disparities=16)
    if name == "graph":
        sgm.set_graph_cache(2)
    offsets = np.array([0, 5000], np.uint32)
    run = {"disparity": lambda: sgm.compute_disparity(ctx, l, r, o, cfg),
           "batch": lambda: sgm.compute_batch(ctx, [l], [r], [o], [cfg]),
           "graph": lambda: sgm.compute_disparity(ctx, l, r, o, cfg),
           "autotune": lambda: sgm.autotune_batch(ctx, [l], [r], [o], [cfg], iterations=1),
           "matcher": lambda: m.run_device(ctx, 4096, 5000, 4096, 5000, 4096, 4096, vx.StereoConfig(), 4096, 4096),
           "frames": lambda: m.run_frames_device(ctx, offsets, offsets, 4096, 4096, 4096, 4096, vx.StereoConfig(),
                                                 4096, 4096),
           "cloud": lambda: dc.compute_device(ctx, d, None, 1.0, 1.0, 1.0, 1.0, vx.DepthToCloudConfig(), 4096, 10, 4096),
           "server": lambda: vx.Server(sgm, ctx, memory_budget_bytes=64 << 20, max_batch=2,
                                       max_inflight_batches=1).close()}[name]
    spare.close()
    g.fail(pool=1)
    g.log()
    before = vx.memory_allocation_count()
    run()
    assert freed(g) and vx.memory_allocation_count() >= before + 2
    g.fail(pool=2)
    if name in ("disparity", "batch"):       # nothing kept: the failure stands
        with pytest.raises(vx.VxError):
            run()
    g.fail()
