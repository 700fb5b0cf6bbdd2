"""Image memory kept by a context: reuse, bounds, threads, and images that outlive their context."""
import threading

import numpy as np
import pytest

import vx_sgm

pytestmark = pytest.mark.gpu


def test_blocks_are_reused_by_shape_and_bounded():
    ctx = vx_sgm.Context(0)
    a = ctx.texture_output_r32float(640, 480)
    ptr, pitch = a.device_ptr, a.pitch
    a.close()
    before = vx_sgm.memory_allocation_count()
    other = ctx.texture_output_r32float(640, 481)              # another height: a block of its own
    same = ctx.texture_output_r32float(640, 480)
    assert same.device_ptr == ptr and same.pitch == pitch and other.device_ptr != ptr
    assert vx_sgm.memory_allocation_count() == before + 1
    # More images than are kept: all are distinct while they live, and fewer come back without an allocation.
    many = [ctx.texture_output_gray8(64, 32) for _ in range(40)]
    assert len({t.device_ptr for t in many}) == 40
    for t in many:
        t.close()
    before = vx_sgm.memory_allocation_count()
    again = [ctx.texture_output_gray8(64, 32) for _ in range(40)]
    assert 24 <= vx_sgm.memory_allocation_count() - before <= 40
    big = ctx.texture_output_r32float(8192, 4096)              # 128 MiB: never kept
    big.close()
    before = vx_sgm.memory_allocation_count()
    ctx.texture_output_r32float(8192, 4096).close()
    assert vx_sgm.memory_allocation_count() == before + 1
    del again, other, same
    ctx.close()


def test_a_released_image_is_no_longer_in_use():
    """Work queued on another stream still reads an image when it is destroyed: the block's next image
    must not change what that work sees."""
    import torch
    ctx = vx_sgm.Context(0)
    w, h = 1024, 1024
    filt = vx_sgm.DepthFilter(ctx)
    stream = torch.cuda.Stream()
    src = ctx.texture_r32float(np.full((h, w), 3.0, np.float32), w, h)
    out = ctx.texture_output_r32float(w, h)
    for _ in range(20):
        filt.apply_median(ctx, src, out, vx_sgm.DepthMedianConfig(5), stream=stream.cuda_stream)
    src.close()
    nxt = ctx.texture_r32float(np.full((h, w), 7.0, np.float32), w, h)
    torch.cuda.synchronize()
    assert (out.download() == 3.0).all() and (nxt.download() == 7.0).all()
    filt.close()


def test_images_outlive_their_context_and_threads_share_it():
    ctx = vx_sgm.Context(0)
    errors = []

    def work(seed):
        rng = np.random.default_rng(seed)
        try:
            for _ in range(30):
                w, h = int(rng.integers(1, 4)) * 32, int(rng.integers(1, 4)) * 16
                data = rng.random((h, w)).astype(np.float32)
                t = ctx.texture_r32float(data, w, h)
                assert np.array_equal(t.download(), data)
                t.close()
        except Exception as e:  # noqa: BLE001
            errors.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    left = ctx.texture_output_gray8(32, 32)
    ctx.close()
    left.close()          # after its context: freed, not kept


@pytest.mark.parametrize("mode", ["thread_local", "relaxed"])
def test_an_image_destroyed_during_a_capture_leaves_it_alone(mode):
    """Freeing memory from another thread (or, in a relaxed capture, from any) does not end a
    stream capture, so neither does destroying an image."""
    import torch
    ctx = vx_sgm.Context(0)
    images = [ctx.texture_output_r32float(320, 200) for _ in range(3)]
    x = torch.zeros(64, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode=mode):
        x += 1
        for img in images[:2]:
            t = threading.Thread(target=img.close)
            t.start()
            t.join()
        if mode == "relaxed":
            images[2].close()
        x += 1
    graph.replay()
    torch.cuda.synchronize()
    assert (x == 2).all()
    del graph
