"""CPU replay of the WTA row loop's work mapping: a warp walks a strip of the row,
its lanes carry the right-view minima of their columns S places up a round, and
the columns that leave go to the row's minima. Every column must end with the
minimum over all its keys, no column outside the row may be written, and the
sums and row arrays must fit the shared memory of a launch. The constants mirror
the kernel's (kernels.cuh: wta_max_threads, kWtaSumsPerWarp, kMaxWidth)."""
import numpy as np
import pytest

NONE = 1 << 40
SUMS_PER_WARP, MAX_WIDTH = 512, 16384


def _lanes_per_pixel(dv, k):
    seg = 1
    while seg < dv // k:
        seg <<= 1
    return seg


def _replay(keys, w, d, k, wide, warps):
    """Right-view minima and the set of (x, d) summed, as the row loop finds them."""
    dv = (d + 15) // 16 * 16
    vec = (d + 7) // 8 * 8 if wide else dv
    seg = _lanes_per_pixel(dv, k)
    ppw = 32 // seg
    s = k if wide else min(k, ppw)
    rounds = -(-w // (warps * ppw))
    right, seen = [NONE] * w, set()
    for warp in range(warps):
        for lane in range(32):
            sub, c = divmod(lane, seg)
            d0, rk, x = k * c, [NONE] * k, warp * rounds * ppw + sub
            assert k * lane + k <= SUMS_PER_WARP

            def leave(xr, lo, hi):
                for j in range(lo, hi):
                    if 0 <= xr - j < w:
                        right[xr - j] = min(right[xr - j], rk[j])
                    else:                                   # only columns left of the row hold keys
                        assert rk[j] == NONE or xr - j < 0

            for _ in range(rounds):
                act = x < w and d0 < vec
                nb = d - d0 if act else 0
                key = [keys[x][d0 + j] if j < nb else NONE for j in range(k)]
                seen.update((x, d0 + j) for j in range(k) if j < nb)
                rk = [min(rk[j - s], key[j]) if j >= s else key[j] for j in range(k)]
                leave(x - d0, k - s, k)
                x += ppw
            leave(x - s - d0, 0, k - s)
    return right, seen


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("warps", [6, 8, 16])
@pytest.mark.parametrize("w,d", [(1, 1), (2, 16), (15, 17), (33, 64), (97, 64), (130, 65), (70, 128), (131, 100), (260, 192), (129, 256), (64, 33)])
def test_right_view_minima_and_coverage(w, d, warps, wide):
    rng = np.random.default_rng(w * 257 + d)
    keys = (rng.integers(0, 2000, (w, d)) * 256 + np.arange(d)).tolist()
    right, seen = _replay(keys, w, d, 8 if wide else 16, wide, warps)
    assert seen == {(x, i) for x in range(w) for i in range(d)}
    want = [min(keys[xr + i][i] for i in range(d) if xr + i < w) for xr in range(w)]
    assert right == want


def test_shared_memory_of_the_widest_row():
    for threads in (384, 512):
        assert (3 * MAX_WIDTH + 3) // 4 * 16 + threads // 32 * SUMS_PER_WARP * 2 <= 227 * 1024


def _carry_replay(keys, w, d, k, seg, warps):
    """As _replay, of lanes that hold k disparities and carry the columns of S = min(k, pixels a warp
    covers) places a round; also the atomics a lane issues for a pixel."""
    ppw = 32 // seg
    s = min(k, ppw)
    rounds = -(-w // (warps * ppw))
    right, atomics = [NONE] * w, 0
    for warp in range(warps):
        for lane in range(32):
            sub, c = divmod(lane, seg)
            d0, rk, x = k * c, [NONE] * k, warp * rounds * ppw + sub

            def leave(xr, js):
                for j in js:
                    if 0 <= xr - j < w:
                        right[xr - j] = min(right[xr - j], rk[j])
                    else:
                        assert rk[j] == NONE or xr - j < 0

            for _ in range(rounds):
                key = [keys[x][d0 + j] if x < w and d0 + j < d else NONE for j in range(k)]
                rk = [min(rk[j - s], key[j]) if j >= s else key[j] for j in range(k)]
                leave(x - d0, range(k - s, k))
                atomics = max(atomics, s)
                x += ppw
            leave(x - s - d0, range(k - s))
    return right, atomics


@pytest.mark.parametrize("paths", [2, 4, 8])
@pytest.mark.parametrize("w,d", [(1, 1), (3, 16), (33, 64), (130, 65), (70, 128), (40, 129), (131, 160), (90, 192), (129, 256)])
def test_wide_slabs_carry_their_columns(w, d, paths):
    """Wide slabs' row loop: 8 disparities a lane, 16 for two paths past D = 128 (kernels.cuh: wta_form);
    no more than one atomic a lane and pixel of the warp."""
    dv = (d + 15) // 16 * 16
    k = 16 if paths == 2 and dv > 128 else 8
    seg = _lanes_per_pixel(dv, k)
    assert seg <= (16 if paths == 2 else 32)
    rng = np.random.default_rng(w * 257 + d)
    keys = (rng.integers(0, 2000, (w, d)) * 256 + np.arange(d)).tolist()
    right, atomics = _carry_replay(keys, w, d, k, seg, 8)
    assert right == [min(keys[xr + i][i] for i in range(d) if xr + i < w) for xr in range(w)]
    assert atomics <= 32 // seg
