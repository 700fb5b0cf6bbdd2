"""CPU replay of the packed across-lanes scan form of the path aggregation
(vx-rs_b200/csrc/aggregate_packed.cu): its words, plain 32-bit adds, per-half
minima, lane geometry and serial recomputation, in numpy, against the shader's
serial order (vx-vision/shaders/SGMStereo.metal:120-172) on random and
adversarial cost sequences, up to the edge of the penalties the form accepts."""
import numpy as np
import pytest

import oracle
import vx_sgm

M32 = 0xFFFFFFFF
LATENCY, THROUGHPUT = 1, 2


def packed_scan_ok(p1, p2, dv):
    return (128 + p1) * dv + p1 + p2 + 66 <= 65536 and p1 + p2 + 128 < 32768


def packed_geometry(nd, dv, kind):
    """(K, segment lanes, pads) as packed_geometry in csrc/kernels.cuh."""
    lat = kind == LATENCY
    ks = [12 if lat else 24, 8 if lat else (32 if dv >= 64 else 16), 8 if lat else 16]
    for k in ks:
        lanes = dv // k
        if nd == dv and dv % k == 0 and lanes & (lanes - 1) == 0:
            return k, lanes, False
    lanes = dv // ks[2]
    seg = 1
    while seg < lanes:
        seg <<= 1
    return ks[2], seg, True


def halves(w):
    return w & 0xFFFF, w >> 16


def word(lo, hi):
    return (np.asarray(lo, np.int64) & 0xFFFF) | (np.asarray(hi, np.int64) & 0xFFFF) << 16


def vadd2(a, b):
    (al, ah), (bl, bh) = halves(a), halves(b)
    return word(al + bl, ah + bh)


def vmin2(*ws):
    lo = np.minimum.reduce([halves(w)[0] for w in ws])
    hi = np.minimum.reduce([halves(w)[1] for w in ws])
    return word(lo, hi)


def serial(L, m, C, D, p1, p2):
    y, prev = np.zeros(D, np.int64), 0
    for d in range(D):
        q1 = 0xFFFF if d == 0 else (prev + p1) & 0xFFFF
        q2 = 0xFFFF if d == D - 1 else (int(L[d + 1]) + p1) & 0xFFFF
        prev = (int(C[d]) + min(int(L[d]), q1, q2, (m + p2) & 0xFFFF) - m) & 0xFFFF
        y[d] = prev
    return y


class Replay:
    def __init__(self, nd, p1, p2, kind):
        self.D, self.p1, self.p2 = nd, p1, p2
        self.dv = (nd + 15) // 16 * 16
        self.K, self.seg, self.pads = packed_geometry(nd, self.dv, kind)
        self.N = self.K // 2
        d = np.arange(self.seg)[:, None] * self.K + np.arange(self.N)[None, :]      # lane, word: low half's d
        self.keep = word(np.where(d < nd, 0xFFFF, 0), np.where(d + self.N < nd, 0xFFFF, 0))
        self.L = np.zeros((self.seg, self.N), np.int64)
        self.mm = 0
        self.redone = 0

    def values(self):
        """The vector in d order."""
        lo, hi = halves(self.L)
        return np.concatenate([lo, hi], 1).reshape(-1)[:self.D]

    def step(self, C):
        K, N, seg, p1, p2 = self.K, self.N, self.seg, self.p1, self.p2
        c = np.zeros(seg * K, np.int64)
        c[:len(C)] = C                                     # the volume's pads are 0
        c = c.reshape(seg, K)
        cw = word(c[:, :N], c[:, N:])
        bu, x2 = 0x10000 - 64 * self.dv - p2 - 65, 0x10001
        p1x2, p2x2, np1x2 = p1 * x2, p2 * x2, ((0x10000 - p1) & 0xFFFF) * x2
        fill = 0xFFFF - p1
        d0 = np.arange(seg, dtype=np.int64) * K
        w0 = d0 | (d0 + N) << 16
        lane_sum = c.sum(1)
        below = np.cumsum(lane_sum) - lane_sum
        e = ((bu - p1) * x2 - w0 * p1 - below * x2 - (c[:, :N].sum(1) << 16)) & M32
        m = self.mm & 0xFFFF
        L = self.L
        M = vadd2(L, np.full_like(L, p1x2))
        nb = np.append(M[1:, 0] & 0xFFFF, 0xFFFF)
        nbw = word(M[:, 0] >> 16, nb)
        o3, q = (self.mm + p2x2) & M32, (p1x2 - self.mm) & M32
        r = (e + w0 * m) & M32
        R, U = np.zeros_like(L), np.zeros_like(L)
        for j in range(N):
            U[:, j] = (vmin2(L[:, j], M[:, j + 1] if j + 1 < N else nbw, np.full(seg, o3)) + r) & M32
            r = (r - cw[:, j] - q) & M32
            R[:, j] = r
        T = vmin2(*[U[:, j] for j in range(N)])
        lane_min = np.minimum(*halves(T))
        z_below = np.append(0xFFFF, np.minimum.accumulate(lane_min)[:-1])
        z = vmin2(word(z_below, z_below), word(np.full(seg, 0xFFFF), T & 0xFFFF))
        M2 = np.zeros_like(L)
        for j in range(N):
            z = vmin2(z, U[:, j])
            (zl, zh), (rl, rh) = halves(z), halves(R[:, j])
            M2[:, j] = word(zl - rl, zh - rh)
        M2 |= ~self.keep & M32
        y = vadd2(M2, np.full_like(L, np1x2))
        signed = lambda w: np.where(np.concatenate(halves(w), 1) >= 0x8000, np.concatenate(halves(w), 1) - 0x10000,  # noqa: E731
                                    np.concatenate(halves(w), 1))
        low = int(signed((y & self.keep) | (0x7FFF7FFF & ~self.keep & M32)).min())
        self.mm = low * x2
        if low < 0 or m > 64:
            lo, hi = halves(M2 & self.keep)
            if m > 64 or (lo & 0x8000).any() or (hi & 0x8000).any():
                self.redone += 1
                old = np.concatenate(halves(L), 1).reshape(-1)
                new = np.full(seg * K, fill, np.int64)
                new[:self.D] = serial(old[:self.D], m, c.reshape(-1), self.D, p1, p2)
                new = new.reshape(seg, K)
                y = word(new[:, :N], new[:, N:])
            lifted = np.concatenate(halves(y | (~self.keep & M32)), 1)
            self.mm = int(lifted.min()) * x2
        self.L = y


def run_sequence(nd, p1, p2, kind, costs):
    r = Replay(nd, p1, p2, kind)
    L, m = np.zeros(nd, np.int64), 0
    want_wraps = 0
    for t, C in enumerate(costs):
        want = serial(L, m, C, nd, p1, p2)
        r.step(C)
        got = r.values()
        assert np.array_equal(got, want), (t, np.argwhere(got != want)[:4])
        L, m = want, int(want.min())
        assert (r.mm & 0xFFFF) == m
        want_wraps += int((want >= 0x8000).any())
    return r.redone, want_wraps


@pytest.mark.parametrize("kind", [LATENCY, THROUGHPUT])
@pytest.mark.parametrize("nd,p1,p2", [(64, 10, 120), (128, 10, 120), (192, 10, 120), (256, 10, 120), (48, 10, 120),
                                      (96, 15, 300), (16, 3690, 400), (1, 10, 120), (7, 0, 120), (100, 10, 120),
                                      (200, 3, 2000), (256, 126, 120), (128, 0, 20000), (32, 1800, 1000),
                                      (80, 590, 7000)])
def test_packed_words_reproduce_the_serial_order(nd, p1, p2, kind):
    """Random costs of several shapes: uniform 0..64, low ones (a good match nearby), runs of 64 (left of the
    image) next to zeros, and sequences that drive the minimum up and then the costs down, which makes values wrap."""
    assert packed_scan_ok(p1, p2, (nd + 15) // 16 * 16)
    rng = np.random.default_rng(nd * 7 + p1)
    steps = 14
    shapes = [rng.integers(0, 65, (steps, nd)), rng.integers(0, 12, (steps, nd)),
              np.where(rng.random((steps, nd)) < 0.5, 64, 0),
              np.where((np.arange(steps) % 3 == 2)[:, None], rng.integers(0, 3, (steps, nd)), 64 - rng.integers(0, 3, (steps, nd))),
              np.where(np.arange(nd)[None, :] > np.arange(steps)[:, None], 64, rng.integers(0, 25, (steps, nd)))]
    redone = wraps = 0
    for costs in shapes:
        a, b = run_sequence(nd, p1, p2, kind, costs)
        redone, wraps = redone + a, wraps + b
    if p1 <= 10 and nd > 1:
        assert wraps > 0 and redone > 0      # both kinds of wrapped pixel were met


@pytest.mark.parametrize("nd,rx,ry", [(64, 2, 2), (192, 4, 3), (100, 2, 2)])
def test_packed_form_reproduces_the_path_costs(nd, rx, ry):
    w, h = 60, 5
    L, R, _ = vx_sgm.synth_pair(1, w, h, 0, w // 2, nd)
    cl, cr = oracle.census(L, rx, ry), oracle.census(R, rx, ry)
    want = oracle.path_costs(cl, cr, nd, 10, 120, 1, 0)
    for y in range(h):
        r = Replay(nd, 10, 120, LATENCY if y % 2 else THROUGHPUT)
        for x in range(w):
            C = np.array([int(cl[y, x] ^ cr[y, x - d]).bit_count() if d <= x else 64 for d in range(nd)])
            r.step(C)
            assert np.array_equal(r.values(), want[y, x]), (x, y)


def test_geometry_covers_every_disparity_count():
    for kind in (LATENCY, THROUGHPUT):
        for nd in range(1, 257):
            dv = (nd + 15) // 16 * 16
            k, seg, pads = packed_geometry(nd, dv, kind)
            assert seg in (1, 2, 4, 8, 16, 32) and seg * k >= dv and (pads or seg * k == nd)
            assert dv % k == 0 or not pads            # a lane's bytes lie inside the vector or past it
            # the variants that are compiled
            if kind == LATENCY:
                assert (k == 8 and seg >= 2) or (k == 12 and not pads and seg in (4, 8, 16))
            elif pads:
                assert k == 16 and seg <= 16
            else:
                assert (k, seg) in ((16, 1), (16, 2), (16, 4), (24, 2), (24, 4), (24, 8), (32, 2), (32, 4), (32, 8))
