"""CPU replay of the packed scan kernels' own words (vx-rs_b200/csrc/aggregate_packed.cuh): the
biased sums V and differences U = A - P1 - v as 32-bit words of two halves, their prefix minimum,
y = V + z, the signed test for wrapped values and the redo, against the shader's serial order
(vx-vision/shaders/SGMStereo.metal:120-172), at the edges of the penalties the kernels take. In
every pixel that is not redone no half may carry into or borrow from the other. And the compiled
kernels against the geometries a plan can have."""
import re

import numpy as np
import pytest

from host_gpu import host_gpu  # noqa: F401
from test_packed_scan_replay import (LATENCY, M32, THROUGHPUT, halves, packed_geometry, packed_scan_ok, serial, vadd2,
                                     vmin2, word)


class Kernel:
    def __init__(self, nd, p1, p2, kind):
        self.D, self.p1, self.p2 = nd, p1, p2
        self.dv = (nd + 15) // 16 * 16
        self.K, self.seg, self.pads = packed_geometry(nd, self.dv, kind)
        self.N = self.K // 2
        d = np.arange(self.seg)[:, None] * self.K + np.arange(self.N)[None, :]
        self.real = d < nd, d + self.N < nd
        self.keep = word(*(np.where(r, 0xFFFF, 0) for r in self.real))
        self.L = np.zeros((self.seg, self.N), np.int64)
        self.mm, self.forced, self.redone, self.looked = 0, False, 0, 0

    def values(self):
        return np.concatenate(halves(self.L), 1).reshape(-1)[:self.D]

    def add(self, a, b, exact, j=0):
        """a + b (a pair of integers) as a 32-bit word; exact: the halves of word j's real disparities
        must stay in 16 bits. (A pad's high half is a pad too: what its low half carries stays there.)"""
        sums = [x + y for x, y in zip(halves(a), b)]
        if exact:
            for s, real in zip(sums, self.real):
                s = s[real[:, j]]
                assert s.size == 0 or (s.min() >= 0 and s.max() <= 0xFFFF)
        return (sums[0] + (sums[1] << 16)) & M32

    def step(self, C):
        K, N, seg, p1, p2 = self.K, self.N, self.seg, self.p1, self.p2
        c = np.zeros(seg * K, np.int64)
        c[:len(C)] = C
        c = c.reshape(seg, K)
        m = self.mm & 0xFFFF
        exact = m <= 64
        bv = 64 * self.dv + p2 + 65
        fill, L = 0xFFFF - p1, self.L
        d0 = np.arange(seg, dtype=np.int64) * K
        below = np.cumsum(c.sum(1)) - c.sum(1)
        base = word(bv + d0 * p1, bv + (d0 + N) * p1)
        base = self.add(base, (below, below + c[:, :N].sum(1)), exact)
        vb = self.add(base, (-d0 * m, -(d0 + N) * m), exact)
        nb = np.append(L[1:, 0] & 0xFFFF, fill)
        nbw = word(halves(L[:, 0])[1], nb)
        p1x2 = np.full(seg, p1 * 0x10001)
        o3 = np.full(seg, word(m + p2, m + p2))
        V, y = np.zeros_like(L), np.zeros_like(L)
        for j in range(N):
            vp = vb if j == 0 else V[:, j - 1]
            V[:, j] = self.add(vp, (c[:, j] + p1 - m, c[:, j + N] + p1 - m), exact, j)
            a = vmin2(L[:, j], vadd2(L[:, j + 1] if j + 1 < N else nbw, p1x2), o3)
            y[:, j] = self.add(a, (65536 - p1 - halves(vp)[0], 65536 - p1 - halves(vp)[1]), exact, j)   # U
        T = vmin2(*[y[:, j] for j in range(N)])
        lane = np.minimum(*halves(T))
        under = np.append(0xFFFF, np.minimum.accumulate(lane)[:-1])
        z = word(under, np.minimum(under, T & 0xFFFF))
        for j in range(N):
            z = vmin2(z, y[:, j])
            y[:, j] = vadd2(V[:, j], z)
        y = (y & self.keep) | (fill * 0x10001 & ~self.keep & M32)
        lifted = np.concatenate(halves((y & self.keep) | (0x7FFF7FFF & ~self.keep & M32)), 1)
        low = int(np.where(lifted >= 0x8000, lifted - 0x10000, lifted).min())
        self.mm = (low & 0xFFFF) * 0x10001
        if low < 0 or self.forced:
            self.looked += 1
            wrapped = halves(vadd2(y, np.full_like(y, p1 * 0x10001)) & self.keep)
            if m > 64 or (wrapped[0] & 0x8000).any() or (wrapped[1] & 0x8000).any():
                self.redone += 1
                old = np.concatenate(halves(L), 1).reshape(-1)
                new = np.full(seg * K, fill, np.int64)
                new[:self.D] = serial(old[:self.D], m, c.reshape(-1), self.D, p1, p2)
                new = new.reshape(seg, K)
                y = word(new[:, :N], new[:, N:])
            lo = int(np.concatenate(halves(y | (~self.keep & M32)), 1).min())
            self.mm, self.forced = lo * 0x10001, lo > 64
        self.L = y


def edge_penalties(dv):
    """Penalties at the edge of the accepted range: the largest P1, the largest P2, both between, none."""
    top = lambda f: max(p for p in range(0, 32768) if packed_scan_ok(*f(p), dv))  # noqa: E731
    p1 = top(lambda p: (p, 0))
    p2 = top(lambda p: (0, p))
    mid = p1 // 2
    out = {(p1, 0), (0, p2), (mid, top(lambda p: (mid, p))), (0, 0), (10, 120)}
    for a, b in out:
        assert packed_scan_ok(a, b, dv)
    assert not packed_scan_ok(p1 + 1, 0, dv) and not packed_scan_ok(0, p2 + 1, dv)
    return sorted(out)


@pytest.mark.parametrize("kind", [LATENCY, THROUGHPUT])
@pytest.mark.parametrize("nd", [1, 15, 16, 31, 48, 64, 80, 96, 100, 128, 144, 192, 240, 255, 256])
def test_kernel_words_at_the_edges_of_the_penalties(nd, kind):
    rng = np.random.default_rng(nd)
    steps = 9
    t = np.arange(steps)[:, None]
    shapes = [rng.integers(0, 65, (steps, nd)), np.where(rng.random((steps, nd)) < 0.5, 64, 0), np.zeros((steps, nd), int),
              np.full((steps, nd), 64), np.where(t % 2, 64, 0) + np.zeros((1, nd), int),
              np.where(np.arange(nd)[None, :] > nd - 2, 0, 64) * (t > 0),
              np.where((t % 3 == 2), rng.integers(0, 3, (steps, nd)), 64 - rng.integers(0, 3, (steps, nd)))]
    for p1, p2 in edge_penalties((nd + 15) // 16 * 16):
        redone = 0
        for costs in shapes:
            k = Kernel(nd, p1, p2, kind)
            L, m = np.zeros(nd, np.int64), 0
            for C in costs:
                k.step(C)
                L = serial(L, m, C, nd, p1, p2)
                m = int(L.min())
                assert np.array_equal(k.values(), L) and (k.mm & 0xFFFF) == m, (p1, p2)
            redone += k.redone
        if (p1, p2) == (10, 120) and nd >= 16:
            assert redone > 0


def test_a_kernel_for_every_geometry_and_no_other(host_gpu):  # noqa: F811
    for kind, ks in ((LATENCY, (8, 12)), (THROUGHPUT, (16, 24, 32))):
        want = {packed_geometry(nd, (nd + 15) // 16 * 16, kind) for nd in range(1, 257)}
        assert len(want) == 13
        names = [re.search(r"packed_kernel<(\d+), (\d+), (\w+), (\w+)>", n)
                 for n in host_gpu.kernels()]
        compiled = {(int(m[1]), int(m[2]), m[3] == "true", m[4]) for m in names if m and int(m[1]) in ks}
        assert {c[:3] for c in compiled} == want
        assert len(compiled) == 2 * len(want)    # full and pooled shadows
