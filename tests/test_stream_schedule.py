"""The streamed warp-per-pair schedule, step by step on the CPU.

The rules that say when a strip starts and ends, how many lanes make a group
and when a pair may be issued (csrc/sw_schedule.cuh) are compiled as they are;
a group of lanes is stepped through streams of pairs as csrc/sw_batched.cu:
wave_stream steps it.  At every step it is asked that a strip starts exactly
when it is due, on a lane that is free; that its blocks cover its columns; and
that the lane above held the strip above on the same columns one step before
(and on the columns before those, where a cell takes its diagonal from there).
"""
import ctypes
import subprocess

import numpy as np
import pytest

from clustkit_gb300 import build

HARNESS = r"""
#include <algorithm>
#include <vector>
#include "sw_schedule.cuh"
using namespace ck;

struct Lane {
    int cur = -1, s = 0, te = 0, jb = 0;     // slot, strip, last step, U * T + jb the first column
    int pend = -1, pend_s = 0, pend_t0 = 0, F = -1;
};
struct Held { int seq = -1, s = 0, j = 0; };  // what a lane computed in a step

// 0, or the number of the first rule that was broken
template <int R>
static int run(int G, const int32_t *pairs, int n, int serial, long long *steps) {
    const int SLOTS = WS_SLOTS * G / 32, U = WS_U;
    std::vector<Lane> lanes(G);
    std::vector<Held> before(G), before2(G), now(G);
    std::vector<WaveSlot> slots(SLOTS);
    std::vector<int> slot_seq(SLOTS, -1);
    for (auto &s : slots) s.live = 0;
    int T = 0, T_issue = -1, g_next = 0, seq = 0, q = 0, done = 0, strips = 0;
    bool exhausted = false;
    for (;; ++T) {
        if (T > 4000000) return 1;  // does not end
        if (!exhausted && T > T_issue && !slots[seq % SLOTS].live &&
            (!serial || seq == 0 || !slots[(seq - 1) % SLOTS].live)) {
            if (q >= n) {
                exhausted = true;
            } else {
                const int la = pairs[4 * q], lb = pairs[4 * q + 1], w = pairs[4 * q + 2], h = pairs[4 * q + 3];
                ++q;
                const int ns = wave_strips(R, la, lb, w, h);
                if (ns <= 0) {
                    ++done;
                } else {
                    WaveSlot &sl = slots[seq % SLOTS];
                    const int c0 = 1 + h - w, m00 = wave_block(R, c0, 0), first = std::min(ns, G);
                    int T0 = T;
                    for (int gl = 0; gl < G; ++gl) {
                        const int m = (gl - g_next) & (G - 1);
                        if (m < first) T0 = std::max(T0, (int)wave_earliest(R, c0, m00, m, lanes[gl].F, T));
                    }
                    sl.la = la; sl.lb = lb; sl.w = w; sl.h = h; sl.c0 = c0; sl.S = ns; sl.m00 = m00; sl.T0 = T0;
                    sl.live = 1;
                    slot_seq[seq % SLOTS] = seq;
                    for (int gl = 0; gl < G; ++gl) {
                        const int m = (gl - g_next) & (G - 1);
                        if (m >= first) continue;
                        Lane &l = lanes[gl];
                        if (l.pend >= 0) return 2;  // a strip not yet started is lost
                        l.pend = seq % SLOTS;
                        l.pend_s = m;
                        l.pend_t0 = strip_t0<R>(sl, m);
                        l.F = strip_te<R>(sl, m + G * ((ns - 1 - m) / G));
                    }
                    T_issue = strip_t0<R>(sl, ns - 1);
                    g_next += ns;
                    ++seq;
                }
            }
        }
        for (int gl = 0; gl < G; ++gl) {
            Lane &l = lanes[gl];
            if (l.pend >= 0 && T >= l.pend_t0) {
                if (T > l.pend_t0) return 3;  // late
                if (l.cur >= 0) return 4;     // the lane is not free
                const WaveSlot &sl = slots[l.pend];
                l.cur = l.pend;
                l.s = l.pend_s;
                l.pend = -1;
                l.te = strip_te<R>(sl, l.s);
                l.jb = sl.c0 + U * (sl.m00 - sl.T0 - l.s);
                const int lo = l.s * R + sl.c0, j0 = std::max(lo, 1), j1 = std::min(lo + R - 1 + 2 * sl.w, (int)sl.lb);
                if (U * T + l.jb > j0 || (j0 <= j1 && U * l.te + l.jb + U - 1 < j1)) return 5;  // columns left out
                ++strips;
            }
        }
        for (int gl = 0; gl < G; ++gl) {
            Lane &l = lanes[gl];
            now[gl] = Held{};
            if (l.cur < 0) continue;
            const WaveSlot &sl = slots[l.cur];
            const int j = U * T + l.jb, lo = l.s * R + sl.c0, top = l.s * R + sl.h + sl.w;
            now[gl] = Held{slot_seq[l.cur], l.s, j};
            // the first row reads the row above: in its band at column c when lo - 1 <= c <= top
            const Held &up = before[(gl + G - 1) & (G - 1)], &up2 = before2[(gl + G - 1) & (G - 1)];
            for (int u = 0; u < U && l.s > 0; ++u) {
                const int c = j + u;
                if (c < std::max(lo, 1) || c > std::min(lo + 2 * sl.w, (int)sl.lb)) continue;  // no cell
                if (c <= top && !(up.seq == now[gl].seq && up.s == l.s - 1 && up.j == j)) return 6;
                if (u == 0 && c - 1 >= 1 && c - 1 <= top &&
                    !(up2.seq == now[gl].seq && up2.s == l.s - 1 && up2.j == j - U)) return 7;
            }
            if (T == l.te) {
                if (l.s == sl.S - 1) {
                    slots[l.cur].live = 0;
                    ++done;
                } else if (l.s + G < sl.S) {
                    if (l.pend >= 0) return 8;
                    l.pend = l.cur;
                    l.pend_s = l.s + G;
                    l.pend_t0 = strip_t0<R>(sl, l.pend_s);
                }
                l.cur = -1;
            }
        }
        before2 = before;
        before = now;
        bool idle = exhausted;
        for (auto &l : lanes) idle = idle && l.cur < 0 && l.pend < 0;
        if (idle) break;
    }
    *steps = T;
    int want = 0;
    for (int i = 0; i < n; ++i) want += std::max(0, (int)wave_strips(R, pairs[4 * i], pairs[4 * i + 1], pairs[4 * i + 2], pairs[4 * i + 3]));
    return done != n || strips != want ? 9 : 0;
}

extern "C" {
int t_group(int R, int w) { return wave_group(R, w); }
int t_run(int R, int G, const int32_t *pairs, int n, int serial, long long *steps) {
    return R == 8 ? run<8>(G, pairs, n, serial, steps) : run<16>(G, pairs, n, serial, steps);
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    at = tmp_path_factory.mktemp("schedule")
    (at / "harness.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(build.CSRC), str(at / "harness.cpp"),
                    "-o", str(at / "harness.so")], check=True)
    return ctypes.CDLL(str(at / "harness.so"))


def _shapes(lib, w):
    """(rows, lanes, one pair at a time) of a call with band half-width w, as wave_shapes picks them."""
    g8, g16 = lib.t_group(8, w), lib.t_group(16, w)
    few = (8 if g8 else 16, 32)
    shapes = {(8, 8) if g8 == 8 else (16, g16), (8, g8) if g8 else (16, g16), few, (16, g16)}
    return [(R, G, 0) for R, G in sorted(shapes)] + [few + (1,)]


def _pairs(rng, n, w, max_rows, hinted):
    out = []
    for _ in range(n):
        kind = rng.integers(0, 4)
        la = int([rng.integers(1, 60), rng.integers(40, 300), rng.integers(200, 900), rng.integers(1, max_rows + 1)][kind])
        la = min(la, max_rows)
        lb = la + int(rng.integers(0, 3)) if rng.random() < 0.4 else la + int(rng.integers(0, 2 * la + 60))
        h = 0
        if hinted:
            h = int(rng.integers(-la, la + 1)) if rng.random() < 0.7 else int(rng.choice([-la, la]))
        out.append((la, lb, lb if w <= 0 or lb <= 50 else w, h))
    return np.array(out, np.int32)


def _run(lib, R, G, serial, pairs):
    steps = ctypes.c_longlong()
    rc = lib.t_run(R, G, pairs.ctypes.data_as(ctypes.c_void_p), len(pairs), serial, ctypes.byref(steps))
    return rc, steps.value


@pytest.mark.parametrize("hinted", [False, True])
@pytest.mark.parametrize("w0", range(1, 264, 16))
def test_every_band_streams_without_a_late_strip(lib, w0, hinted):
    for w in range(w0, min(w0 + 16, 264)):
        rng = np.random.default_rng(1000 * w + hinted)
        for R, G, serial in _shapes(lib, w):
            assert G in (8, 16, 32) and (serial or 2 * w <= (G - 1) * (R + 2) + 1)
            for n in (1, 40):
                rc, _ = _run(lib, R, G, serial, _pairs(rng, n, w, 2500, hinted))
                assert rc == 0, (w, R, G, serial, n)


@pytest.mark.parametrize("w", [0, -1, 264, 279, 280, 600, 4000])
def test_bands_too_wide_to_rotate(lib, w):
    """The whole matrix, or a band past 263: every pair has at most 512 rows."""
    rng = np.random.default_rng(abs(w))
    for hinted in (False, True):
        for R, G, serial in _shapes(lib, w):
            assert (R, G) == (16, 32)
            for n in (1, 60):
                assert _run(lib, R, G, serial, _pairs(rng, n, w, 512, hinted))[0] == 0


@pytest.mark.parametrize("R", [8, 16])
def test_group_changes_where_rotation_ends(lib, R):
    """The last band of each group size runs without a gap between a lane's
    strips; one more would start strips late."""
    edges = [w for w in range(1, 400) if lib.t_group(R, w) != lib.t_group(R, w + 1)]
    assert edges == ([35, 75, 155] if R == 8 else [63, 135])
    for w, G in zip(edges, (8, 16, 32)):
        pair = np.array([[3000, 3400, w, 0]] * 3, np.int32)
        assert lib.t_group(R, w) == G
        assert _run(lib, R, G, 0, pair)[0] == 0
        pair[:, 2] = w + 1 + R  # past the bound by more than its slack
        assert _run(lib, R, G, 0, pair)[0] == 3
