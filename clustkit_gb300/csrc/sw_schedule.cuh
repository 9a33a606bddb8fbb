// sw_schedule.cuh -- when the strips of the warp-per-pair phase run: integer
// rules alone, for the kernel (sw_batched.cu: wave_stream, where the schedule is
// described) and for host code.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define CK_HD __host__ __device__ __forceinline__
#else
#define CK_HD inline
#endif

namespace ck {

constexpr int WS_U = 2;       // columns a step
constexpr int WS_SLOTS = 16;  // pairs a warp's groups have in flight, in its slots in shared memory

struct WaveSlot {
    unsigned long long acc;   // score << 27 | (16383 - row) << 13 | matches
    int64_t a_off, b_off;     // residues of the row and column sequences
    int64_t p;                // pair index
    int32_t la, lb, w, h, c0, S, m00, T0;
    int32_t gs;               // running best score of the pair (first-maximum trigger)
    int32_t live;
};

// strips of R rows that hold a column of the matrix
CK_HD int32_t wave_strips(int32_t R, int32_t la, int32_t lb, int32_t w, int32_t h) {
    const int32_t n = (la + R - 1) / R;
    const int64_t lim = (int64_t)lb - 1 - h + w;
    const int64_t s_lim = lim < 0 ? 0 : lim / R + 1;
    return s_lim < n ? (int32_t)s_lim : n;
}

// blocks between the band's first column c0 and the first column of strip s
CK_HD int32_t wave_block(int32_t R, int32_t c0, int32_t s) {
    const int32_t lo = s * R + c0;
    return ((lo > 1 ? lo : 1) - c0) / WS_U;
}

// steps at which strip s starts (its first column's block) and ends (its last's)
template <int R>
CK_HD int32_t strip_t0(const WaveSlot &sl, int32_t s) {
    return sl.T0 + s + wave_block(R, sl.c0, s) - sl.m00;
}
template <int R>
CK_HD int32_t strip_te(const WaveSlot &sl, int32_t s) {
    const int32_t hi = s * R + sl.c0 + R - 1 + 2 * sl.w;
    const int32_t J1 = hi < sl.lb ? hi : sl.lb;
    const int32_t te = sl.T0 + s + (J1 - sl.c0) / WS_U - sl.m00;
    const int32_t t0 = strip_t0<R>(sl, s);
    return te > t0 ? te : t0;  // a strip whose band lies left of column 1 ends where it starts
}

// The earliest T0 of a pair issued at step T for the lane of its strip m, which
// is busy up to step F.
CK_HD int32_t wave_earliest(int32_t R, int32_t c0, int32_t m00, int32_t m, int32_t F, int32_t T) {
    const int32_t r = F + 1 - m - (wave_block(R, c0, m) - m00);
    return r > T ? r : T;
}

// The smallest group that strips of R rows can rotate through in a band of
// half-width w.  A lane may start its next strip, G strips on, once its last is
// done: that one's last column is R - 1 + 2w after its first row's first, the
// other's first at least G R after it and G steps later, so
// 2w <= (G - 1)(R + U) + 1 is enough (clipping at the matrix only shortens the
// first).  Pairs of at most G strips never rotate: those with a longer side of
// at most 50, whose band is the whole matrix, have at most 7 strips of 8 rows;
// and where the band is too wide for 32 lanes of 16 rows, every pair has at most
// 512 rows (wave_split), 32 strips.  0: none.
inline int32_t wave_group(int32_t R, int32_t w) {
    if (w >= 1)
        for (int32_t G = 8; G <= 32; G <<= 1)
            if (2 * (int64_t)w <= (G - 1) * (R + WS_U) + 1) return G;
    return R == 16 ? 32 : 0;
}

}  // namespace ck
