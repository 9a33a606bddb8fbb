// sketch.cu -- bottom-s MinHash sketches (clustkit/sketch.py:17-183).
//
// Output for a sequence of length L: s zeros if L < k; otherwise the sorted
// multiset of the s smallest values fmix64(v_i ^ seed) over the L-k+1 k-mers,
// where v_i = sum_m code[i+m] * alphabet^(k-1-m) in wrapping uint64 (the
// value clustkit's rolling update produces), padded with UINT64_MAX.
//
// One warp per sequence.  sketch_select_kernel (s up to 1,768) hashes
// the k-mers against a threshold that a uniform hash would leave between s and
// C of (C a power of two a few standard deviations above s), keeps those at or
// below it in shared memory, and sorts them in registers; it is bound by
// instruction issue (hashing and the sort are about half each).  Larger
// sketches take sketch_kernel, which keeps the s best so far in shared memory
// and merges new ones in by sorting there.
#include <cmath>
#include <type_traits>

#include "ck_common.cuh"

namespace ck {

__device__ __forceinline__ uint64_t fmix64(uint64_t key, uint64_t seed) {
    uint64_t h = key ^ seed;
    h ^= h >> 33;
    h *= 0xFF51AFD7ED558CCDULL;
    h ^= h >> 33;
    h *= 0xC4CEB9FE1A85EC53ULL;
    h ^= h >> 33;
    return h;
}

// C = 32 * NPL 32-bit keys, lane l holding positions l * NPL .. l * NPL + NPL - 1,
// into ascending order: a bitonic network in which a stride below NPL pairs
// two registers and a larger one two lanes.
template <int NPL>
__device__ __forceinline__ void warp_sort_keys(uint32_t (&v)[NPL], int lane) {
    auto within = [&](auto stride, bool up_lane, int k_reg) {
        constexpr int J = decltype(stride)::value;
#pragma unroll
        for (int r = 0; r < NPL; ++r) {
            if (r & J) continue;
            const bool up = k_reg ? (r & k_reg) == 0 : up_lane;
            const uint32_t a = v[r], b = v[r | J];
            v[r] = up ? min(a, b) : max(a, b);
            v[r | J] = up ? max(a, b) : min(a, b);
        }
    };
    auto merge_within = [&](bool up_lane, int k_reg) {
        if constexpr (NPL > 32) within(std::integral_constant<int, 32>{}, up_lane, k_reg);
        if constexpr (NPL > 16) within(std::integral_constant<int, 16>{}, up_lane, k_reg);
        if constexpr (NPL > 8) within(std::integral_constant<int, 8>{}, up_lane, k_reg);
        if constexpr (NPL > 4) within(std::integral_constant<int, 4>{}, up_lane, k_reg);
        if constexpr (NPL > 2) within(std::integral_constant<int, 2>{}, up_lane, k_reg);
        within(std::integral_constant<int, 1>{}, up_lane, k_reg);
    };
    // runs of 2 .. NPL / 2 positions: registers alone, the direction by register
    if constexpr (NPL > 2) within(std::integral_constant<int, 1>{}, false, 2);
    if constexpr (NPL > 4) {
        within(std::integral_constant<int, 2>{}, false, 4);
        within(std::integral_constant<int, 1>{}, false, 4);
    }
    if constexpr (NPL > 8) {
        within(std::integral_constant<int, 4>{}, false, 8);
        within(std::integral_constant<int, 2>{}, false, 8);
        within(std::integral_constant<int, 1>{}, false, 8);
    }
    if constexpr (NPL > 16) {
        within(std::integral_constant<int, 8>{}, false, 16);
        within(std::integral_constant<int, 4>{}, false, 16);
        within(std::integral_constant<int, 2>{}, false, 16);
        within(std::integral_constant<int, 1>{}, false, 16);
    }
    if constexpr (NPL > 32) {
        within(std::integral_constant<int, 16>{}, false, 32);
        within(std::integral_constant<int, 8>{}, false, 32);
        within(std::integral_constant<int, 4>{}, false, 32);
        within(std::integral_constant<int, 2>{}, false, 32);
        within(std::integral_constant<int, 1>{}, false, 32);
    }
    // runs of NPL positions, then of 2, 4, .. 32 lanes' positions
    merge_within((lane & 1) == 0, 0);
#pragma unroll 1
    for (int k = 2; k <= 32; k <<= 1) {
        const bool up = (lane & k) == 0;
#pragma unroll 1
        for (int j = k >> 1; j > 0; j >>= 1) {
            const bool keep_min = ((lane & j) == 0) == up;
#pragma unroll
            for (int r = 0; r < NPL; ++r) {
                const uint32_t o = __shfl_xor_sync(0xffffffffu, v[r], j);
                v[r] = keep_min ? min(v[r], o) : max(v[r], o);
            }
        }
        merge_within(up, 0);
    }
}

// Value of the k-mer at p; V is 32 bits wide where every value fits.
template <class V>
__device__ __forceinline__ uint64_t kmer_value(const uint8_t *p, int32_t k, V alphabet) {
    V v = 0;
#pragma unroll 5
    for (int32_t m = 0; m < k; ++m) v = v * alphabet + (V)__ldg(p + m);
    return (uint64_t)v;
}

// Sketches by threshold: with nk > C hashes a threshold that leaves about `aim`
// of them (s < aim < C) if they are spread evenly.  A count outside [s, C] -- one
// random sequence in a thousand, and many repeats, whose k-mers come in many
// copies -- takes a second pass that needs no threshold: it sorts whenever the
// buffer is full and goes on below the s-th smallest so far.  (Moving the
// threshold until the count fits took up to 66 passes where one value has more
// than C - s copies.  Going on from a full buffer in the first pass costs its
// loop a test, 5 % of the whole.)
// The hashes are sorted by their leading bits (as many as fit beside the slot
// number in 32 bits: a compare-exchange is then one instruction a key, not
// the five or six that 64-bit keys take), and the few neighbours whose leading
// bits agree are put right in shared memory.
// 200,000 sequences (median 300 residues), k = 5, s = 128: 3.62 -> 0.45 ms
// (sketch_kernel, sorting 64-bit keys in shared memory, before).  5,000 of 2,000
// residues: random ones 54 us, repeats of 4 with 2 % changed 106 (sketch_kernel
// 279 and 227; by moving the threshold 54 and 2,117).
// warps of a block: 8 while their buffers fit 48 KB, else as many as do (C <= 2048: 16 KB a warp)
template <int NPL>
constexpr int select_warps() { return NPL <= 16 ? 8 : 48 * 1024 / (32 * NPL * 8); }
// resident blocks: registers for as many as the buffers leave room for (NPL >= 32), or without spills
template <int NPL>
constexpr int select_blocks() { return NPL >= 16 ? 4 : 6; }

template <int NPL, class V>
__global__ void __launch_bounds__(32 * select_warps<NPL>(), select_blocks<NPL>())
sketch_select_kernel(const uint8_t *__restrict__ flat, int64_t flat_len, const int64_t *__restrict__ offsets,
                     const int32_t *__restrict__ lengths, int64_t N, int32_t k, int32_t s, int32_t aim, V alphabet,
                     uint64_t seed, uint64_t *__restrict__ out, int32_t *err) {
    constexpr int C = 32 * NPL;
    constexpr int IDX_BITS = NPL == 2 ? 6 : NPL == 4 ? 7 : NPL == 8 ? 8 : NPL == 16 ? 9 : NPL == 32 ? 10 : 11;
    constexpr uint32_t FULL = 0xffffffffu;
    extern __shared__ uint64_t s_buf[];
    const int lane = threadIdx.x & 31;
    uint64_t *buf = s_buf + (size_t)(threadIdx.x >> 5) * C;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const uint64_t MAXV = ~0ULL;

    for (int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < N; q += warps) {
        uint64_t *o = out + q * (int64_t)s;
        const int32_t L = lengths[q];
        const int64_t off = offsets[q];
        const bool bad = L < 0 || off < 0 || off + L > flat_len;
        if (bad || L < k) {
            if (bad && lane == 0) atomicOr(err, ERRBIT_SEQ_EXTENT);
            for (int t = lane; t < s; t += 32) o[t] = 0ULL;
            continue;
        }
        const uint8_t *seq = flat + off;
        const int32_t nk = L - k + 1;
        auto hash = [&](int32_t i) { return fmix64(kmer_value<V>(seq + i, k, alphabet), seed); };
        // hashes below cap into buf (the first C of them); their number.  (One
        // equal to MAXV may be left out: the padding stands for it.)
        uint64_t cap = nk <= C ? MAXV : MAXV / (uint64_t)nk * (uint64_t)aim;
        int32_t cnt = 0;
        for (int32_t base = 0; base < nk; base += 32) {
            const int32_t i = base + lane;
            uint64_t hv = 0;
            bool take = false;
            if (i < nk) {
                hv = hash(i);
                take = hv < cap;
            }
            const uint32_t bal = __ballot_sync(FULL, take);
            const int32_t at = cnt + __popc(bal & ((1u << lane) - 1u));
            if (take && at < C) buf[at] = hv;
            cnt += __popc(bal);
        }
        int32_t next = nk;  // the second pass's next k-mer
        if (cnt > C || (cnt < s && nk > C)) {
            if (cnt < s) cap = MAXV;
            cnt = next = 0;
        }
        for (;;) {
            __syncwarp();
            while (next < nk && cnt + 32 <= C) {
                const int32_t i = next + lane;
                uint64_t hv = 0;
                bool take = false;
                if (i < nk) {
                    hv = hash(i);
                    take = hv < cap;
                }
                const uint32_t bal = __ballot_sync(FULL, take);
                if (take) buf[cnt + __popc(bal & ((1u << lane) - 1u))] = hv;
                cnt += __popc(bal);
                next += 32;
            }
            for (int t = cnt + lane; t < C; t += 32) buf[t] = MAXV;
            __syncwarp();
            // sort keys: leading bits of the hash (none is above cap), then the slot
            const int width = 64 - __clzll((long long)cap);
            const int shift = width > 32 - IDX_BITS ? width - (32 - IDX_BITS) : 0;
            uint32_t v[NPL];
#pragma unroll
            for (int r = 0; r < NPL; ++r) {
                const int t = r * 32 + lane;  // any order will do here: neighbouring lanes read neighbouring slots
                v[r] = t < cnt ? ((uint32_t)(buf[t] >> shift) << IDX_BITS) | (uint32_t)t : 0xffffffffu;
            }
            warp_sort_keys<NPL>(v, lane);
            // slots -> values in place (read, then written).  A pad key names slot
            // C - 1, which holds MAXV whenever there is a pad
            uint64_t val[NPL];
#pragma unroll
            for (int r = 0; r < NPL; ++r) val[r] = buf[v[r] & (C - 1)];
            __syncwarp();
#pragma unroll
            for (int r = 0; r < NPL; ++r) buf[lane * NPL + r] = val[r];
            __syncwarp();
            // neighbours with equal leading bits: exchanged until none is out of order
            for (;;) {
                bool moved = false;
                for (int par = 0; par < 2; ++par) {
                    for (int t = 2 * lane + par; t + 1 < cnt; t += 64) {
                        const uint64_t a = buf[t], b = buf[t + 1];
                        if (a > b) { buf[t] = b; buf[t + 1] = a; moved = true; }
                    }
                    __syncwarp();
                }
                if (!__any_sync(FULL, moved)) break;
            }
            if (next >= nk) break;
            cnt = s;  // of a full buffer (s + 32 <= C): only what is below the largest of these matters now
            cap = buf[s - 1];
        }
        for (int t = lane; t < s; t += 32) o[t] = t < cnt ? buf[t] : MAXV;
        __syncwarp();
    }
}

__device__ __forceinline__ void warp_bitonic_sort(uint64_t *buf, int cap, int lane) {
    for (int k = 2; k <= cap; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int t = lane; t < (cap >> 1); t += 32) {
                const int i = 2 * j * (t / j) + (t % j);
                const int ixj = i + j;
                const bool up = (i & k) == 0;
                const uint64_t a = buf[i], b = buf[ixj];
                if ((a > b) == up) { buf[i] = b; buf[ixj] = a; }
            }
            __syncwarp();
        }
    }
}

__global__ void sketch_kernel(const uint8_t *__restrict__ flat, int64_t flat_len,
                              const int64_t *__restrict__ offsets, const int32_t *__restrict__ lengths,
                              int64_t N, int32_t k, int32_t s, int32_t BUF, uint64_t alphabet,
                              uint64_t seed, uint64_t *__restrict__ out, int32_t *err) {
    extern __shared__ uint64_t s_buf[];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const int cap = 2 * BUF;
    uint64_t *buf = s_buf + (size_t)wib * cap;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const uint64_t MAXV = ~0ULL;

    for (int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < N; q += warps) {
        uint64_t *o = out + q * (int64_t)s;
        const int32_t L = lengths[q];
        const int64_t off = offsets[q];
        if (L < 0 || off < 0 || off + L > flat_len) {
            if (lane == 0) atomicOr(err, ERRBIT_SEQ_EXTENT);
            for (int t = lane; t < s; t += 32) o[t] = 0ULL;
            continue;
        }
        if (L < k) {
            for (int t = lane; t < s; t += 32) o[t] = 0ULL;
            continue;
        }
        const uint8_t *seq = flat + off;
        const int32_t nk = L - k + 1;
        for (int t = lane; t < cap; t += 32) buf[t] = MAXV;
        __syncwarp();
        int32_t cnt = 0, npend = 0;
        uint64_t tau = MAXV;
        for (int32_t base = 0; base < nk; base += 32) {
            const int32_t i = base + lane;
            bool take = false;
            uint64_t hv = 0;
            if (i < nk) {
                uint64_t v = 0;
                for (int32_t m = 0; m < k; ++m) v = v * alphabet + (uint64_t)seq[i + m];
                hv = fmix64(v, seed);
                take = (cnt < s) || (hv < tau);
            }
            const unsigned bal = __ballot_sync(0xffffffffu, take);
            if (take) buf[BUF + npend + __popc(bal & ((1u << lane) - 1u))] = hv;
            npend += __popc(bal);
            const bool last = base + 32 >= nk;
            if (npend > 0 && (npend + 32 > BUF || last)) {
                __syncwarp();
                warp_bitonic_sort(buf, cap, lane);
                const int32_t total = cnt + npend;
                cnt = total < s ? total : s;
                for (int t = s + lane; t < cap; t += 32) buf[t] = MAXV;
                __syncwarp();
                tau = (cnt == s) ? buf[s - 1] : MAXV;
                npend = 0;
            }
        }
        __syncwarp();
        for (int t = lane; t < s; t += 32) o[t] = t < cnt ? buf[t] : MAXV;
        __syncwarp();
    }
}

struct SketchCall {
    const uint8_t *flat; int64_t flat_len; const int64_t *offsets; const int32_t *lengths; int64_t N;
    int32_t k, s, aim, alphabet; uint64_t seed; uint64_t *out; int32_t *err; cudaStream_t st;
};

template <int NPL, class V>
static int32_t launch_select_v(const SketchCall &c) {
    constexpr size_t per_warp = (size_t)32 * NPL * sizeof(uint64_t);
    constexpr int warps = select_warps<NPL>();
    const int64_t want = (c.N + warps - 1) / warps, most = (int64_t)sm_count() * 64;
    sketch_select_kernel<NPL, V><<<(unsigned)(want < most ? want : most), warps * 32, per_warp * warps, c.st>>>(
        c.flat, c.flat_len, c.offsets, c.lengths, c.N, c.k, c.s, c.aim, (V)c.alphabet, c.seed, c.out, c.err);
    CK_CUDA(cudaGetLastError());
    return CK_OK;
}

// 32-bit k-mer values where none can wrap: residue codes are bytes, so a value
// is at most 255 * (1 + a + ... + a^(k-1))
template <int NPL>
static int32_t launch_select(const SketchCall &c) {
    double most = 0.0;
    for (int32_t m = 0; m < c.k; ++m) most = most * c.alphabet + 255.0;
    return most < 4294967296.0 ? launch_select_v<NPL, uint32_t>(c) : launch_select_v<NPL, uint64_t>(c);
}

int32_t sketch_launch(const uint8_t *flat, int64_t flat_len, const int64_t *offsets,
                      const int32_t *lengths, int64_t N, int32_t k, int32_t s, int32_t alphabet,
                      uint64_t seed, uint64_t *out, int32_t *d_err, cudaStream_t st) {
    if (k < 1 || k > 32 || s < 1 || s > 4096 || alphabet < 1 || N < 0) {
        set_error(CK_ERR_UNSUPPORTED, "sketch: need 1 <= k <= 32, 1 <= s <= 4096, alphabet >= 1");
        return CK_ERR_UNSUPPORTED;
    }
    if (N == 0) return CK_OK;
    // the threshold form's buffer: C with aim = (s + C) / 2 at least 3.2
    // standard deviations (of about sqrt(aim)) from s and from C, so that about
    // one sequence in a thousand needs a second pass
    for (int32_t C = 64; C <= 2048; C <<= 1) {
        const double mid = 0.5 * ((double)s + C), near = s + 5.5 * sqrt((double)s) + 15.0;
        if (C <= s || 0.5 * (C - s) < 3.2 * sqrt(mid)) continue;
        const SketchCall c{flat, flat_len, offsets, lengths, N, k, s, (int32_t)(mid < near ? mid : near), alphabet,
                           seed, out, d_err, st};
        switch (C) {
            case 64: return launch_select<2>(c);
            case 128: return launch_select<4>(c);
            case 256: return launch_select<8>(c);
            case 512: return launch_select<16>(c);
            case 1024: return launch_select<32>(c);
            default: return launch_select<64>(c);
        }
    }
    int32_t BUF = 32;
    while (BUF < s) BUF <<= 1;
    const size_t per_warp = (size_t)2 * BUF * sizeof(uint64_t);
    int warps_per_block = (int)((48 * 1024) / per_warp);
    if (warps_per_block > 8) warps_per_block = 8;
    size_t smem = per_warp * (warps_per_block > 0 ? warps_per_block : 1);
    if (warps_per_block < 1) {
        warps_per_block = 1;
        CK_CUDA(cudaFuncSetAttribute(sketch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem));
    }
    int64_t want = (N + warps_per_block - 1) / warps_per_block;
    int64_t cap = (int64_t)sm_count() * 16;
    const int blocks = (int)(want < cap ? want : cap);
    sketch_kernel<<<blocks, warps_per_block * 32, smem, st>>>(flat, flat_len, offsets, lengths, N, k, s,
                                                              BUF, (uint64_t)alphabet, seed, out, d_err);
    CK_CUDA(cudaGetLastError());
    return CK_OK;
}

}  // namespace ck
