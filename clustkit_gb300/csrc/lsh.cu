// lsh.cu -- LSH candidate pairs from MinHash sketches on the device.
//
// Same pairs as clustkit/lsh.py:20-178: for every table t a bucket id per
// sequence, h = seed_t; h = h * 0x517CC1B727220A95 + sketch[band index] over
// the table's band, then h = (h ^ h >> 33) * 0xC4CEB9FE1A85EC53, h ^= h >> 33
// (wrapping uint64); sequences are ordered by bucket id, every bucket
// contributes all pairs among its first 1000 members, and the pairs of all
// tables, packed as lo * N + hi (lo < hi), are sorted and de-duplicated.
//
// Tie order inside a bucket: clustkit orders a table with numpy's argsort
// (an unstable introsort); here the radix sort is stable, so a bucket's
// members come in ascending sequence id.  The two agree on every bucket of at
// most 1000 members (all pairs of such a bucket are taken in either order);
// in a larger bucket clustkit keeps whichever 1000 members its sort happens to
// put first, and this keeps the 1000 lowest ids.
//
// Layout: sketches are transposed once to [s][N] so a table's band columns are
// read coalesced.  Tables are processed in batches (as many as fit a few GB of
// scratch; every table at once for moderate N): a batch's bucket ids are made
// in (table, sequence) order and sorted together, stably, so each bucket is one
// run with its members in ascending sequence id, and the run, scan, pair-count
// and emit steps cover the whole batch in one launch each; one radix sort +
// unique de-duplicates all tables, most repeats being left out before it.  The sort moves 12 bytes an item and looks
// at as many bits of the id as tell a table's buckets apart, and not at the
// table (6 passes over 12.8 M items, 0.84 ms; sorted by table and all 64 bits
// as 16-byte keys, it was 9 passes and 1.56).
//
// Tables that read the same columns in the same order have the same buckets,
// whatever their seeds: the seed adds one constant (seed * mul^bands) to every
// sequence's value and the mixing after it is a bijection of 64 bits, so two
// ids agree in one such table exactly when they agree in the other.  Only the
// first of them is worked on: with one band there are at most s distinct
// tables (448 tables over a sketch of 128 leave 128 or fewer).
//
// A batch is hashed, sorted and emitted in one go.  Its pair count is on the
// host before the emission, so one batch sizes the raw buffer exactly; of
// several, the first one's count, in proportion to the tables, and a quarter sizes it,
// and only a call that outgrows that runs its batches a second time, into a
// buffer of the counted size.  100,000 sequences, 448 tables of one band: the
// whole call 24.0 -> 5.5 ms (the old form hashed and sorted all 448
// tables twice).
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <cub/device/device_select.cuh>
#include <thrust/iterator/counting_iterator.h>

#include <cmath>
#include <set>
#include <vector>

#include "ck_common.cuh"

namespace ck {

constexpr uint64_t LSH_MUL = 0x517CC1B727220A95ull;
constexpr uint64_t LSH_FMIX = 0xC4CEB9FE1A85EC53ull;
constexpr int32_t LSH_MAX_BUCKET = 1000;

__global__ void transpose_sketch_kernel(const uint64_t *__restrict__ sk, int64_t n, int32_t s,
                                        uint64_t *__restrict__ skT) {
    // 32 x 32 tiles through shared memory: reads along s, writes along n
    __shared__ uint64_t tile[32][33];
    const int64_t i0 = (int64_t)blockIdx.x * 32;
    const int32_t c0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int64_t i = i0 + r;
        const int32_t c = c0 + threadIdx.x;
        if (i < n && c < s) tile[r][threadIdx.x] = sk[i * s + c];
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int32_t c = c0 + r;
        const int64_t i = i0 + threadIdx.x;
        if (i < n && c < s) skT[(int64_t)c * n + i] = tile[threadIdx.x][r];
    }
}

// bucket ids of tables t0 .. t0 + tb - 1 for every sequence, table-major; the
// value is the item's number, table * n + sequence (tables from the batch's first)
__global__ void lsh_hash_kernel(const uint64_t *__restrict__ skT, int64_t n, const int32_t *__restrict__ band,
                                int32_t nb, const uint64_t *__restrict__ seeds, int32_t t0, int32_t tb,
                                uint64_t *__restrict__ keys, uint32_t *__restrict__ vals) {
    const int64_t total = (int64_t)tb * n;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < total;
         k += (int64_t)gridDim.x * blockDim.x) {
        const int32_t tl = (int32_t)(k / n);
        const int64_t i = k - (int64_t)tl * n;
        const int32_t t = t0 + tl;
        const int32_t *bt = band + (int64_t)t * nb;
        uint64_t h = seeds[t];
        for (int32_t b = 0; b < nb; ++b) h = h * LSH_MUL + skT[(int64_t)bt[b] * n + i];
        h = (h ^ (h >> 33)) * LSH_FMIX;
        h ^= h >> 33;
        keys[k] = h;
        vals[k] = (uint32_t)k;
    }
}

// True where a bucket begins in the sorted items.  Two different buckets of a
// table that share the sorted bits may lie mixed: that sets *mixed.
struct LshBucketStart {
    const uint64_t *keys;
    const uint32_t *vals;
    uint32_t n;
    int32_t unsorted;  // low bits of a key that were not sorted
    int32_t *mixed;
    __device__ bool operator()(int32_t i) const {
        if (i == 0) return true;
        const uint64_t a = keys[i - 1], b = keys[i];
        if (a >> unsorted != b >> unsorted || vals[i - 1] / n != vals[i] / n) return true;
        if (a != b) *mixed = 1;
        return a != b;
    }
};

// the batch's pair total, pair_off[runs], for the host; -1 of mixed buckets
__global__ void lsh_total_kernel(const int32_t *__restrict__ n_runs, const int64_t *__restrict__ pair_off,
                                 const int32_t *__restrict__ mixed, int64_t *__restrict__ total) {
    if (threadIdx.x == 0 && blockIdx.x == 0) *total = *mixed ? -1 : pair_off[*n_runs];
}

// members of bucket r that count (the first 1000), of the R buckets of m items
__device__ __forceinline__ int32_t lsh_members(const int32_t *__restrict__ starts, int64_t r, int32_t R, int64_t m) {
    return min((r + 1 < R ? starts[r + 1] : (int32_t)m) - starts[r], LSH_MAX_BUCKET);
}

// pairs a bucket contributes; zero past the last one
__global__ void lsh_bucket_pairs_kernel(const int32_t *__restrict__ starts, const int32_t *__restrict__ n_runs,
                                        int64_t m, int64_t *__restrict__ npairs) {
    const int32_t R = *n_runs;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r <= m; r += (int64_t)gridDim.x * blockDim.x) {
        if (r >= R) { npairs[r] = 0; continue; }
        const int64_t c = lsh_members(starts, r, R, m);
        npairs[r] = c >= 2 ? c * (c - 1) / 2 : 0;
    }
}

// Emission by bucket: a thread writes the pairs of a bucket of at most 32
// members (pair (x, y), x < y, at offset y(y - 1) / 2 + x of the bucket's
// range), and lists larger buckets for lsh_emit_big_kernel.  The raw pairs
// are sorted and de-duplicated afterwards, so only the set matters.
constexpr int32_t LSH_SMALL_BUCKET = 32;
__global__ void lsh_emit_runs_kernel(const uint32_t *__restrict__ order, const int32_t *__restrict__ run_start,
                                     const int64_t *__restrict__ pair_off, const int32_t *__restrict__ n_runs,
                                     int64_t m, uint32_t n, uint64_t *__restrict__ out, int32_t *__restrict__ big,
                                     int32_t *__restrict__ n_big) {
    const int32_t R = *n_runs;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < R; r += (int64_t)gridDim.x * blockDim.x) {
        const int32_t c = lsh_members(run_start, r, R, m);
        if (c < 2) continue;
        if (c > LSH_SMALL_BUCKET) {
            big[atomicAdd(n_big, 1)] = (int32_t)r;
            continue;
        }
        const int32_t s0 = run_start[r];
        const uint32_t base = order[s0] / n * n;  // the table's first item
        uint64_t *o = out + pair_off[r];
        for (int32_t y = 1; y < c; ++y) {
            const uint32_t b = order[s0 + y] - base;
            for (int32_t x = 0; x < y; ++x) {
                const uint32_t v = order[s0 + x] - base;  // below b: members are in ascending order
                *o++ = (uint64_t)v * n + b;
            }
        }
    }
}

// The listed buckets (more than 32 members, at most 1000 taken): grid (buckets,
// LSH_BIG_PARTS); a bucket's members are dealt out over its blocks' warps, whose
// lanes split each member's pairs with the members before it.  (A warp a
// bucket left the largest, half a million pairs, to one warp: 1.08 ms of the
// call on 100,000 sequences, now 0.15.)
constexpr int LSH_BIG_PARTS = 16;
__global__ void lsh_emit_big_kernel(const uint32_t *__restrict__ order, const int32_t *__restrict__ run_start,
                                    const int64_t *__restrict__ pair_off, const int32_t *__restrict__ n_runs,
                                    int64_t m, const int32_t *__restrict__ big, const int32_t *__restrict__ n_big,
                                    uint32_t n, uint64_t *__restrict__ out) {
    const int32_t lane = threadIdx.x & 31;
    const int32_t nb = *n_big;
    const int32_t warps = (int32_t)(blockDim.x >> 5) * LSH_BIG_PARTS;
    const int32_t warp = (int32_t)(blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5));
    for (int32_t w = blockIdx.x; w < nb; w += gridDim.x) {
        const int32_t r = big[w];
        const int32_t c = lsh_members(run_start, r, *n_runs, m);
        const int32_t s0 = run_start[r];
        const uint32_t base = order[s0] / n * n;
        uint64_t *o = out + pair_off[r];
        for (int32_t y = 1 + warp; y < c; y += warps) {
            const uint32_t b = order[s0 + y] - base;
            uint64_t *row = o + (int64_t)y * (y - 1) / 2;
            for (int32_t x = lane; x < y; x += 32) row[x] = (uint64_t)(order[s0 + x] - base) * n + b;
        }
    }
}

// The same two emissions where several tables find most pairs again and again:
// a pair goes out only if it is not in its set of `seen`, four keys in one
// 32-byte sector (all ones at first, at most 64 MB, which stay in L2), and takes
// a free place there.  A race or a full set lets a pair out twice; none is lost,
// since whoever puts a key into a set also writes it.  A warp queues its pairs
// and takes room for many at a time from *n_out.  Bound by the latency of the
// sets' reads (25 M in 0.35 ms); four rounds ahead help the large buckets (255 ->
// 175 us) and not the small ones, whose warps have few pairs (175 -> 336).
// 100,000 sequences, 124 distinct tables: of 25.5 M raw pairs 6.5 M are written
// (4.6 M are distinct), and sorting them takes 0.32 ms instead of 1.17.
//
// Used from 12 distinct tables and 4 M raw pairs on: the sort of the repeats has
// to cost more than looking every pair up, and how many there are is not known
// before.  Whole call without and with, ms:
//   pairs that most tables find: 22 M raw of 124 tables 5.83 5.14, 32 M of 199
//     4.19 3.18, 11 M of 448 7.48 7.18; families of ten, 20 tables 0.78 0.75, 40
//     1.23 1.00; the same buckets in every table, 72 M of 16 3.50 1.44, 40 M of
//     12 2.01 1.36 (and 27 M of 8 1.43 1.21, 7 M of 2 0.57 0.64)
//   pairs that few find: 300,000 in families, 12 tables 1.00 1.08, 40 2.40 2.47;
//     unlike tables, 71 M of 16 3.61 4.32, 171 M of 40 8.56 10.25 (36 M of 8 1.93
//     2.34)
//   fewer than 4 M: 1.6 M of 8 1.40 1.44, 1.8 M of 30 1.16 1.20
constexpr int32_t LSH_FILTER_TABLES = 12;
constexpr int64_t LSH_FILTER_PAIRS = (int64_t)1 << 22;
constexpr int LSH_AHEAD = 4, LSH_QUEUE = 256, LSH_FILTER_THREADS = 256, LSH_FILTER_PARTS = 32;
struct LshFilter {
    uint64_t *seen;  // sets of four keys, 32 bytes
    uint64_t mask;   // sets - 1
    uint64_t *out;
    unsigned long long *n_out;
    uint64_t *queue;  // the warp's, LSH_QUEUE + 32 LSH_AHEAD
    int32_t held;

    __device__ void flush(int lane) {
        __syncwarp();
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(n_out, (unsigned long long)held);
        at = __shfl_sync(0xffffffffu, at, 0);
        for (int i = lane; i < held; i += 32) out[at + i] = queue[i];
        __syncwarp();
        held = 0;
    }
    // U rounds of keys, all lanes together; ~0 where the lane has none.
    // The sets of all are read before the first is looked at.
    template <int U> __device__ void put(const uint64_t (&key)[U], int lane) {
        uint64_t a[U], b[U], c[U], d[U], *set[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            set[u] = seen + 4 * ((key[u] * 0x9E3779B97F4A7C15ull) >> 32 & mask);
            asm volatile("ld.global.v4.u64 {%0, %1, %2, %3}, [%4];"
                         : "=l"(a[u]), "=l"(b[u]), "=l"(c[u]), "=l"(d[u]) : "l"(set[u]));
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t k = key[u];
            const bool in = k != ~0ull && a[u] != k && b[u] != k && c[u] != k && d[u] != k;
            if (in && d[u] == ~0ull) set[u][a[u] == ~0ull ? 0 : b[u] == ~0ull ? 1 : c[u] == ~0ull ? 2 : 3] = k;
            const uint32_t m = __ballot_sync(0xffffffffu, in);
            if (in) queue[held + __popc(m & ((1u << lane) - 1))] = k;
            held += __popc(m);
        }
        if (held >= LSH_QUEUE) flush(lane);
    }
};

__global__ void __launch_bounds__(LSH_FILTER_THREADS)
    lsh_filter_runs_kernel(const uint32_t *__restrict__ order, const int32_t *__restrict__ run_start,
                           const int32_t *__restrict__ n_runs, int64_t m, uint32_t n, LshFilter f,
                           int32_t *__restrict__ big, int32_t *__restrict__ n_big) {
    __shared__ uint64_t queues[LSH_FILTER_THREADS / 32][LSH_QUEUE + 32 * LSH_AHEAD];
    const int lane = threadIdx.x & 31;
    f.queue = queues[threadIdx.x >> 5];
    f.held = 0;
    const int32_t R = *n_runs;
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; r0 < R; r0 += step) {
        // a lane a bucket, then the warp's pairs laid end to end
        const int64_t r = r0 + lane;
        int32_t c = r < R ? lsh_members(run_start, r, R, m) : 0;
        if (c > LSH_SMALL_BUCKET) {
            big[atomicAdd(n_big, 1)] = (int32_t)r;
            c = 0;
        }
        const int32_t s0 = c >= 2 ? run_start[r] : 0;
        const uint32_t base = c >= 2 ? order[s0] / n * n : 0;
        int32_t end = c * (c - 1) / 2;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t v = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += v;
        }
        const int32_t total = __shfl_sync(0xffffffffu, end, 31);
        for (int32_t i0 = 0; i0 < total; i0 += 32) {
            const int32_t i = min(i0 + lane, total - 1);
            int owner = 0;  // lanes whose pairs end at i or before
#pragma unroll
            for (int o = 16; o; o >>= 1)
                if (__shfl_sync(0xffffffffu, end, owner + o - 1) <= i) owner += o;
            const int32_t before = __shfl_sync(0xffffffffu, end, max(owner - 1, 0));
            const int32_t p = i - (owner ? before : 0);  // pair y(y - 1)/2 + x of its bucket
            int32_t y = (int32_t)((sqrtf((float)(8 * p + 1)) + 1.0f) * 0.5f);
            if (y * (y - 1) / 2 > p) --y;
            if (y * (y + 1) / 2 <= p) ++y;
            const int32_t from = __shfl_sync(0xffffffffu, s0, owner);
            const uint32_t b = __shfl_sync(0xffffffffu, base, owner);
            const uint32_t hi = order[from + y] - b, lo = order[from + p - y * (y - 1) / 2] - b;
            const uint64_t key[1] = {i0 + lane < total ? (uint64_t)lo * n + hi : ~0ull};
            f.put(key, lane);
        }
    }
    f.flush(lane);
}

__global__ void __launch_bounds__(LSH_FILTER_THREADS)
    lsh_filter_big_kernel(const uint32_t *__restrict__ order, const int32_t *__restrict__ run_start,
                          const int32_t *__restrict__ n_runs, int64_t m, const int32_t *__restrict__ big,
                          const int32_t *__restrict__ n_big, uint32_t n, LshFilter f) {
    __shared__ uint64_t queues[LSH_FILTER_THREADS / 32][LSH_QUEUE + 32 * LSH_AHEAD];
    const int lane = threadIdx.x & 31;
    f.queue = queues[threadIdx.x >> 5];
    f.held = 0;
    const int32_t nb = *n_big;
    const int32_t warps = (int32_t)(blockDim.x >> 5) * LSH_FILTER_PARTS;
    const int32_t warp = (int32_t)(blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5));
    for (int32_t w = blockIdx.x; w < nb; w += gridDim.x) {
        const int32_t r = big[w];
        const int32_t c = lsh_members(run_start, r, *n_runs, m);
        const int32_t s0 = run_start[r];
        const uint32_t base = order[s0] / n * n;
        for (int32_t y = 1 + warp; y < c; y += warps) {
            const uint32_t b = order[s0 + y] - base;
            for (int32_t x0 = lane; x0 - lane < y; x0 += 32 * LSH_AHEAD) {
                uint64_t key[LSH_AHEAD];
#pragma unroll
                for (int u = 0; u < LSH_AHEAD; ++u) {
                    const int32_t x = x0 + 32 * u;
                    key[u] = x < y ? (uint64_t)(order[s0 + x] - base) * n + b : ~0ull;
                }
                f.put(key, lane);
            }
        }
    }
    f.flush(lane);
}

__global__ void lsh_unpack_kernel(const uint64_t *__restrict__ keys, int64_t m, int64_t n,
                                  int32_t *__restrict__ pairs) {
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x) {
        pairs[2 * k] = (int32_t)(keys[k] / (uint64_t)n);
        pairs[2 * k + 1] = (int32_t)(keys[k] % (uint64_t)n);
    }
}

static int grid_of(int64_t work, int threads) {
    int64_t b = (work + threads - 1) / threads;
    const int64_t cap = (int64_t)sm_count() * 32;
    if (b > cap) b = cap;
    return (int)(b < 1 ? 1 : b);
}

struct LshArgs {
    const uint64_t *sk; int64_t n; int32_t s; int32_t tables, bands;
    const int32_t *band_idx_host; const uint64_t *seeds_host;
    int32_t *out_pairs; int64_t capacity; int64_t *out_count; cudaStream_t st;
};

static int32_t lsh_impl(void *pv) {
    LshArgs &a = *(LshArgs *)pv;
    int32_t status = CK_OK;
    const int64_t n = a.n;
    cudaStream_t st = a.st;
    *a.out_count = 0;
    if (n < 2 || a.tables == 0) return CK_OK;
    // the distinct tables (same columns in the same order: same buckets)
    std::vector<int32_t> band_h;
    std::vector<uint64_t> seed_h;
    {
        std::set<std::vector<int32_t>> seen;
        for (int32_t t = 0; t < a.tables; ++t) {
            const int32_t *row = a.band_idx_host + (size_t)t * a.bands;
            if (!seen.insert(std::vector<int32_t>(row, row + a.bands)).second) continue;
            band_h.insert(band_h.end(), row, row + a.bands);
            seed_h.push_back(a.seeds_host[t]);
        }
    }
    const int32_t T = (int32_t)seed_h.size();
    // tables per batch: about 4 GB of keys, values and run data (40 B an item),
    // and fewer than 2^31 items (runs are counted in int)
    int64_t tb64 = ((int64_t)4 << 30) / (40 * n);
    if (tb64 * n > ((int64_t)1 << 30)) tb64 = ((int64_t)1 << 30) / n;
    if (tb64 < 1) tb64 = 1;
    if (tb64 > T) tb64 = T;
    const int32_t TB = (int32_t)tb64;
    const int64_t items = (int64_t)TB * n;
    // Sorted bits of a bucket id, from the top: as many (whole digits) as leave
    // two buckets of a table less than one chance in 64 to share them, in all
    // the batch's n^2 TB / 2 comparisons.  A batch where some do is sorted
    // again by all 64.
    int sorted = 8;
    while (sorted < 64 && std::ldexp((double)n * (double)n * TB, 5 - sorted) > 1.0) sorted += 8;
    // band indices and seeds on the device
    int32_t *d_band = (int32_t *)scratch(SLOT_SEARCH_TMP0, band_h.size() * 4 + (size_t)T * 8 + 16, &status);
    uint64_t *skT = (uint64_t *)scratch(SLOT_SEARCH_TMP1, (size_t)n * a.s * 8, &status);
    uint64_t *k0 = (uint64_t *)scratch(SLOT_SEARCH_TMP2, (size_t)items * 8 * 2, &status);
    uint32_t *v0 = (uint32_t *)scratch(SLOT_SEARCH_TMP3, (size_t)items * 4 * 2, &status);
    // run data: pair offsets (items + 1), starts, then the list of buckets of
    // more than 32 members (at most items / 33 of them)
    const int64_t n_big_max = items / (LSH_SMALL_BUCKET + 1) + 1;
    char *rle = (char *)scratch(SLOT_SEARCH_TMP4, (size_t)(items + 1) * 8 + (size_t)(items + n_big_max) * 4, &status);
    int32_t *n_runs = (int32_t *)scratch(SLOT_MAXLEN, 64, &status);
    if (!d_band || !skT || !k0 || !v0 || !rle || !n_runs) return status;
    int32_t *n_big = n_runs + 8, *d_mixed = n_runs + 9;
    uint64_t *d_seeds = (uint64_t *)(((uintptr_t)(d_band + band_h.size()) + 15) & ~(uintptr_t)15);
    uint64_t *k1 = k0 + items;
    uint32_t *v1 = v0 + items;
    int64_t *pair_off = (int64_t *)rle;
    int32_t *starts = (int32_t *)(pair_off + items + 1);
    int32_t *big = starts + items;
    int64_t *d_total = (int64_t *)(n_runs + 4);
    CK_CUDA(cudaMemcpyAsync(d_band, band_h.data(), band_h.size() * 4, cudaMemcpyHostToDevice, st));
    CK_CUDA(cudaMemcpyAsync(d_seeds, seed_h.data(), (size_t)T * 8, cudaMemcpyHostToDevice, st));
    {
        dim3 grid((unsigned)((n + 31) / 32), (unsigned)((a.s + 31) / 32));
        transpose_sketch_kernel<<<grid, dim3(32, 8), 0, st>>>(a.sk, n, a.s, skT);
        CK_CUDA(cudaGetLastError());
    }
    // temp storage sizes (the largest of the calls below, at a full batch)
    const thrust::counting_iterator<int32_t> numbers(0);
    size_t t_sort = 0, t_select = 0, t_scan = 0;
    {
        cub::DoubleBuffer<uint64_t> dk(k0, k1);
        cub::DoubleBuffer<uint32_t> dv(v0, v1);
        CK_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, t_sort, dk, dv, items, 0, 64, st));
        CK_CUDA(cub::DeviceSelect::If(nullptr, t_select, numbers, starts, n_runs, (int)items,
                                      LshBucketStart{k0, v0, (uint32_t)n, 0, d_mixed}, st));
        CK_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, t_scan, pair_off, pair_off, (int)items + 1, st));
    }
    const size_t t_max = std::max(t_sort, std::max(t_select, t_scan));
    void *tmp = scratch(SLOT_SORT_TEMP, t_max, &status);
    if (!tmp) return status;

    // one batch: bucket ids, stable sort, runs, pair offsets; *total its pair
    // count.  Items are made in (table, sequence) order, so equal sorted bits
    // keep a table's items together and their sequences ascending.
    auto batch = [&](int32_t t0, int32_t tb, cub::DoubleBuffer<uint32_t> &dv, int64_t *total) -> int32_t {
        const int64_t m = (int64_t)tb * n;
        for (int by = sorted;; by = 64) {
            cub::DoubleBuffer<uint64_t> dk(k0, k1);
            dv = cub::DoubleBuffer<uint32_t>(v0, v1);
            lsh_hash_kernel<<<grid_of(m, 256), 256, 0, st>>>(skT, n, d_band, a.bands, d_seeds, t0, tb, dk.Current(),
                                                             dv.Current());
            CK_CUDA(cudaGetLastError());
            CK_CUDA(cudaMemsetAsync(d_mixed, 0, 4, st));
            size_t tbytes = t_max;
            CK_CUDA(cub::DeviceRadixSort::SortPairs(tmp, tbytes, dk, dv, m, 64 - by, 64, st));
            tbytes = t_max;
            CK_CUDA(cub::DeviceSelect::If(tmp, tbytes, numbers, starts, n_runs, (int)m,
                                          LshBucketStart{dk.Current(), dv.Current(), (uint32_t)n, 64 - by, d_mixed},
                                          st));
            lsh_bucket_pairs_kernel<<<grid_of(m + 1, 256), 256, 0, st>>>(starts, n_runs, m, pair_off);
            CK_CUDA(cudaGetLastError());
            tbytes = t_max;
            CK_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tbytes, pair_off, pair_off, (int)m + 1, st));
            // pair_off[R] (R = runs) is the batch's total; runs <= m, entries past R are 0
            lsh_total_kernel<<<1, 32, 0, st>>>(n_runs, pair_off, d_mixed, d_total);
            CK_CUDA(cudaGetLastError());
            CK_CUDA(cudaMemcpyAsync(total, d_total, 8, cudaMemcpyDeviceToHost, st));
            CK_CUDA(cudaStreamSynchronize(st));
            if (*total >= 0) return CK_OK;
        }
    };

    uint64_t *rk = nullptr, *seen = nullptr;  // raw pairs; keys seen, where repeats are left out
    uint64_t places = 0;
    unsigned long long *d_kept = (unsigned long long *)(n_runs + 10);
    const auto forget = [&]() -> int32_t {
        if (!seen) return CK_OK;
        CK_CUDA(cudaMemsetAsync(seen, 0xff, (size_t)places * 8, st));
        CK_CUDA(cudaMemsetAsync(d_kept, 0, 8, st));
        return CK_OK;
    };
    // emission of the batch just prepared, at `out` (or behind what is kept)
    auto emit = [&](int32_t tb, cub::DoubleBuffer<uint32_t> &dv, uint64_t *out) -> int32_t {
        const int64_t m = (int64_t)tb * n;
        CK_CUDA(cudaMemsetAsync(n_big, 0, 4, st));
        if (seen) {
            const LshFilter f{seen, places / 4 - 1, rk, d_kept, nullptr, 0};
            lsh_filter_runs_kernel<<<8 * sm_count(), LSH_FILTER_THREADS, 0, st>>>(dv.Current(), starts, n_runs, m,
                                                                                  (uint32_t)n, f, big, n_big);
            CK_CUDA(cudaGetLastError());
            lsh_filter_big_kernel<<<dim3((unsigned)sm_count(), LSH_FILTER_PARTS), LSH_FILTER_THREADS, 0, st>>>(
                dv.Current(), starts, n_runs, m, big, n_big, (uint32_t)n, f);
            CK_CUDA(cudaGetLastError());
            return CK_OK;
        }
        lsh_emit_runs_kernel<<<grid_of(m, 256), 256, 0, st>>>(dv.Current(), starts, pair_off, n_runs, m, (uint32_t)n,
                                                              out, big, n_big);
        CK_CUDA(cudaGetLastError());
        lsh_emit_big_kernel<<<dim3((unsigned)sm_count(), LSH_BIG_PARTS), 128, 0, st>>>(
            dv.Current(), starts, pair_off, n_runs, m, big, n_big, (uint32_t)n, out);
        CK_CUDA(cudaGetLastError());
        return CK_OK;
    };

    // scratch of the sort and unique that de-duplicate m raw pairs (packed keys
    // of enough bits for n * n)
    int bits = 1;
    while (bits < 64 && ((uint64_t)1 << bits) <= (uint64_t)n * (uint64_t)n) ++bits;
    auto dedup_bytes = [&](int64_t m, size_t *bytes) -> int32_t {
        size_t ts = 0, tu = 0;
        uint64_t *none = nullptr;
        cub::DoubleBuffer<uint64_t> both(none, none);
        CK_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, ts, both, m, 0, bits, st));
        CK_CUDA(cub::DeviceSelect::Unique(nullptr, tu, none, none, (int64_t *)nullptr, m, st));
        *bytes = std::max(ts, tu);
        return CK_OK;
    };

    // room for `room` raw pairs, twice over for the de-duplicating sort; a
    // guess that does not fit the device is no error (the counted size may)
    const int32_t n_batches = (T + TB - 1) / TB;
    int64_t room = 0, raw = 0;
    bool fits = true;
    for (int32_t b = 0; b < n_batches; ++b) {
        const int32_t t0 = b * TB, tb = T - t0 < TB ? T - t0 : TB;
        cub::DoubleBuffer<uint32_t> dv(v0, v1);
        int64_t tot = 0;
        CK_TRY(batch(t0, tb, dv, &tot));
        if (b == 0) {
            room = n_batches == 1 ? tot : (int64_t)((double)(tot + tot / 4) * T / TB) + 1;
            if (room > 0) {
                // the de-duplicating sort's own scratch first: the guess must leave it that
                size_t t_dedup = 0;
                CK_TRY(dedup_bytes(room, &t_dedup));
                tmp = scratch(SLOT_SORT_TEMP, std::max(t_max, t_dedup), &status);
                if (tmp) rk = (uint64_t *)scratch(SLOT_FALLBACK, (size_t)room * 8 * 2, &status);
            }
            if (!rk && room > 0) {
                if (n_batches == 1) return status;
                cudaGetLastError();  // the failed allocation: later launches are checked for their own errors
                reset_thread_status();
                status = CK_OK;
                room = 0;
                tmp = scratch(SLOT_SORT_TEMP, t_max, &status);
                if (!tmp) return status;
            }
            if (T >= LSH_FILTER_TABLES && room >= LSH_FILTER_PAIRS) {
                places = (uint64_t)1 << 16;
                while (places < ((uint64_t)1 << 23) && places < (uint64_t)room / 4) places *= 2;
                seen = (uint64_t *)scratch(SLOT_SORT_KEYS_ALT, (size_t)places * 8, &status);
                if (!seen) {  // done without
                    cudaGetLastError();
                    reset_thread_status();
                    status = CK_OK;
                }
                CK_TRY(forget());
            }
        }
        if (tot > 0 && raw + tot <= room && fits) CK_TRY(emit(tb, dv, rk + raw));
        else if (tot > 0) fits = false;
        raw += tot;
    }
    if (raw == 0) return CK_OK;
    if (!fits) {
        rk = (uint64_t *)scratch(SLOT_FALLBACK, (size_t)raw * 8 * 2, &status);
        if (!rk) return status;
        int64_t at = 0;
        CK_TRY(forget());
        for (int32_t b = 0; b < n_batches; ++b) {
            const int32_t t0 = b * TB, tb = T - t0 < TB ? T - t0 : TB;
            cub::DoubleBuffer<uint32_t> dv(v0, v1);
            int64_t tot = 0;
            CK_TRY(batch(t0, tb, dv, &tot));
            if (tot > 0) CK_TRY(emit(tb, dv, rk + at));
            at += tot;
        }
    }
    if (seen) {
        CK_CUDA(cudaMemcpyAsync(&raw, d_kept, 8, cudaMemcpyDeviceToHost, st));
        CK_CUDA(cudaStreamSynchronize(st));
    }
    // de-duplicate: sort, unique
    cub::DoubleBuffer<uint64_t> rb(rk, rk + raw);
    int64_t *n_uniq = (int64_t *)(n_runs + 2);
    size_t t_dedup = 0;
    CK_TRY(dedup_bytes(raw, &t_dedup));
    tmp = scratch(SLOT_SORT_TEMP, t_dedup, &status);
    if (!tmp) return status;
    size_t tbytes = t_dedup;
    CK_CUDA(cub::DeviceRadixSort::SortKeys(tmp, tbytes, rb, raw, 0, bits, st));
    tbytes = t_dedup;
    CK_CUDA(cub::DeviceSelect::Unique(tmp, tbytes, rb.Current(), rb.Alternate(), n_uniq, raw, st));
    int64_t m = 0;
    CK_CUDA(cudaMemcpyAsync(&m, n_uniq, 8, cudaMemcpyDeviceToHost, st));
    CK_CUDA(cudaStreamSynchronize(st));
    *a.out_count = m;
    if (m > a.capacity) {
        set_error(CK_ERR_OUT_OF_MEMORY, "LSH: more candidate pairs than the output capacity (count returned)");
        return CK_ERR_OUT_OF_MEMORY;
    }
    lsh_unpack_kernel<<<grid_of(m, 256), 256, 0, st>>>(rb.Alternate(), m, n, a.out_pairs);
    CK_CUDA(cudaGetLastError());
    CK_CUDA(cudaStreamSynchronize(st));
    return CK_OK;
}

}  // namespace ck

using namespace ck;

extern "C" int32_t ck_lsh_candidates_device(int32_t ctx, const uint64_t *d_sketches, int64_t n, int32_t s,
                                            int32_t num_tables, int32_t num_bands,
                                            const int32_t *band_idx_host, const uint64_t *seeds_host,
                                            int32_t *d_out_pairs, int64_t capacity, int64_t *out_count,
                                            void *stream) {
    std::lock_guard<std::mutex> lock(library_mutex());
    reset_thread_status();
    if (!out_count || n < 0 || n >= ((int64_t)1 << 31) || s < 1 || num_tables < 0 || num_bands < 1 ||
        num_bands > s || capacity < 0 || (n > 0 && !d_sketches) || (num_tables > 0 && (!band_idx_host || !seeds_host)) ||
        (capacity > 0 && !d_out_pairs)) {
        set_error(CK_ERR_INVALID_ARGUMENT, "LSH: bad arguments");
        return CK_ERR_INVALID_ARGUMENT;
    }
    for (int64_t i = 0; i < (int64_t)num_tables * num_bands; ++i)
        if (band_idx_host[i] < 0 || band_idx_host[i] >= s) {
            set_error(CK_ERR_OUT_OF_RANGE, "LSH: band index outside the sketch");
            return CK_ERR_OUT_OF_RANGE;
        }
    LshArgs a{d_sketches, n, s, num_tables, num_bands, band_idx_host, seeds_host, d_out_pairs, capacity,
              out_count, (cudaStream_t)stream};
    return run_in_context(ctx, lsh_impl, &a);
}
