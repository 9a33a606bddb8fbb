// search.cu -- k-mer inverted index and Phase-A k-mer scoring for search.
//
// Index (clustkit/kmer_index.py:77-166): CSR over all alpha^k k-mer values;
// kmer_freqs[v] = occurrences of v, kmer_offsets = exclusive prefix sum,
// kmer_entries = (sequence << 32 | position) grouped by k-mer and, inside a
// k-mer, in (sequence, position) order.  k-mers holding a code >= alpha are
// not indexed.  Built on the GPU: every position emits (k-mer, entry), a
// stable radix sort by k-mer keeps the (sequence, position) order.
//
// Phase A (clustkit/kmer_index.py:470-534, :858-902): for each query k-mer
// (valid, frequency <= freq_thresh) every posting adds one hit to its target;
// counts saturate at 32767 as clustkit's int16 counters do; targets with
// count >= min_total_hits survive; at most top_k survive per query, chosen by
// count (ties: lower target id first), returned in target-id order.
#include <cub/block/block_scan.cuh>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <cub/device/device_segmented_sort.cuh>
#include <cooperative_groups.h>

#include <algorithm>
#include <vector>

#include "ck_common.cuh"

namespace ck {

// ----------------------------------------------------------------- index build
__global__ void kmer_pos_count_kernel(const int32_t *lengths, int64_t n, int32_t k, int64_t *cnt) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t L = lengths[i];
        cnt[i] = L >= k ? (int64_t)(L - k + 1) : 0;
    }
}

// Occurrences in (sequence, position) order, a warp a sequence; the k-mers'
// frequencies as well where `freqs`.  K > 0: k, at compile time.  39 M: 145 us
// (470 MB written; 275 with the atomics and k a variable).
template <int K>
__global__ void kmer_emit_kernel(const uint8_t *__restrict__ flat, int64_t flat_len,
                                 const int64_t *__restrict__ offsets,
                                 const int32_t *__restrict__ lengths, int64_t n, int32_t any_k,
                                 int32_t alpha, const int64_t *__restrict__ pos_base,
                                 uint32_t *__restrict__ keys, int64_t *__restrict__ vals,
                                 int32_t *__restrict__ freqs, uint32_t sentinel, int32_t *err) {
    const int32_t k = K ? K : any_k;
    const int lane = threadIdx.x & 31;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < n; q += warps) {
        const int32_t L = lengths[q];
        const int64_t o = offsets[q];
        if (L < k) continue;
        const int64_t base = pos_base[q];
        const bool bad = o < 0 || o + L > flat_len;
        if (bad && lane == 0) atomicOr(err, ERRBIT_SEQ_EXTENT);
        const uint8_t *s = bad ? flat : flat + o;
#pragma unroll 2
        for (int32_t p = lane; p <= L - k; p += 32) {
            uint32_t v = 0;
            bool ok = !bad;
            if (!bad)
#pragma unroll
                for (int32_t m = 0; m < k; ++m) {
                    const uint32_t c = __ldg(s + p + m);
                    ok &= c < (uint32_t)alpha;
                    v = v * (uint32_t)alpha + c;
                }
            keys[base + p] = ok ? v : sentinel;
            vals[base + p] = ((int64_t)q << 32) | (int64_t)p;
            if (freqs && ok) atomicAdd(&freqs[v], 1);
        }
    }
}

// offsets[u] = the first of the P sorted keys at or above u, u <= nk (the
// sentinel nk sorts last): a key sets those from the key before it (exclusive)
// to its own.  A lane takes four keys (64 us for 39 M; one key a lane 101) and a
// long gap is written by the whole warp.  The last lane of all, behind the
// keys, ends the offsets.
__global__ void kmer_bounds_kernel(const uint32_t *__restrict__ keys, uint32_t P, uint32_t nk,
                                   int64_t *__restrict__ offsets) {
    const int lane = threadIdx.x & 31;
    const uint32_t groups = (P >> 2) + 1, step = gridDim.x * blockDim.x;
    for (uint32_t g0 = blockIdx.x * blockDim.x + threadIdx.x - lane; g0 < groups; g0 += step) {
        const uint32_t i = 4 * (g0 + lane);
        uint32_t key[4];
        if (i + 4 <= P) {
            const uint4 x = *(const uint4 *)(keys + i);
            key[0] = x.x, key[1] = x.y, key[2] = x.z, key[3] = x.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) key[j] = i + j < P ? keys[i + j] : nk;
        }
        uint32_t before = __shfl_up_sync(0xffffffffu, key[3], 1);
        if (lane == 0 && i > 0) before = keys[i - 1];
        uint32_t from = i > 0 ? before + 1 : 0;
        uint32_t left = key[3] + 1 > from && i <= P ? key[3] + 1 - from : 0;  // offsets the lane's keys set
        if (left > 0 && left < 64) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                for (; from <= key[j] && from <= nk; ++from) offsets[from] = i + j < P ? i + j : P;
            left = 0;
        }
        for (uint32_t wide = __ballot_sync(0xffffffffu, left > 0); wide; wide &= wide - 1) {
            const int x = __ffs(wide) - 1;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t f = __shfl_sync(0xffffffffu, from, x), t = min(__shfl_sync(0xffffffffu, key[j], x), nk);
                const uint32_t at = min(4 * (g0 + x) + j, P);
                for (uint32_t u = f + lane; u <= t; u += 32) offsets[u] = at;
                if (lane == x && f <= t) from = t + 1;
            }
        }
    }
}

__global__ void kmer_freqs_kernel(const int64_t *__restrict__ offsets, int64_t nk, int32_t *__restrict__ freqs) {
    for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < nk; u += (int64_t)gridDim.x * blockDim.x)
        freqs[u] = (int32_t)(offsets[u + 1] - offsets[u]);
}

__global__ void widen_kernel(const int32_t *in, int64_t n, int64_t *out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= n;
         i += (int64_t)gridDim.x * blockDim.x)
        out[i] = i < n ? (int64_t)in[i] : 0;
}

static int grid_for(int64_t n, int threads, int cap_per_sm = 16) {
    int64_t b = (n + threads - 1) / threads;
    int64_t cap = (int64_t)sm_count() * cap_per_sm;
    if (b > cap) b = cap;
    return (int)(b < 1 ? 1 : b);
}

struct IndexBuildArgs {
    const uint8_t *flat; int64_t flat_len; const int64_t *offsets; const int32_t *lengths; int64_t n;
    int32_t k, alpha; int64_t *kmer_offsets; int64_t *kmer_entries; int64_t capacity;
    int32_t *kmer_freqs; int64_t *out_total; cudaStream_t st;
};

static int32_t index_build_impl(void *pv) {
    IndexBuildArgs &a = *(IndexBuildArgs *)pv;
    int32_t status = CK_OK;
    int64_t nk = 1;
    for (int32_t i = 0; i < a.k; ++i) nk *= a.alpha;
    int32_t *err = device_error_word(&status);
    if (!err) return status;
    const size_t n1 = (size_t)(a.n > 0 ? a.n : 1);
    int64_t *cnt = (int64_t *)scratch(SLOT_SEARCH_TMP0, (n1 + 1) * 8, &status);
    if (!cnt) return status;
    kmer_pos_count_kernel<<<grid_for(a.n, 256), 256, 0, a.st>>>(a.lengths, a.n, a.k, cnt);
    CK_CUDA(cudaGetLastError());
    CK_CUDA(cudaMemsetAsync(cnt + a.n, 0, 8, a.st));
    size_t tb = 0;
    CK_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, cnt, cnt, a.n + 1, a.st));
    void *tmp = scratch(SLOT_SEARCH_TMP4, tb, &status);
    if (!tmp) return status;
    CK_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, cnt, cnt, a.n + 1, a.st));
    int64_t P = 0;
    CK_CUDA(cudaMemcpyAsync(&P, cnt + a.n, 8, cudaMemcpyDeviceToHost, a.st));
    CK_CUDA(cudaStreamSynchronize(a.st));
    if (P >= ((int64_t)1 << 31)) {
        set_error(CK_ERR_INVALID_ARGUMENT, "kmer index: more than 2^31-1 k-mer positions in one build");
        return CK_ERR_INVALID_ARGUMENT;
    }
    if (P > a.capacity) {
        set_error(CK_ERR_INVALID_ARGUMENT, "kmer index: entries capacity below the number of k-mer positions");
        return CK_ERR_INVALID_ARGUMENT;
    }
    // Offsets and frequencies: read off the sorted keys, or counted by atomics as
    // the occurrences are made and scanned.  39 M occurrences of 3.2 M 5-mers:
    // 72 us for reading them off; the atomics, the scan and the widening took 143.
    // Few k-mers meet in the atomics (20 M occurrences of 8,000 3-mers: whole
    // build 1.33 -> 0.82 ms).  An index with an eighth as many occurrences as
    // k-mers costs the same either way (0.19 ms), a sparser one is mostly gaps.
    const bool dense = P > 0 && nk <= 8 * P;
    if (!dense) CK_CUDA(cudaMemsetAsync(a.kmer_freqs, 0, (size_t)nk * 4, a.st));
    const size_t P1 = (size_t)(P > 0 ? P : 1);
    uint32_t *k0 = (uint32_t *)scratch(SLOT_SEARCH_TMP1, P1 * 4, &status);
    uint32_t *k1 = (uint32_t *)scratch(SLOT_SEARCH_TMP2, P1 * 4, &status);
    int64_t *v0 = (int64_t *)scratch(SLOT_SEARCH_TMP3, P1 * 8, &status);
    if (!k0 || !k1 || !v0) return status;
    const uint32_t sentinel = (uint32_t)nk;
    const auto emit = a.k == 5   ? kmer_emit_kernel<5>
                      : a.k == 4 ? kmer_emit_kernel<4>
                      : a.k == 3 ? kmer_emit_kernel<3>
                                 : kmer_emit_kernel<0>;
    if (a.n > 0)
        emit<<<grid_for(a.n * 32, 256), 256, 0, a.st>>>(a.flat, a.flat_len, a.offsets, a.lengths, a.n, a.k, a.alpha,
                                                        cnt, k0, v0, dense ? nullptr : a.kmer_freqs, sentinel, err);
    CK_CUDA(cudaGetLastError());
    int bits = 1;
    while (((int64_t)1 << bits) <= (int64_t)sentinel) ++bits;
    if (P > 0) {
        // the caller's entries buffer is the sort's second value buffer
        cub::DoubleBuffer<uint32_t> dk(k0, k1);
        cub::DoubleBuffer<int64_t> dv(v0, a.kmer_entries);
        size_t sb = 0;
        CK_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, sb, dk, dv, (int)P, 0, bits, a.st));
        void *stmp = scratch(SLOT_SEARCH_TMP4, sb, &status);
        if (!stmp) return status;
        CK_CUDA(cub::DeviceRadixSort::SortPairs(stmp, sb, dk, dv, (int)P, 0, bits, a.st));
        if (dv.Current() != a.kmer_entries)
            CK_CUDA(cudaMemcpyAsync(a.kmer_entries, dv.Current(), (size_t)P * 8, cudaMemcpyDeviceToDevice, a.st));
        if (dense) {
            kmer_bounds_kernel<<<grid_for(P / 4 + 1, 256, 32), 256, 0, a.st>>>(dk.Current(), (uint32_t)P, (uint32_t)nk,
                                                                                a.kmer_offsets);
            CK_CUDA(cudaGetLastError());
            kmer_freqs_kernel<<<grid_for(nk, 256), 256, 0, a.st>>>(a.kmer_offsets, nk, a.kmer_freqs);
            CK_CUDA(cudaGetLastError());
        }
    }
    if (!dense) {
        widen_kernel<<<grid_for(nk + 1, 256), 256, 0, a.st>>>(a.kmer_freqs, nk, a.kmer_offsets);
        CK_CUDA(cudaGetLastError());
        size_t tb2 = 0;
        CK_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb2, a.kmer_offsets, a.kmer_offsets, nk + 1, a.st));
        void *tmp2 = scratch(SLOT_SEARCH_TMP4, tb2, &status);
        if (!tmp2) return status;
        CK_CUDA(cub::DeviceScan::ExclusiveSum(tmp2, tb2, a.kmer_offsets, a.kmer_offsets, nk + 1, a.st));
    }
    int64_t total = 0;
    CK_CUDA(cudaMemcpyAsync(&total, a.kmer_offsets + nk, 8, cudaMemcpyDeviceToHost, a.st));
    int32_t h = 0;
    CK_CUDA(cudaMemcpyAsync(&h, err, 4, cudaMemcpyDeviceToHost, a.st));
    CK_CUDA(cudaMemsetAsync(err, 0, 4, a.st));
    CK_CUDA(cudaStreamSynchronize(a.st));
    if (h) {
        set_error(CK_ERR_OUT_OF_RANGE, "kmer index: sequence extent outside the flat buffer");
        return CK_ERR_OUT_OF_RANGE;
    }
    *a.out_total = total;
    return CK_OK;
}

// ----------------------------------------------------------------- phase A
// Targets that reach min_hits are listed as they cross it; up to CAND_CAP per
// query the select works on that list, beyond it on the full count row.
constexpr int32_t CAND_CAP = 4096;

// Grid (blocks, nq): the warps of a query's blocks take its k-mer positions
// in turn; a warp walks one posting list, lanes adding hits in parallel.
// Target of posting entry h: from the compact int32 copy when there is one
// (clustkit's kmer_entries_compact, clustkit/database.py:128-135: half the
// bytes per posting for the Phase-A walks), else the full entry's high half.
__device__ __forceinline__ int32_t entry_target(const int64_t *__restrict__ entries,
                                                const int32_t *__restrict__ targets, int64_t h) {
    return targets ? __ldg(targets + h) : (int32_t)(entries[h] >> 32);
}

// Dense pair list of a search batch for the SW engine: pair q * K + c is
// (seq0 + q, targets[q * K + c]) for the query's first n[q] candidates and
// (empty, empty) after them (an empty sequence aligns to nothing).
__global__ void search_pairs_kernel(int32_t nq, int32_t K, int32_t seq0, int32_t empty_idx,
                                    const int32_t *__restrict__ n, const int32_t *__restrict__ targets,
                                    int2 *__restrict__ pairs) {
    const int64_t M = (int64_t)nq * K;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < M; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t q = (int32_t)(i / K), c = (int32_t)(i - (int64_t)q * K);
        pairs[i] = c < __ldg(n + q) ? make_int2(seq0 + q, __ldg(targets + i)) : make_int2(empty_idx, empty_idx);
    }
}

__global__ void compact_targets_kernel(const int64_t *__restrict__ entries, int64_t n,
                                       int32_t *__restrict__ targets) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        targets[i] = (int32_t)(entries[i] >> 32);
}

__global__ void phase_a_count_kernel(const uint8_t *__restrict__ qflat, int64_t qflat_len,
                                     const int64_t *__restrict__ qoff,
                                     const int32_t *__restrict__ qlen, int32_t k, int32_t alpha,
                                     const int64_t *__restrict__ kmer_offsets,
                                     const int64_t *__restrict__ kmer_entries,
                                     const int32_t *__restrict__ kmer_targets,
                                     const int32_t *__restrict__ kmer_freqs, int32_t freq_thresh,
                                     int32_t num_db, int32_t *__restrict__ counts, int32_t min_hits,
                                     int32_t *__restrict__ cand, int32_t *__restrict__ n_cand,
                                     int32_t *err) {
    const int32_t q = blockIdx.y;
    const int lane = threadIdx.x & 31;
    const int32_t L = qlen[q];
    const int64_t o = qoff[q];
    if (L < 0 || o < 0 || o + L > qflat_len) {
        if (threadIdx.x == 0 && blockIdx.x == 0) atomicOr(err, ERRBIT_SEQ_EXTENT);
        return;
    }
    const uint8_t *s = qflat + o;
    int32_t *c = counts + (int64_t)q * num_db;
    const int32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (int32_t p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p <= L - k; p += warps) {
        uint32_t v = 0;
        bool ok = true;
        for (int32_t m = 0; m < k; ++m) {
            const uint32_t r = s[p + m];
            ok &= r < (uint32_t)alpha;
            v = v * (uint32_t)alpha + r;
        }
        if (!ok || kmer_freqs[v] > freq_thresh) continue;
        const int64_t b = kmer_offsets[v], e = kmer_offsets[v + 1];
        for (int64_t h = b + lane; h < e; h += 32) {
            const int32_t t = entry_target(kmer_entries, kmer_targets, h);
            if (t >= 0 && t < num_db) {
                // the hit that lifts a target to min_hits lists it (once: counts only grow)
                if (atomicAdd(&c[t], 1) == min_hits - 1) {
                    const int32_t pos = atomicAdd(&n_cand[q], 1);
                    if (pos < CAND_CAP) cand[(int64_t)q * CAND_CAP + pos] = t;
                }
            } else {
                atomicOr(err, ERRBIT_PAIR_INDEX);
            }
        }
    }
}

constexpr int SELECT_THREADS = 1024;
constexpr int SELECT_UNROLL = 8;  // row values a thread loads at once

// Block-wide radix selection, 8 bits per level from bit `top_shift` down, over
// the values get(i), i < n, that are >= min_hits: sh[2] = their number; when it
// exceeds top_k, sh[0] = thr, the top_k-th largest value, and sh[1] = the
// number of values above thr (so top_k - sh[1] of those equal to thr are
// taken); else sh[0] = -1.
template <class Get>
__device__ void radix_threshold(Get get, int32_t n, int32_t min_hits, int32_t top_k, int top_shift, int32_t *hist,
                                int32_t *sh) {
    const int tid = threadIdx.x;
    if (tid == 0) { sh[0] = 0; sh[1] = 0; sh[2] = 0; }
    uint32_t mask = 0;
    for (int shift = top_shift; shift >= 0; shift -= 8) {
        for (int i = tid; i < 256; i += SELECT_THREADS) hist[i] = 0;
        __syncthreads();
        const uint32_t prefix = (uint32_t)sh[0];
        // SELECT_UNROLL independent loads per thread before any is used:
        // one block reads a whole count row per pass, so the pass is bound
        // by the loads it keeps in flight
        for (int32_t base = 0; base < n; base += SELECT_UNROLL * SELECT_THREADS) {
            int32_t v[SELECT_UNROLL];
#pragma unroll
            for (int u = 0; u < SELECT_UNROLL; ++u) {
                const int32_t i = base + u * SELECT_THREADS + tid;
                v[u] = i < n ? get(i) : 0;
            }
#pragma unroll
            for (int u = 0; u < SELECT_UNROLL; ++u) {
                const int32_t i = base + u * SELECT_THREADS + tid;
                if (i < n && v[u] >= min_hits && ((uint32_t)v[u] & mask) == prefix)
                    atomicAdd(&hist[((uint32_t)v[u] >> shift) & 255u], 1);
            }
        }
        __syncthreads();
        if (tid == 0) {
            if (shift == top_shift) {
                int32_t total = 0;
                for (int b = 0; b < 256; ++b) total += hist[b];
                sh[2] = total;
            }
            if (sh[2] > top_k) {
                int32_t above = sh[1], b = 255;
                for (; b > 0; --b) {
                    if (above + hist[b] >= top_k) break;
                    above += hist[b];
                }
                sh[0] = (int32_t)(prefix | ((uint32_t)b << shift));
                sh[1] = above;
            }
        }
        __syncthreads();
        if (sh[2] <= top_k) break;
        mask |= 255u << shift;
    }
    __syncthreads();
    if (tid == 0 && sh[2] <= top_k) { sh[0] = -1; sh[1] = 0; }
    __syncthreads();
}

// Bitonic sort of n (<= 2 * CAND_CAP 32-bit, or CAND_CAP 64-bit) keys in shared memory, ascending.
template <class K>
__device__ void block_bitonic(K *a, int32_t n, K pad) {
    const int tid = threadIdx.x;
    int32_t P = 1;
    while (P < n) P <<= 1;
    for (int32_t i = n + tid; i < P; i += SELECT_THREADS) a[i] = pad;
    __syncthreads();
    for (int32_t k = 2; k <= P; k <<= 1) {
        for (int32_t j = k >> 1; j > 0; j >>= 1) {
            for (int32_t i = tid; i < P; i += SELECT_THREADS) {
                const int32_t l = i ^ j;
                if (l > i) {
                    const K x = a[i], y = a[l];
                    if (((i & k) == 0) == (x > y)) { a[i] = y; a[l] = x; }
                }
            }
            __syncthreads();
        }
    }
}

// One block per query.  The surviving targets (value >= min_hits; values are
// the counts clamped to `clamp`): all of them in target-id order when at most
// top_k, else the top_k by value -- ties to the lower target id -- in
// descending value order, as clustkit's argsort(-scores) gives them
// (kmer_index.py:893-899, :1320-1325).  This kernel takes the queries whose
// candidate list is complete (min_hits >= 1, at most CAND_CAP listed: sorted
// by id in shared memory); the others are selected from their whole count row
// by the row_* kernels.
__global__ void __launch_bounds__(SELECT_THREADS)
phase_a_select_kernel(const int32_t *__restrict__ counts, int32_t num_db, int32_t min_hits, int32_t top_k,
                      int32_t clamp, int32_t top_shift, const int32_t *__restrict__ cand,
                      const int32_t *__restrict__ n_cand, int32_t *__restrict__ out_targets,
                      int32_t *__restrict__ out_scores, int32_t *__restrict__ out_n,
                      int32_t *__restrict__ capped_n) {
    using BlockScan = cub::BlockScan<int32_t, SELECT_THREADS>;
    __shared__ typename BlockScan::TempStorage scan_tmp;
    __shared__ uint64_t s_buf[CAND_CAP];  // sorted candidate ids, later the capped output's sort keys
    __shared__ int32_t hist[256];
    __shared__ int32_t sh[4], sh_run_eq, sh_run_sel;
    const int32_t q = blockIdx.x;
    const int tid = threadIdx.x;
    const int32_t *c = counts + (int64_t)q * num_db;
    int32_t *o_t = out_targets + (int64_t)q * top_k;
    int32_t *o_s = out_scores ? out_scores + (int64_t)q * top_k : nullptr;
    auto val = [&](int32_t t) { const int32_t v = c[t]; return v > clamp ? clamp : v; };
    if (!(min_hits >= 1 && n_cand[q] <= CAND_CAP)) return;  // a row query: the row_* kernels
    int32_t *s_id = (int32_t *)s_buf;
    {
        const int32_t n = n_cand[q];
        const int32_t *list = cand + (int64_t)q * CAND_CAP;
        for (int32_t i = tid; i < n; i += SELECT_THREADS) s_id[i] = list[i];
        block_bitonic<int32_t>(s_id, n, INT32_MAX);
        radix_threshold([&](int32_t i) { return val(s_id[i]); }, n, min_hits, top_k, top_shift, hist, sh);
        const int32_t thr = sh[0], take_eq = top_k - sh[1];
        if (tid == 0) { sh_run_eq = 0; sh_run_sel = 0; }
        __syncthreads();
        for (int32_t base = 0; base < n; base += SELECT_THREADS) {
            const int32_t i = base + tid;
            const int32_t t = i < n ? s_id[i] : 0;
            const int32_t v = i < n ? val(t) : -1;
            const int32_t is_eq = (i < n && thr >= 0 && v == thr) ? 1 : 0;
            int32_t eq_rank, eq_tot;
            BlockScan(scan_tmp).ExclusiveSum(is_eq, eq_rank, eq_tot);
            __syncthreads();
            const bool sel = i < n && (thr < 0 || v > thr || (is_eq && sh_run_eq + eq_rank < take_eq));
            int32_t pos, sel_tot;
            BlockScan(scan_tmp).ExclusiveSum(sel ? 1 : 0, pos, sel_tot);
            if (sel) {
                o_t[sh_run_sel + pos] = t;
                if (o_s) o_s[sh_run_sel + pos] = v;
            }
            __syncthreads();
            if (tid == 0) { sh_run_eq += eq_tot; sh_run_sel += sel_tot; }
            __syncthreads();
        }
    }
    const int32_t total = sh[2];
    const int32_t n_out = total < top_k ? total : top_k;
    __syncthreads();
    // capped: the kept targets in descending value order, ties by id
    if (total > top_k && top_k <= CAND_CAP) {
        for (int32_t i = tid; i < n_out; i += SELECT_THREADS) {
            const int32_t t = o_t[i];
            s_buf[i] = ((uint64_t)(uint32_t)(0x7fffffff - val(t)) << 32) | (uint32_t)t;
        }
        block_bitonic<uint64_t>(s_buf, n_out, ~0ull);
        for (int32_t i = tid; i < n_out; i += SELECT_THREADS) {
            const int32_t t = (int32_t)(s_buf[i] & 0xffffffffu);
            o_t[i] = t;
            if (o_s) o_s[i] = 0x7fffffff - (int32_t)(s_buf[i] >> 32);
        }
    }
    if (tid == 0) {
        out_n[q] = n_out;
        if (capped_n) capped_n[q] = (total > top_k && top_k > CAND_CAP) ? n_out : 0;
    }
}

// ----------------------------------------------------------------- row select
// The same selection for the queries whose survivors are not all in their
// candidate list, over the whole count row, by ROW_BLOCKS blocks per query
// (one block scanning a 500,000-counter row took 0.37 ms for one query).
// The row is cut into ROW_SLOTS warp slices in target order.  The radix
// threshold runs digit by digit: row_hist_kernel adds each block's histogram
// of the surviving values that match the digits so far into the query's
// global one and its last block picks the digit (the state stays on the
// device: no host synchronisation).  Then row_count_kernel counts each
// slice's values above and at the threshold, row_offsets_kernel turns those
// into each slice's output position and its share of the ties (lowest ids
// first), row_write_kernel writes the kept targets in id order and
// row_sort_kernel puts a capped row in (value desc, id asc) order.
// Per-query state: threshold (or -1: keep every survivor), count above its
// last digit, survivors, mode (0 in progress, 1 threshold known, 2 a list
// query: left to phase_a_select_kernel).  The digit pick runs in the last
// histogram block of each query (no launch of its own).
constexpr int ROW_BLOCKS = 128;
constexpr int ROW_THREADS = 256;
constexpr int ROW_SLOTS = ROW_BLOCKS * (ROW_THREADS / 32);  // 1,024 warp slices per row

__device__ __forceinline__ int32_t row_value(const int32_t *c, int64_t t, int32_t clamp) {
    const int32_t v = c[t];
    return v > clamp ? clamp : v;
}

// One radix digit of every row query's threshold.  Each block adds its
// slice's histogram into the query's global one; the last block of the query
// to finish (a counter, after a fence) picks the digit as radix_threshold
// does, records the state and clears the histogram and the counter for the
// next pass.  The first pass also sets every query's mode (a list query is
// marked and skipped).
__global__ void __launch_bounds__(ROW_THREADS)
row_hist_kernel(const int32_t *__restrict__ counts, int32_t num_db, int32_t min_hits, int32_t clamp, int32_t shift,
                uint32_t mask, int32_t first, int32_t last, const int32_t *__restrict__ n_cand, int32_t top_k,
                int32_t *__restrict__ state, int32_t *__restrict__ ghist, int32_t *__restrict__ done, int32_t W) {
    __shared__ int32_t h[256];
    __shared__ int32_t is_last;
    const int32_t q = blockIdx.y;
    int32_t *s = state + 4 * q;
    uint32_t prefix = 0;
    if (first) {
        if (min_hits >= 1 && n_cand[q] <= CAND_CAP) {  // a list query, the same for the whole block
            if (blockIdx.x == 0 && threadIdx.x == 0) { s[0] = 0; s[1] = 0; s[2] = 0; s[3] = 2; }
            return;
        }
    } else {
        if (s[3] != 0) return;  // the same for the whole block
        prefix = (uint32_t)s[0];
    }
    for (int i = threadIdx.x; i < 256; i += ROW_THREADS) h[i] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t slot = (int64_t)blockIdx.x * (ROW_THREADS / 32) + (threadIdx.x >> 5);
    const int64_t a0 = slot * W, a1 = a0 + W < num_db ? a0 + W : num_db;
    const int32_t *c = counts + (int64_t)q * num_db;
    for (int64_t base = a0; base < a1; base += 32 * SELECT_UNROLL) {
        int32_t v[SELECT_UNROLL];
#pragma unroll
        for (int u = 0; u < SELECT_UNROLL; ++u) {
            const int64_t t = base + u * 32 + lane;
            v[u] = t < a1 ? row_value(c, t, clamp) : 0;
        }
#pragma unroll
        for (int u = 0; u < SELECT_UNROLL; ++u) {
            const int64_t t = base + u * 32 + lane;
            if (t < a1 && v[u] >= min_hits && ((uint32_t)v[u] & mask) == prefix)
                atomicAdd(&h[((uint32_t)v[u] >> shift) & 255u], 1);
        }
    }
    __syncthreads();
    int32_t *g = ghist + (int64_t)q * 256;
    for (int i = threadIdx.x; i < 256; i += ROW_THREADS)
        if (h[i]) atomicAdd(&g[i], h[i]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(&done[q], 1) == (int32_t)gridDim.x - 1;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    for (int i = threadIdx.x; i < 256; i += ROW_THREADS) h[i] = __ldcg(&g[i]);
    __syncthreads();
    if (threadIdx.x == 0) {
        int32_t above = first ? 0 : s[1], total = first ? 0 : s[2];
        bool decided = false;
        if (first) {
            for (int b = 0; b < 256; ++b) total += h[b];
            if (total <= top_k) { s[0] = -1; s[1] = 0; s[2] = total; s[3] = 1; decided = true; }
        }
        if (!decided) {
            int32_t b = 255;
            for (; b > 0; --b) {
                if (above + h[b] >= top_k) break;
                above += h[b];
            }
            s[0] = (int32_t)(prefix | ((uint32_t)b << shift));
            s[1] = above;
            s[2] = total;
            s[3] = last ? 1 : 0;
        }
        done[q] = 0;
    }
    for (int i = threadIdx.x; i < 256; i += ROW_THREADS) g[i] = 0;
}

__global__ void __launch_bounds__(ROW_THREADS)
row_count_kernel(const int32_t *__restrict__ counts, int32_t num_db, int32_t min_hits, int32_t clamp,
                 const int32_t *__restrict__ state, int32_t W, int32_t *__restrict__ wcnt) {
    const int32_t q = blockIdx.y;
    if (state[4 * q + 3] != 1) return;
    const int32_t thr = state[4 * q];
    const int lane = threadIdx.x & 31;
    const int64_t slot = (int64_t)blockIdx.x * (ROW_THREADS / 32) + (threadIdx.x >> 5);
    const int64_t a0 = slot * W, a1 = a0 + W < num_db ? a0 + W : num_db;
    const int32_t *c = counts + (int64_t)q * num_db;
    int32_t n_strict = 0, n_eq = 0;
    for (int64_t base = a0; base < a1; base += 32 * SELECT_UNROLL) {
        int32_t v[SELECT_UNROLL];
#pragma unroll
        for (int u = 0; u < SELECT_UNROLL; ++u) {
            const int64_t t = base + u * 32 + lane;
            v[u] = t < a1 ? row_value(c, t, clamp) : 0;
        }
#pragma unroll
        for (int u = 0; u < SELECT_UNROLL; ++u) {
            const int64_t t = base + u * 32 + lane;
            const bool surv = t < a1 && v[u] >= min_hits;
            n_strict += __popc(__ballot_sync(0xffffffffu, surv && (thr < 0 || v[u] > thr)));
            n_eq += __popc(__ballot_sync(0xffffffffu, surv && thr >= 0 && v[u] == thr));
        }
    }
    if (lane == 0) {
        wcnt[((int64_t)q * ROW_SLOTS + slot) * 2] = n_strict;
        wcnt[((int64_t)q * ROW_SLOTS + slot) * 2 + 1] = n_eq;
    }
}

// One thread per slice: ties are taken from the lowest slices (lowest ids)
// until take_eq; each slice's output starts after the kept targets of the
// slices before it.
__global__ void __launch_bounds__(ROW_SLOTS)
row_offsets_kernel(const int32_t *__restrict__ state, const int32_t *__restrict__ wcnt, int32_t top_k,
                   int32_t *__restrict__ woff, int32_t *__restrict__ out_n, int32_t *__restrict__ capped_n) {
    using Scan = cub::BlockScan<int32_t, ROW_SLOTS>;
    __shared__ typename Scan::TempStorage tmp;
    const int32_t q = blockIdx.x;
    if (state[4 * q + 3] != 1) return;
    const int32_t thr = state[4 * q], take_eq = top_k - state[4 * q + 1], total = state[4 * q + 2];
    const int32_t i = threadIdx.x;
    const int32_t strict = wcnt[((int64_t)q * ROW_SLOTS + i) * 2], eq = wcnt[((int64_t)q * ROW_SLOTS + i) * 2 + 1];
    int32_t eq_base;
    Scan(tmp).ExclusiveSum(eq, eq_base);
    __syncthreads();
    int32_t take = take_eq - eq_base;
    take = thr < 0 ? 0 : (take < 0 ? 0 : (take > eq ? eq : take));
    int32_t out_base;
    Scan(tmp).ExclusiveSum(strict + take, out_base);
    woff[((int64_t)q * ROW_SLOTS + i) * 2] = eq_base;
    woff[((int64_t)q * ROW_SLOTS + i) * 2 + 1] = out_base;
    if (i == 0) {
        const int32_t n_out = total < top_k ? total : top_k;
        out_n[q] = n_out;
        if (capped_n) capped_n[q] = (total > top_k && top_k > CAND_CAP) ? n_out : 0;
    }
}

__global__ void __launch_bounds__(ROW_THREADS)
row_write_kernel(const int32_t *__restrict__ counts, int32_t num_db, int32_t min_hits, int32_t clamp,
                 const int32_t *__restrict__ state, int32_t W, const int32_t *__restrict__ woff, int32_t top_k,
                 int32_t *__restrict__ out_targets, int32_t *__restrict__ out_scores) {
    const int32_t q = blockIdx.y;
    if (state[4 * q + 3] != 1) return;
    const int32_t thr = state[4 * q], take_eq = top_k - state[4 * q + 1];
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    const int64_t slot = (int64_t)blockIdx.x * (ROW_THREADS / 32) + (threadIdx.x >> 5);
    const int64_t a0 = slot * W, a1 = a0 + W < num_db ? a0 + W : num_db;
    const int32_t *c = counts + (int64_t)q * num_db;
    int32_t *o_t = out_targets + (int64_t)q * top_k;
    int32_t *o_s = out_scores ? out_scores + (int64_t)q * top_k : nullptr;
    int32_t eq_seen = woff[((int64_t)q * ROW_SLOTS + slot) * 2], written = woff[((int64_t)q * ROW_SLOTS + slot) * 2 + 1];
    for (int64_t base = a0; base < a1; base += 32 * SELECT_UNROLL) {
        int32_t v[SELECT_UNROLL];
#pragma unroll
        for (int u = 0; u < SELECT_UNROLL; ++u) {
            const int64_t t = base + u * 32 + lane;
            v[u] = t < a1 ? row_value(c, t, clamp) : 0;
        }
#pragma unroll
        for (int u = 0; u < SELECT_UNROLL; ++u) {
            const int64_t t = base + u * 32 + lane;
            const bool surv = t < a1 && v[u] >= min_hits;
            const bool strict = surv && (thr < 0 || v[u] > thr);
            const bool is_eq = surv && thr >= 0 && v[u] == thr;
            const uint32_t eq_b = __ballot_sync(0xffffffffu, is_eq);
            const bool sel = strict || (is_eq && eq_seen + __popc(eq_b & lt) < take_eq);
            const uint32_t sel_b = __ballot_sync(0xffffffffu, sel);
            if (sel) {
                const int32_t at = written + __popc(sel_b & lt);
                o_t[at] = (int32_t)t;
                if (o_s) o_s[at] = v[u];
            }
            eq_seen += __popc(eq_b);
            written += __popc(sel_b);
        }
    }
}

// A capped row of at most CAND_CAP kept targets in (value desc, id asc)
// order, in shared memory (longer capped rows take the segmented sort).
__global__ void __launch_bounds__(SELECT_THREADS)
row_sort_kernel(const int32_t *__restrict__ counts, int32_t num_db, int32_t clamp, const int32_t *__restrict__ state,
                int32_t top_k, int32_t *__restrict__ out_targets, int32_t *__restrict__ out_scores) {
    __shared__ uint64_t s_buf[CAND_CAP];
    const int32_t q = blockIdx.x;
    if (state[4 * q + 3] != 1 || state[4 * q + 2] <= top_k || top_k > CAND_CAP) return;
    const int32_t *c = counts + (int64_t)q * num_db;
    int32_t *o_t = out_targets + (int64_t)q * top_k;
    int32_t *o_s = out_scores ? out_scores + (int64_t)q * top_k : nullptr;
    for (int32_t i = threadIdx.x; i < top_k; i += SELECT_THREADS) {
        const int32_t t = o_t[i];
        s_buf[i] = ((uint64_t)(uint32_t)(0x7fffffff - row_value(c, t, clamp)) << 32) | (uint32_t)t;
    }
    block_bitonic<uint64_t>(s_buf, top_k, ~0ull);
    for (int32_t i = threadIdx.x; i < top_k; i += SELECT_THREADS) {
        o_t[i] = (int32_t)(s_buf[i] & 0xffffffffu);
        if (o_s) o_s[i] = 0x7fffffff - (int32_t)(s_buf[i] >> 32);
    }
}

// Rows capped at more than CAND_CAP targets leave the select in id order; a
// segmented sort of (score desc, id asc) keys puts them in the order the
// shorter capped rows get in shared memory.  Rows that were not capped are
// empty segments.
__global__ void cap_keys_kernel(const int32_t *__restrict__ t, const int32_t *__restrict__ sc,
                                const int32_t *__restrict__ capped_n, int32_t top_k, uint64_t *__restrict__ keys,
                                int32_t *__restrict__ beg, int32_t *__restrict__ end) {
    const int32_t q = blockIdx.y;
    const int32_t n = capped_n[q];
    const int64_t row = (int64_t)q * top_k;
    if (blockIdx.x == 0 && threadIdx.x == 0) { beg[q] = (int32_t)row; end[q] = (int32_t)(row + n); }
    for (int32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
        keys[row + j] = ((uint64_t)(uint32_t)(0x7fffffff - sc[row + j]) << 32) | (uint32_t)t[row + j];
}

__global__ void cap_unpack_kernel(const uint64_t *__restrict__ keys, const int32_t *__restrict__ capped_n,
                                  int32_t top_k, int32_t *__restrict__ t, int32_t *__restrict__ sc) {
    const int32_t q = blockIdx.y;
    const int32_t n = capped_n[q];
    const int64_t row = (int64_t)q * top_k;
    for (int32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const uint64_t k = keys[row + j];
        t[row + j] = (int32_t)(k & 0xffffffffu);
        sc[row + j] = 0x7fffffff - (int32_t)(k >> 32);
    }
}

// ----------------------------------------------------------------- similar k-mers
// clustkit/kmer_index.py:1187-1291: with k = 5 every 5-mer whose BLOSUM62
// column sum against a query 5-mer reaches the threshold T adds that sum to
// each target of its posting list (frequency in (0, freq_thresh]).  Stage 1
// (nbr_weight_kernel) sums, per query, each 5-mer's scores over the query's
// positions; stage 2 walks the posting lists of the 5-mers with a sum.
//
// Stage 1.  A block takes one query and NB_PREFIXES first residue pairs
// (a0, a1) -- 56,000 5-mers, whose sums fit its shared memory -- and its warps
// take the query's positions.  The pairs (a2, a3) ordered by score against two
// query residues depend on these residues alone: nbr_tables_kernel orders them
// for all 400 pairs of residues once a call (640 KB).  At a position the pairs
// that can still reach the threshold after (a0, a1), with the best last
// residue, are then a prefix of one such list: the lanes hold the prefix
// lengths of the block's (a0, a1), and the concatenated prefixes go to the
// lanes 32 at a time, so no lane tests a combination that clustkit's bound
// would prune.  A combination's last residues are one AND: the residues that
// reach the threshold (a table by query residue and score needed) and the
// indexed 5-mers of those four residues (one bit each, kmer_valid_kernel: 640
// KB, where the frequencies themselves are 12.8 MB).  The block then writes its
// 5-mers with a sum, in order, to its region of the weights.
// Summing first makes stage 2's work distinct 5-mers in index order (a 64-query
// batch lists 144 M triples; many repeat a 5-mer of the same query), and leaves
// nothing whose size the host would have to know.
// 64 queries against 200,000 sequences: 1.1 ms (the first form listed triples,
// a warp testing all 400 continuations of every surviving pair (a0,
// a1) and a lane reading up to 20 frequencies for each: 8.1 ms).
constexpr int32_t NB_PAIRS = 400;
constexpr int32_t NB_KMERS = 3200000;    // 20^5
constexpr int32_t NB_VALID = 160000;     // 20^4
constexpr int32_t NB_PREFIXES = 7;       // (a0, a1) pairs of a block; 6 where the matrix's tables need the room
constexpr int32_t NB_REGION = NB_PREFIXES * 8000;  // room for a block's 5-mers
constexpr int NB_WARPS = 32;
constexpr int32_t NB_QUERIES = 64;       // queries whose weights are held at a time (336,000 bytes a block of 5-mers)

// Bit a of valid[u]: the 5-mer of the four residues u and last residue a has a
// frequency in 1 .. freq_thresh.  A warp turns 640 frequencies into 20 ballots,
// whose bits are then 32 words of 20.
__global__ void kmer_valid_kernel(const int32_t *__restrict__ freqs, int32_t freq_thresh,
                                  uint32_t *__restrict__ valid) {
    const int lane = threadIdx.x & 31;
    const int32_t base = (int32_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32;
    if (base >= NB_VALID) return;  // a multiple of 32
    const int32_t bit = 20 * lane, first = bit >> 5;
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int r = 0; r < 20; ++r) {
        const int32_t f = __ldg(freqs + (int64_t)base * 20 + r * 32 + lane);
        const uint32_t bal = __ballot_sync(0xffffffffu, f != 0 && f <= freq_thresh);
        if (r == first) lo = bal;
        if (r == first + 1) hi = bal;
    }
    valid[base + lane] = __funnelshift_r(lo, hi, bit & 31) & 0xfffffu;
}

// One warp per pair of query residues (q2, q3): the pairs (a2, a3) by score,
// descending: ordered[at] = a2 * 20 + a3 | bin << 16 with bin = score - 2 smin,
// and from[b] = the number of pairs of bin b or above.
__global__ void __launch_bounds__(32)
nbr_tables_kernel(const int8_t *__restrict__ sub, int32_t smin, int32_t bins, uint32_t *__restrict__ ordered_all,
                  int32_t *__restrict__ from_all) {
    constexpr uint32_t FULL = 0xffffffffu;
    __shared__ int32_t from[512];
    const int lane = threadIdx.x;
    const int8_t *Sa = sub + blockIdx.x / 20 * 20, *Sb = sub + blockIdx.x % 20 * 20;
    uint32_t *ordered = ordered_all + (size_t)blockIdx.x * NB_PAIRS;
    for (int32_t b = lane; b < bins; b += 32) from[b] = 0;
    __syncwarp();
    for (int32_t t = lane; t < NB_PAIRS; t += 32) atomicAdd(&from[Sa[t / 20] + Sb[t % 20] - 2 * smin], 1);
    __syncwarp();
    int32_t above = 0;  // pairs in the bins already passed (higher scores)
    for (int32_t top = bins - 1; top >= 0; top -= 32) {
        const int32_t b = top - lane;
        const int32_t n = b >= 0 ? from[b] : 0;
        int32_t incl = n;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int32_t x = __shfl_up_sync(FULL, incl, d);
            if (lane >= d) incl += x;
        }
        if (b >= 0) from[b] = above + incl - n;
        above += __shfl_sync(FULL, incl, 31);
    }
    __syncwarp();
    for (int32_t t = lane; t < NB_PAIRS; t += 32) {
        const int32_t b = Sa[t / 20] + Sb[t % 20] - 2 * smin;
        ordered[atomicAdd(&from[b], 1)] = (uint32_t)t | ((uint32_t)b << 16);  // each bin's count goes on top
    }
    __syncwarp();
    for (int32_t b = lane; b < bins; b += 32) from_all[(size_t)blockIdx.x * bins + b] = from[b];
}

// Shared memory of stage 1: the sums, the matrix, the table of last residues
// (20 rows of `range` + 1 words, range = largest - smallest matrix entry).
__host__ __device__ constexpr size_t nbr_smem(int32_t prefixes, int32_t range) {
    return ((size_t)prefixes * 8000 + 400 + 20 * (size_t)(range + 1)) * 4;
}

// Grid (blocks of 5-mers, queries).  Region q * gridDim.x + block of the
// weights gets n[region] 5-mers: kmer (counted from the block's first) and
// weight, in 5-mer order.  *listed grows by the (query position, 5-mer) pairs
// that reached the threshold.
__global__ void __launch_bounds__(NB_WARPS * 32, 1)
nbr_weight_kernel(const uint8_t *__restrict__ qflat, int64_t qflat_len, const int64_t *__restrict__ qoff,
                  const int32_t *__restrict__ qlen, const int8_t *__restrict__ sub, int32_t smin, int32_t range,
                  int32_t T, const uint32_t *__restrict__ valid, const uint32_t *__restrict__ ordered_all,
                  const int32_t *__restrict__ from_all, int32_t prefixes, int32_t *__restrict__ n,
                  uint16_t *__restrict__ kmer, int32_t *__restrict__ weight, unsigned long long *__restrict__ listed,
                  int32_t *err) {
    constexpr uint32_t FULL = 0xffffffffu;
    extern __shared__ int32_t nb_smem[];
    __shared__ int32_t warp_n[NB_WARPS];
    const int32_t size = prefixes * 8000;
    int32_t *W = nb_smem, *S = nb_smem + size;
    uint32_t *reach = (uint32_t *)(S + 400);  // [query residue][score needed - smin]: last residues that give it
    const int32_t q = blockIdx.y, region = q * gridDim.x + blockIdx.x;
    const int32_t L = qlen[q];
    const int64_t o = qoff[q];
    // both exits are the same for the whole block (before its first barrier)
    const bool bad = L < 0 || o < 0 || o + L > qflat_len;
    if (bad || L < 5) {
        if (threadIdx.x == 0) {
            n[region] = 0;
            if (bad && blockIdx.x == 0) atomicOr(err, ERRBIT_SEQ_EXTENT);
        }
        return;
    }
    for (int i = threadIdx.x; i < size / 4; i += NB_WARPS * 32) ((int4 *)W)[i] = make_int4(0, 0, 0, 0);
    for (int i = threadIdx.x; i < 400; i += NB_WARPS * 32) S[i] = sub[i];
    __syncthreads();
    for (int i = threadIdx.x; i < 20 * (range + 1); i += NB_WARPS * 32) {
        const int32_t a = i / (range + 1), need = i - a * (range + 1) + smin;
        uint32_t m = 0;
        for (int b = 0; b < 20; ++b) m |= S[a * 20 + b] >= need ? 1u << b : 0u;
        reach[i] = m;
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int32_t bins = 2 * range + 1;
    const uint8_t *sq = qflat + o;
    // this lane's first residues (the first `prefixes` lanes)
    const int32_t a01 = blockIdx.x * prefixes + lane;
    const bool has = lane < prefixes && a01 < NB_PAIRS;
    const int32_t a0 = has ? a01 / 20 : 0, a1 = has ? a01 % 20 : 0;
    uint32_t count = 0;
    for (int32_t p = warp; p <= L - 5; p += NB_WARPS) {
        const int32_t q0 = sq[p], q1 = sq[p + 1], q2 = sq[p + 2], q3 = sq[p + 3], q4 = sq[p + 4];
        if (q0 >= 20 || q1 >= 20 || q2 >= 20 || q3 >= 20 || q4 >= 20) continue;  // the same for the whole warp
        const uint32_t *reach4 = reach + q4 * (range + 1);
        int32_t m4 = S[q4 * 20 + (lane < 20 ? lane : 0)];  // the best last residue's score
        m4 = __reduce_max_sync(FULL, m4);
        const int32_t s01 = S[q0 * 20 + a0] + S[q1 * 20 + a1];
        // how many (a2, a3) can reach T: those of bin `need` or above
        const int32_t need = T - m4 - s01 - 2 * smin;
        const int32_t pair = q2 * 20 + q3;
        const int32_t mine = has && need < bins ? __ldg(from_all + pair * bins + (need > 0 ? need : 0)) : 0;
        int32_t incl = mine;
#pragma unroll
        for (int d = 1; d < 8; d <<= 1) {  // prefixes <= 7
            const int32_t x = __shfl_up_sync(FULL, incl, d);
            if (lane >= d) incl += x;
        }
        const int32_t excl = incl - mine, cells = __shfl_sync(FULL, incl, 7);
        const uint32_t *ordered = ordered_all + pair * NB_PAIRS;
        for (int32_t k0 = 0; k0 < cells; k0 += 32) {
            const int32_t k = k0 + lane;
            int32_t a = 0;  // the last prefix that starts at or before k
#pragma unroll
            for (int step = 4; step; step >>= 1)
                if (__shfl_sync(FULL, excl, a + step) <= k) a += step;
            const int32_t at = k - __shfl_sync(FULL, excl, a);
            const int32_t sa = __shfl_sync(FULL, s01, a);
            if (k < cells) {
                const uint32_t x = __ldg(ordered + at);
                const int32_t s4 = sa + (int32_t)(x >> 16) + 2 * smin, v4 = a * NB_PAIRS + (int32_t)(x & 0xffffu);
                const int32_t w = T - s4 - smin;  // at most m4 - smin
                uint32_t bits = reach4[w < 0 ? 0 : w] & __ldg(valid + blockIdx.x * prefixes * NB_PAIRS + v4);
                count += __popc(bits);
                while (bits) {
                    const int b = __ffs(bits) - 1;
                    bits &= bits - 1;
                    atomicAdd(&W[v4 * 20 + b], s4 + S[q4 * 20 + b]);
                }
            }
        }
    }
    count = __reduce_add_sync(FULL, count);
    if (lane == 0 && count) atomicAdd(listed, (unsigned long long)count);
    __syncthreads();
    // the block's 5-mers with a sum (T >= 1, so a listed 5-mer's is positive):
    // each warp a slice, counted, then written behind the slices before it
    const int32_t slice = (size / 32 + NB_WARPS - 1) / NB_WARPS * 32;
    const int32_t w0 = warp * slice, w1 = w0 + slice < size ? w0 + slice : size;
    int32_t here = 0;
    for (int32_t i = w0 + lane; i < w1; i += 32) here += W[i] != 0;
    here = __reduce_add_sync(FULL, here);
    if (lane == 0) warp_n[warp] = here;
    __syncthreads();
    const int32_t wn = warp_n[lane];
    const int32_t total = __reduce_add_sync(FULL, wn);
    int32_t at = __reduce_add_sync(FULL, lane < warp ? wn : 0);
    uint16_t *ko = kmer + (size_t)region * NB_REGION;
    int32_t *wo = weight + (size_t)region * NB_REGION;
    for (int32_t i0 = w0; i0 < w1; i0 += 32) {
        const int32_t x = i0 + lane < w1 ? W[i0 + lane] : 0;
        const uint32_t bal = __ballot_sync(FULL, x != 0);
        if (x != 0) {
            const int32_t to = at + __popc(bal & ((1u << lane) - 1u));
            ko[to] = (uint16_t)(i0 + lane);
            wo[to] = x;
        }
        at += __popc(bal);
    }
    if (threadIdx.x == 0) n[region] = total;
}

__global__ void fill_kernel(int32_t *a, int32_t n, int32_t v) {
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) a[i] = v;
}

// Stage 2 on the count rows, for few queries.  A persistent grid; each block
// takes runs of a region's 5-mers (a ticket counter; regions in query order, so
// the blocks in flight add into one or two queries' count rows, which stay in
// L2).  A warp takes 32 5-mers at once: each lane loads one and its
// posting-list bounds -- 32 independent loads instead of 32 chains -- then the
// warp walks the concatenated lists, lane k of each round taking entry k of
// the stream (its list found by a binary search over the lanes' exclusive
// prefix sums of list lengths) and adding the 5-mer's weight to the entry's
// target in the query's row.  Bound by L2's atomic units (about 200 G adds/s).
constexpr int32_t NB_RUN = 1024;  // 5-mers of a run

// A region's first run: the runs before it (one block; regions in order).
__global__ void __launch_bounds__(1024)
nbr_runs_kernel(const int32_t *__restrict__ n, int32_t regions, int32_t *__restrict__ run0) {
    using Scan = cub::BlockScan<int32_t, 1024>;
    __shared__ typename Scan::TempStorage tmp;
    int32_t run = 0, sum;
    for (int32_t g0 = 0; g0 < regions; g0 += 1024) {
        const int32_t g = g0 + threadIdx.x;
        int32_t at;
        Scan(tmp).ExclusiveSum(g < regions ? (n[g] + NB_RUN - 1) / NB_RUN : 0, at, sum);
        if (g < regions) run0[g] = run + at;
        run += sum;
        __syncthreads();
    }
    if (threadIdx.x == 0) run0[regions] = run;
}

__global__ void __launch_bounds__(256)
nbr_walk_kernel(const int32_t *__restrict__ n, const int32_t *__restrict__ run0, const uint16_t *__restrict__ kmer,
                const int32_t *__restrict__ weight, int32_t regions, int32_t n_blocks, int32_t block_kmers,
                const int64_t *__restrict__ kmer_offsets, const int64_t *__restrict__ kmer_entries,
                const int32_t *__restrict__ kmer_targets, int32_t num_db, int32_t *__restrict__ counts,
                unsigned long long *__restrict__ ticket, const unsigned long long *__restrict__ order, int32_t *err) {
    constexpr uint32_t FULL = 0xffffffffu;
    __shared__ int32_t s_run;
    if (order && order[0] == order[1] && order[2] == 0) return;  // the walk by target ranges has taken the call
    const int lane = threadIdx.x & 31;
    const int32_t runs = run0[regions];
    for (;;) {
        if (threadIdx.x == 0) {
            const unsigned long long t = atomicAdd(ticket, 1ull);
            s_run = t < (unsigned long long)runs ? (int32_t)t : -1;
        }
        __syncthreads();
        const int32_t run = s_run;
        __syncthreads();  // every thread has read s_run before it is written again
        if (run < 0) break;  // the same for the whole block
        int32_t g = 0, hi = regions;  // the last region whose first run is at or before this one
        while (hi - g > 1) {
            const int32_t mid = (g + hi) >> 1;
            if (run0[mid] <= run) g = mid; else hi = mid;
        }
        const int32_t c0 = (run - run0[g]) * NB_RUN, c1 = c0 + NB_RUN < n[g] ? c0 + NB_RUN : n[g];
        const int32_t v0 = g % n_blocks * block_kmers;
        int32_t *row = counts + (int64_t)(g / n_blocks) * num_db;
        for (int32_t base = c0 + (threadIdx.x >> 5) * 32; base < c1; base += 256) {
            const int32_t e = base + lane;
            int64_t b = 0;
            int32_t len = 0, w = 0;
            if (e < c1) {
                const int32_t v = v0 + kmer[(size_t)g * NB_REGION + e];
                w = weight[(size_t)g * NB_REGION + e];
                b = kmer_offsets[v];
                len = (int32_t)(kmer_offsets[v + 1] - b);
            }
            int32_t incl = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int32_t t = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += t;
            }
            const int32_t excl = incl - len;
            const int32_t total = __shfl_sync(FULL, incl, 31);
            // rounds are warp-uniform so that every shuffle reads a live lane
            for (int32_t k0 = 0; k0 < total; k0 += 32) {
                const int32_t k = k0 + lane;
                // the stream's entry k belongs to the last lane whose list starts
                // at or before k (lanes with empty lists share their successor's
                // start and lose to it)
                int32_t o = 0;
#pragma unroll
                for (int step = 16; step; step >>= 1) {
                    const int32_t cand = o + step;
                    if (__shfl_sync(FULL, excl, cand) <= k) o = cand;
                }
                const int64_t h = __shfl_sync(FULL, b, o) + (k - __shfl_sync(FULL, excl, o));
                const int32_t wo = __shfl_sync(FULL, w, o);
                if (k < total) {
                    const int32_t t = entry_target(kmer_entries, kmer_targets, h);
                    if (t < 0 || t >= num_db) {
                        atomicOr(err, ERRBIT_PAIR_INDEX);
                    } else {
                        // no candidate list here (most of the database crosses
                        // min_hits in this mode; the select scans the row): the
                        // add's result is unused
                        atomicAdd(&row[t], wo);
                    }
                }
            }
        }
    }
}

// Stage 2 by target ranges, for calls of several queries.  Here the targets
// are cut into ranges of at most NB_RANGE, whose counters for one query fit a
// block's shared memory: a work unit is (range, some blocks of 5-mers, query);
// its block adds the postings that fall in the range into shared memory and
// then adds the counters to the query's row, coalesced.  Every list is cut at
// the range boundaries once per call (frag_kernel), so a block reads only its
// range's part of a list.  Units are taken range by range, then 5-mers by
// 5-mers, with all queries' units of these together, so that the cuts and
// postings in use stay in L2 (in query order the same walk read 45 GB from
// DRAM).  A lane walks its own 5-mer's part, eight postings (a sector) a load
// and two loads in flight, with the next 5-mer's cut and the one after's
// weight on their way: a part is a few postings long, sharing parts among
// lanes cost more shuffles than the idle lanes do, and one load at a time left
// the walk waiting for L2.
// The cuts need lists in target order, as the index build leaves them;
// order_kernel checks that (and that targets lie in the database), and a call
// whose lists are not goes to the walk above.  So does one whose lists are too
// short to be cut (nbr_least_postings).
// 64 queries, 200,000 sequences: 5.3 ms, with 0.2 for the cuts and the check;
// the walk on the count rows took 11.4 (listed triples, repeats and all).
constexpr int32_t NB_RANGE = 56 * 1024;   // counters of a block: 224 KB of shared memory
// 917,504 targets, 25.6 MB of cuts each.  Past it (1,500,000 targets, 27 ranges)
// 64 queries take 53.2 ms on the count rows and would 39.7 by ranges at 350
// residues a target, 19.7 and 27.2 at 120; 4 queries 4.5 and 6.3, 1.7 and 3.7
constexpr int32_t NB_MAX_RANGES = 16;
constexpr int NB_RW_THREADS = 1024;
constexpr int32_t NB_RANGE_MIN_QUERIES = 4;

// Postings an index needs for the cuts to pay in a call of nq queries, against
// the walk on the count rows: a query reads its lists' cuts range by range (they
// leave L2 as the ranges become more) and adds the counters to its row, and the
// cutting and checking are spread over the queries.  Phase A of 300-residue
// queries, count rows and ranges, ms: 57,000 targets of 120 residues 4 queries
// 0.29 0.32, 64 2.07 1.80; of 350 0.45 0.41, 3.85 2.23.  460,000 (9 ranges) of
// 120 0.70 1.16, 7.26 8.54; of 350 1.59 1.93, 17.8 12.6.  900,000 (16) of 120
// 1.15 2.12, 12.5 15.8; of 350 2.96 3.58, 32.7 23.5.  5,000 of 350 0.24 0.26,
// 1.51 1.34.  The line below is fitted to 300 such calls (500 to 1,500,000
// targets, 4 to 64 queries): 0.3 % over the better walk of each, 9 % at most; by
// ranges from 4 queries on cost 17 % and up to 2.2 times.
static int64_t nbr_least_postings(double ranges, double targets, double nq) {
    const double squared = ranges * ranges;
    return (int64_t)(NB_KMERS * (0.05 * squared + 2e-5 * targets + (1.5 + 2.0 * ranges + 2.5 * squared) / nq));
}

// postings the walk can number: an octet's end and the step past it stay below 2^32
constexpr int64_t NB_MAX_POSTINGS = 0xffffff00;

// Whether every list is in target order: the places where a target is below
// the one before it, over the whole index, less those where a list starts
// (order[0] - order[1], 0 when all are in order); order[2] counts targets
// outside the database, and is not zero for an index too short or too long for
// the walk by ranges.
__global__ void order_kernel(const int64_t *__restrict__ kmer_offsets, const int64_t *__restrict__ kmer_entries,
                             const int32_t *__restrict__ kmer_targets, int32_t n_kmers, int32_t num_db, int64_t least,
                             unsigned long long *__restrict__ order) {
    const int64_t total = kmer_offsets[n_kmers], step = (int64_t)gridDim.x * blockDim.x;
    const int64_t me = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (total < least || total > NB_MAX_POSTINGS) {  // left to the walk on the count rows
        if (me == 0) order[2] = 1;
        return;
    }
    uint32_t falls = 0, starts = 0, outside = 0;
    for (int64_t h = me * 4; h < total; h += step * 4) {
        int32_t before = h > 0 ? entry_target(kmer_entries, kmer_targets, h - 1) : -1;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (h + i >= total) break;
            const int32_t t = entry_target(kmer_entries, kmer_targets, h + i);
            falls += t < before;
            outside += t < 0 || t >= num_db;
            before = t;
        }
    }
    for (int64_t v = me; v < n_kmers; v += step) {
        const int64_t b = kmer_offsets[v], e = kmer_offsets[v + 1];
        if (b > 0 && b < e)
            starts += entry_target(kmer_entries, kmer_targets, b) < entry_target(kmer_entries, kmer_targets, b - 1);
        outside += b < 0 || b > e || e > total;
    }
    falls = __reduce_add_sync(0xffffffffu, falls);
    starts = __reduce_add_sync(0xffffffffu, starts);
    outside = __reduce_add_sync(0xffffffffu, outside);
    if ((threadIdx.x & 31) == 0) {
        if (falls) atomicAdd(order, (unsigned long long)falls);
        if (starts) atomicAdd(order + 1, (unsigned long long)starts);
        if (outside) atomicAdd(order + 2, (unsigned long long)outside);
    }
}
__device__ __forceinline__ bool lists_in_order(const unsigned long long *order) {
    return order[0] == order[1] && order[2] == 0;
}

// frag[r * n_kmers + v] = (first posting of v in range r, their number), by a
// binary search for each boundary; the lists of a warp's 32 5-mers lie side by
// side, so its searches share lines.  Lists that no walk reads stay empty.
__global__ void frag_kernel(const int64_t *__restrict__ kmer_offsets, const int64_t *__restrict__ kmer_entries,
                            const int32_t *__restrict__ kmer_targets, const int32_t *__restrict__ kmer_freqs,
                            int32_t freq_thresh, int32_t n_kmers, int32_t range, int32_t n_ranges,
                            const unsigned long long *__restrict__ order, uint2 *__restrict__ frag) {
    if (!lists_in_order(order)) return;
    const int32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n_kmers) return;
    const int32_t f = kmer_freqs[v];
    const int64_t b = kmer_offsets[v];
    const bool walked = f != 0 && f <= freq_thresh;
    const uint32_t end = (uint32_t)(walked ? kmer_offsets[v + 1] : b);
    uint32_t at = (uint32_t)b;
    for (int32_t r = 0; r < n_ranges; ++r) {
        uint32_t lo = at, hi = end;
        if (r + 1 == n_ranges) lo = hi;
        const int32_t bound = (r + 1) * range;  // at most 16 x 57,344
        while (lo < hi) {
            const uint32_t mid = lo + (hi - lo) / 2;
            if (entry_target(kmer_entries, kmer_targets, mid) < bound) lo = mid + 1; else hi = mid;
        }
        frag[(size_t)r * n_kmers + v] = make_uint2(at, lo - at);
        at = lo;
    }
}

// eight targets from a 32-byte boundary
__device__ __forceinline__ void load_targets(const int32_t *p, int32_t (&t)[8]) {
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7])
        : "l"(p));
}

__global__ void __launch_bounds__(NB_RW_THREADS, 1)
nbr_range_walk_kernel(const int32_t *__restrict__ n, const uint16_t *__restrict__ kmer,
                      const int32_t *__restrict__ weight, int32_t nq, int32_t n_blocks, int32_t block_kmers,
                      int32_t set_blocks, const uint2 *__restrict__ frag, const int64_t *__restrict__ kmer_offsets,
                      const int64_t *__restrict__ kmer_entries, const int32_t *__restrict__ kmer_targets,
                      int32_t num_db, int32_t range, int32_t n_ranges, const unsigned long long *__restrict__ order,
                      int32_t *__restrict__ counts, unsigned long long *__restrict__ ticket) {
    extern __shared__ int32_t acc[];
    __shared__ int32_t s_unit;
    if (!lists_in_order(order)) return;
    // eight targets a load where the compact index starts on a 32-byte boundary;
    // a load that would pass the index's end is not made as one
    const bool octets = kmer_targets && ((uintptr_t)kmer_targets & 31) == 0;
    const uint32_t total = (uint32_t)kmer_offsets[NB_KMERS];
    const int32_t sets = (n_blocks + set_blocks - 1) / set_blocks, units = n_ranges * sets * nq;
    for (int32_t i = threadIdx.x; i < range; i += NB_RW_THREADS) acc[i] = 0;
    for (;;) {
        if (threadIdx.x == 0) {
            const unsigned long long t = atomicAdd(ticket, 1ull);
            s_unit = t < (unsigned long long)units ? (int32_t)t : -1;
        }
        __syncthreads();
        const int32_t u = s_unit;
        if (u < 0) break;  // the same for the whole block
        const int32_t r = u / (sets * nq), set = u / nq % sets, q = u % nq;
        const int32_t t0 = r * range, nt = num_db - t0 < range ? num_db - t0 : range;
        int32_t *mine = acc - t0;  // only ever indexed by targets of the range
        const int32_t b1 = (set + 1) * set_blocks < n_blocks ? (set + 1) * set_blocks : n_blocks;
        for (int32_t b = set * set_blocks; b < b1; ++b) {
            const int32_t region = q * n_blocks + b, size = n[region];
            const uint16_t *ks = kmer + (size_t)region * NB_REGION;
            const int32_t *ws = weight + (size_t)region * NB_REGION;
            const uint2 *fr = frag + (size_t)r * NB_KMERS + b * block_kmers;
            int32_t c = threadIdx.x;
            uint32_t v_next = c + NB_RW_THREADS < size ? __ldg(ks + c + NB_RW_THREADS) : 0u;
            uint2 f = c < size ? __ldg(fr + __ldg(ks + c)) : make_uint2(0u, 0u);
            int32_t w = c < size ? __ldg(ws + c) : 0;
            for (; c < size; c += NB_RW_THREADS) {
                const uint2 part = f;
                const int32_t score = w;
                if (c + NB_RW_THREADS < size) {
                    f = __ldg(fr + v_next);
                    w = __ldg(ws + c + NB_RW_THREADS);
                    if (c + 2 * NB_RW_THREADS < size) v_next = __ldg(ks + c + 2 * NB_RW_THREADS);
                }
                if (part.y == 0) continue;
                const uint32_t end = part.x + part.y;
                if (octets && ((end + 7) & ~7u) <= total) {
                    for (uint32_t h = part.x & ~7u; h < end; h += 16) {
                        int32_t t[8], t2[8];
                        const bool two = h + 8 < end;
                        load_targets(kmer_targets + h, t);
                        if (two) load_targets(kmer_targets + h + 8, t2);
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            if (h + i - part.x < part.y) atomicAdd(&mine[t[i]], score);
                        if (two) {
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                if (h + 8 + i < end) atomicAdd(&mine[t2[i]], score);
                        }
                    }
                } else {
                    for (uint32_t h = part.x; h < end; ++h)
                        atomicAdd(&mine[entry_target(kmer_entries, kmer_targets, h)], score);
                }
            }
        }
        __syncthreads();
        // the counters go to the query's row and are zero again for the next unit
        int32_t *row = counts + (int64_t)q * num_db + t0;
        for (int32_t i = threadIdx.x; i < nt; i += NB_RW_THREADS) {
            const int32_t x = acc[i];
            if (x) { atomicAdd(&row[i], x); acc[i] = 0; }
        }
        __syncthreads();  // also: every thread has read s_unit before it is written again
    }
}

// ----------------------------------------------------------------- Phase B
// clustkit's C scorer (csrc/kmer_score.c:195-415): after Phase A the top
// phase_a_topk targets by (count desc, id asc) are rescored by their hits'
// diagonals -- per target the longest run of hits in one diagonal bin
// (tpos - qpos + qlen) / diag_bin_width, the first such bin on ties -- and
// kept when that run reaches min_diag_hits, with the diagonal hint
// bin * width - qlen + width / 2.  Here every selected target owns a dense
// row of bin counters (its bins: (qlen + tlen) / width + 1), found through a
// per-query target -> selection-index row.
__global__ void pb_mark_kernel(const int32_t *__restrict__ sel, const int32_t *__restrict__ sel_n, int32_t topk,
                               const int32_t *__restrict__ db_len, const int32_t *__restrict__ qlen, int32_t width,
                               int32_t num_db, int32_t *__restrict__ idx_row, int64_t *__restrict__ nbins) {
    const int32_t q = blockIdx.y;
    const int32_t n = sel_n[q];
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < topk; i += gridDim.x * blockDim.x) {
        int64_t nb = 0;
        if (i < n) {
            const int32_t t = sel[(int64_t)q * topk + i];
            idx_row[(int64_t)q * num_db + t] = i;
            nb = (int64_t)(qlen[q] + db_len[t]) / width + 1;
        }
        nbins[(int64_t)q * topk + i] = nb;
    }
}

__global__ void pb_bin_count_kernel(const uint8_t *__restrict__ qflat, int64_t qflat_len,
                                    const int64_t *__restrict__ qoff, const int32_t *__restrict__ qlen, int32_t k,
                                    int32_t alpha, const int64_t *__restrict__ kmer_offsets,
                                    const int64_t *__restrict__ kmer_entries, const int32_t *__restrict__ kmer_freqs,
                                    int32_t freq_thresh, int32_t num_db, const int32_t *__restrict__ idx_row,
                                    int32_t topk, const int64_t *__restrict__ base, int32_t width,
                                    int32_t *__restrict__ bins, int64_t bins_cap, int32_t *err) {
    const int32_t q = blockIdx.y;
    const int lane = threadIdx.x & 31;
    const int32_t L = qlen[q];
    const int64_t o = qoff[q];
    if (L < 0 || o < 0 || o + L > qflat_len) {
        if (threadIdx.x == 0 && blockIdx.x == 0) atomicOr(err, ERRBIT_SEQ_EXTENT);
        return;
    }
    const uint8_t *s = qflat + o;
    const int32_t *ix = idx_row + (int64_t)q * num_db;
    const int64_t *bq = base + (int64_t)q * topk;
    const int32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (int32_t p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p <= L - k; p += warps) {
        uint32_t v = 0;
        bool ok = true;
        for (int32_t m = 0; m < k; ++m) {
            const uint32_t r = s[p + m];
            ok &= r < (uint32_t)alpha;
            v = v * (uint32_t)alpha + r;
        }
        if (!ok || kmer_freqs[v] > freq_thresh) continue;
        const int64_t b = kmer_offsets[v], e = kmer_offsets[v + 1];
        for (int64_t h = b + lane; h < e; h += 32) {
            const int64_t entry = kmer_entries[h];
            const int32_t t = (int32_t)(entry >> 32);
            if (t < 0 || t >= num_db) { atomicOr(err, ERRBIT_PAIR_INDEX); continue; }
            const int32_t i = ix[t];
            if (i < 0) continue;
            const int64_t dbin = ((int64_t)(int32_t)(entry & 0xffffffff) - p + L) / width;
            const int64_t at = bq[i] + dbin;
            if (dbin < 0 || at >= bq[i + 1]) { atomicOr(err, ERRBIT_SEQ_EXTENT); continue; }
            if (at >= bins_cap) { atomicOr(err, ERRBIT_CAPACITY); continue; }
            atomicAdd(&bins[at], 1);
        }
    }
}

// A warp per selected target: its longest run (first bin on ties); kept ones
// are written into the (cleared) count row and listed for the final selection.
// The bins it reads are reset to zero, so a kept-zero bin buffer needs no
// clearing before the next call.
__global__ void pb_best_kernel(const int32_t *__restrict__ sel, const int32_t *__restrict__ sel_n, int32_t topk,
                               const int64_t *__restrict__ base, int32_t *__restrict__ bins, int64_t bins_cap,
                               const int32_t *__restrict__ qlen, int32_t width, int32_t min_diag_hits,
                               int32_t num_db, int32_t *__restrict__ counts, int32_t *__restrict__ hint_sel,
                               int32_t *__restrict__ cand, int32_t *__restrict__ n_cand) {
    const int32_t q = blockIdx.y;
    const int lane = threadIdx.x & 31;
    const int32_t n = sel_n[q];
    const int32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (int32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
        const int64_t b0 = base[(int64_t)q * topk + i];
        const int64_t b1 = min(base[(int64_t)q * topk + i + 1], bins_cap);
        int32_t best = 0, first = INT32_MAX;
        for (int64_t x = b0 + lane; x < b1; x += 32) {
            const int32_t c = bins[x];
            if (c) bins[x] = 0;
            if (c > best) { best = c; first = (int32_t)(x - b0); }
        }
        const int32_t m = __reduce_max_sync(0xffffffffu, best);
        const int32_t fb = __reduce_min_sync(0xffffffffu, (best == m && m > 0) ? first : INT32_MAX);
        if (lane == 0 && m >= min_diag_hits && m > 0) {
            const int32_t t = sel[(int64_t)q * topk + i];
            counts[(int64_t)q * num_db + t] = m;
            hint_sel[(int64_t)q * topk + i] = fb * width - qlen[q] + width / 2;
            const int32_t at = atomicAdd(&n_cand[q], 1);
            if (at < CAND_CAP) cand[(int64_t)q * CAND_CAP + at] = t;
        }
    }
}

__global__ void pb_hints_kernel(const int32_t *__restrict__ out_t, const int32_t *__restrict__ out_n, int32_t mc,
                                const int32_t *__restrict__ idx_row, int32_t num_db,
                                const int32_t *__restrict__ hint_sel, int32_t topk, int32_t *__restrict__ out_d) {
    const int32_t q = blockIdx.y;
    for (int32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < out_n[q]; j += gridDim.x * blockDim.x) {
        const int32_t t = out_t[(int64_t)q * mc + j];
        const int32_t i = idx_row[(int64_t)q * num_db + t];
        out_d[(int64_t)q * mc + j] = i >= 0 ? hint_sel[(int64_t)q * topk + i] : 0;
    }
}

struct PhaseAArgs {
    const int8_t *sub_host; int32_t score_thresh;  // similar k-mers when sub_host != nullptr
    const uint8_t *qflat; int64_t qflat_len; const int64_t *qoff; const int32_t *qlen; int32_t nq; int32_t max_qlen;
    int32_t k, alpha; const int64_t *kmer_offsets; const int64_t *kmer_entries; const int32_t *kmer_targets;
    const int32_t *kmer_freqs; int32_t freq_thresh; int32_t num_db; int32_t min_hits; int32_t top_k;
    int32_t *out_targets; int32_t *out_scores; int32_t *out_n; cudaStream_t st;
    bool ordered = true;  // capped rows in (score desc, id asc) order, not only the set
    int64_t list_capacity = -1;  // similar k-mers: caller's bound on (position, 5-mer) pairs, < 0 none
};

// The select, then the order of rows capped above CAND_CAP.  `ordered`:
// the rows are a call's output (without it only the set matters, as for the
// Phase-B selection); their scores go to a scratch row when the caller
// takes none.
static int32_t select_rows(const int32_t *counts, int32_t nq, int32_t num_db, int32_t min_hits, int32_t top_k,
                           int32_t clamp, int32_t top_shift, const int32_t *cand, const int32_t *n_cand,
                           int32_t *out_t, int32_t *out_s, int32_t *out_n, bool ordered, cudaStream_t st) {
    int32_t status = CK_OK;
    if (nq <= 0) return CK_OK;
    const bool sort = top_k > CAND_CAP && ordered;
    int32_t *aux = nullptr;
    if (sort) {
        if ((int64_t)nq * top_k >= INT32_MAX) {
            set_error(CK_ERR_UNSUPPORTED, "search select: nq * top_k must stay below 2^31");
            return CK_ERR_UNSUPPORTED;
        }
        aux = (int32_t *)scratch(SLOT_SEARCH_TMP3, (size_t)nq * 12, &status);
        if (!aux) return status;
        if (!out_s) {
            out_s = (int32_t *)scratch(SLOT_SEARCH_SCORES, (size_t)nq * top_k * 4, &status);
            if (!out_s) return status;
        }
    }
    // queries selected from their whole row: the row_* kernels
    const size_t rs_ints = (size_t)nq * (4 + 256 + 1 + 4 * ROW_SLOTS);
    int32_t *rs = (int32_t *)scratch(SLOT_SEARCH_ROWSEL, rs_ints * 4, &status);
    if (!rs) return status;
    int32_t *state = rs, *ghist = rs + 4 * (size_t)nq, *done = ghist + 256 * (size_t)nq;
    int32_t *wcnt = done + (size_t)nq, *woff = wcnt + 2 * (size_t)ROW_SLOTS * nq;
    CK_CUDA(cudaMemsetAsync(ghist, 0, (size_t)nq * 257 * 4, st));  // histograms and block counters
    const int64_t slice = ((int64_t)num_db + ROW_SLOTS - 1) / ROW_SLOTS;
    const int32_t W = (int32_t)std::max<int64_t>(32, (slice + 31) / 32 * 32);
    const dim3 rg((unsigned)ROW_BLOCKS, (unsigned)nq);
    for (int shift = top_shift; shift >= 0; shift -= 8) {
        // the digits already fixed: bits shift + 8 .. top_shift + 7
        const uint32_t mask = (uint32_t)((((uint64_t)1 << (top_shift + 8)) - 1) & ~(((uint64_t)1 << (shift + 8)) - 1));
        row_hist_kernel<<<rg, ROW_THREADS, 0, st>>>(counts, num_db, min_hits, clamp, shift, mask,
                                                    shift == top_shift, shift == 0, n_cand, top_k, state, ghist,
                                                    done, W);
        CK_CUDA(cudaGetLastError());
    }
    row_count_kernel<<<rg, ROW_THREADS, 0, st>>>(counts, num_db, min_hits, clamp, state, W, wcnt);
    CK_CUDA(cudaGetLastError());
    row_offsets_kernel<<<nq, ROW_SLOTS, 0, st>>>(state, wcnt, top_k, woff, out_n, aux);
    CK_CUDA(cudaGetLastError());
    row_write_kernel<<<rg, ROW_THREADS, 0, st>>>(counts, num_db, min_hits, clamp, state, W, woff, top_k, out_t, out_s);
    CK_CUDA(cudaGetLastError());
    row_sort_kernel<<<nq, SELECT_THREADS, 0, st>>>(counts, num_db, clamp, state, top_k, out_t, out_s);
    CK_CUDA(cudaGetLastError());
    // queries whose candidate lists hold all their survivors
    phase_a_select_kernel<<<nq, SELECT_THREADS, 0, st>>>(counts, num_db, min_hits, top_k, clamp, top_shift, cand,
                                                         n_cand, out_t, out_s, out_n, aux);
    CK_CUDA(cudaGetLastError());
    if (!sort) return CK_OK;
    const size_t items = (size_t)nq * top_k;
    uint64_t *k0 = (uint64_t *)scratch(SLOT_SORT_KEYS, items * 8, &status);
    uint64_t *k1 = (uint64_t *)scratch(SLOT_SORT_KEYS_ALT, items * 8, &status);
    if (!k0 || !k1) return status;
    int32_t *beg = aux + nq, *end = aux + 2 * (size_t)nq;
    const dim3 g((unsigned)std::min(64, (top_k + 255) / 256), (unsigned)nq);
    cap_keys_kernel<<<g, 256, 0, st>>>(out_t, out_s, aux, top_k, k0, beg, end);
    CK_CUDA(cudaGetLastError());
    size_t tb = 0;
    CK_CUDA(cub::DeviceSegmentedSort::SortKeys(nullptr, tb, k0, k1, (int)items, nq, beg, end, st));
    void *tmp = scratch(SLOT_SORT_TEMP, tb, &status);
    if (!tmp) return status;
    CK_CUDA(cub::DeviceSegmentedSort::SortKeys(tmp, tb, k0, k1, (int)items, nq, beg, end, st));
    cap_unpack_kernel<<<g, 256, 0, st>>>(k1, aux, top_k, out_t, out_s);
    CK_CUDA(cudaGetLastError());
    return CK_OK;
}

// Error when a bounded call's pairs of query position and 5-mer pass its bound.
__global__ void nbr_bound_kernel(const unsigned long long *__restrict__ listed, int64_t cap, int32_t *err) {
    if (threadIdx.x == 0 && blockIdx.x == 0 && *listed > (unsigned long long)cap) atomicOr(err, ERRBIT_LIST);
}

// Similar k-mers: the weights of NB_QUERIES queries at a time, and their walk.
static int32_t similar_weights_and_walk(const PhaseAArgs &a, const int8_t *d_sub, int32_t *counts, int32_t *err) {
    int32_t status = CK_OK;
    int32_t smin = a.sub_host[0], smax = a.sub_host[0];
    for (int i = 1; i < 400; ++i) {
        smin = std::min<int32_t>(smin, a.sub_host[i]);
        smax = std::max<int32_t>(smax, a.sub_host[i]);
    }
    const int32_t srange = smax - smin, bins = 2 * srange + 1;
    constexpr size_t SMEM = 227 * 1024 - 256;  // a block's most, less its static part
    const int32_t prefixes = nbr_smem(NB_PREFIXES, srange) <= SMEM ? NB_PREFIXES : NB_PREFIXES - 1;
    const size_t smem = nbr_smem(prefixes, srange);
    const int32_t n_blocks = (NB_PAIRS + prefixes - 1) / prefixes, block_kmers = prefixes * 8000;
    const int32_t chunk = std::min(a.nq, NB_QUERIES);
    const size_t regions = (size_t)chunk * n_blocks;
    // totals and tickets (8-byte words), then each region's count and first run
    unsigned long long *words = (unsigned long long *)scratch(SLOT_SEARCH_TMP0, 8 * 8 + (2 * regions + 1) * 4, &status);
    if (!words) return status;
    unsigned long long *listed = words, *ticket = words + 1, *ticket2 = words + 2, *order = words + 4;
    int32_t *n = (int32_t *)(words + 8), *run0 = n + regions;
    // the bits of indexed 5-mers and the ordered residue pairs
    uint32_t *valid = (uint32_t *)scratch(SLOT_SEARCH_TMP2, ((size_t)2 * NB_VALID + (size_t)NB_PAIRS * bins) * 4, &status);
    if (!valid) return status;
    uint32_t *ordered = valid + NB_VALID;
    int32_t *from = (int32_t *)(ordered + NB_VALID);
    int32_t *weight = (int32_t *)scratch(SLOT_SEARCH_TMP1, regions * NB_REGION * 6, &status);
    if (!weight) return status;
    uint16_t *kmer = (uint16_t *)(weight + regions * NB_REGION);
    // by target ranges: several queries, on a database of at most NB_MAX_RANGES ranges
    int32_t n_ranges = (int32_t)(((int64_t)a.num_db + NB_RANGE - 1) / NB_RANGE), range = 0;
    uint2 *frag = nullptr;
    if (a.nq >= NB_RANGE_MIN_QUERIES && n_ranges >= 1 && n_ranges <= NB_MAX_RANGES) {
        range = (a.num_db + n_ranges - 1) / n_ranges;
        frag = (uint2 *)scratch(SLOT_SEARCH_TMP4, (size_t)n_ranges * NB_KMERS * 8, &status);
        if (!frag) return status;
    } else {
        n_ranges = 0;
    }
    CK_CUDA(cudaFuncSetAttribute(nbr_weight_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    CK_CUDA(cudaMemsetAsync(words, 0, 8 * 8, a.st));
    kmer_valid_kernel<<<NB_VALID / 256, 256, 0, a.st>>>(a.kmer_freqs, a.freq_thresh, valid);
    CK_CUDA(cudaGetLastError());
    nbr_tables_kernel<<<NB_PAIRS, 32, 0, a.st>>>(d_sub, smin, bins, ordered, from);
    CK_CUDA(cudaGetLastError());
    if (n_ranges > 0) {
        order_kernel<<<sm_count() * 8, 256, 0, a.st>>>(a.kmer_offsets, a.kmer_entries, a.kmer_targets, NB_KMERS,
                                                       a.num_db, nbr_least_postings(n_ranges, a.num_db, a.nq), order);
        CK_CUDA(cudaGetLastError());
        frag_kernel<<<(NB_KMERS + 255) / 256, 256, 0, a.st>>>(a.kmer_offsets, a.kmer_entries, a.kmer_targets,
                                                              a.kmer_freqs, a.freq_thresh, NB_KMERS, range, n_ranges,
                                                              order, frag);
        CK_CUDA(cudaGetLastError());
        CK_CUDA(cudaFuncSetAttribute(nbr_range_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, NB_RANGE * 4));
    }
    for (int32_t q0 = 0; q0 < a.nq; q0 += chunk) {
        const int32_t nq = std::min(chunk, a.nq - q0);
        const int32_t nr = nq * n_blocks;
        int32_t *rows = counts + (size_t)q0 * a.num_db;
        if (q0 > 0) CK_CUDA(cudaMemsetAsync(ticket, 0, 16, a.st));
        nbr_weight_kernel<<<dim3((unsigned)n_blocks, (unsigned)nq), NB_WARPS * 32, smem, a.st>>>(
            a.qflat, a.qflat_len, a.qoff + q0, a.qlen + q0, d_sub, smin, srange, a.score_thresh, valid, ordered, from,
            prefixes, n, kmer, weight, listed, err);
        CK_CUDA(cudaGetLastError());
        if (n_ranges > 0) {
            // about 12 units an SM, of at least one block of 5-mers, at most an
            // eighth of them (their cuts and postings have to stay in L2)
            const int32_t want = std::max(8, std::min(n_blocks, 12 * sm_count() / (nq * n_ranges)));
            const int32_t set_blocks = (n_blocks + want - 1) / want;
            nbr_range_walk_kernel<<<sm_count(), NB_RW_THREADS, (size_t)range * 4, a.st>>>(
                n, kmer, weight, nq, n_blocks, block_kmers, set_blocks, frag, a.kmer_offsets, a.kmer_entries,
                a.kmer_targets, a.num_db, range, n_ranges, order, rows, ticket2);
            CK_CUDA(cudaGetLastError());
        }
        nbr_runs_kernel<<<1, 1024, 0, a.st>>>(n, nr, run0);
        CK_CUDA(cudaGetLastError());
        // one resident block per slot (8 of 256 threads per SM)
        nbr_walk_kernel<<<8 * sm_count(), 256, 0, a.st>>>(n, run0, kmer, weight, nr, n_blocks, block_kmers,
                                                          a.kmer_offsets, a.kmer_entries, a.kmer_targets, a.num_db,
                                                          rows, ticket, n_ranges > 0 ? order : nullptr, err);
        CK_CUDA(cudaGetLastError());
    }
    if (a.list_capacity >= 0) {
        nbr_bound_kernel<<<1, 32, 0, a.st>>>(listed, a.list_capacity, err);
        CK_CUDA(cudaGetLastError());
    }
    return CK_OK;
}

static int32_t phase_a_impl(void *pv) {
    PhaseAArgs &a = *(PhaseAArgs *)pv;
    int32_t status = CK_OK;
    int32_t *err = device_error_word(&status);
    if (!err) return status;
    if (a.nq == 0) return CK_OK;
    const size_t nc = (size_t)a.nq * (size_t)a.num_db;
    int32_t *counts = (int32_t *)scratch(SLOT_SEARCH_COUNTS, nc * 4 + 4, &status);
    if (!counts) return status;
    int32_t *cand = (int32_t *)scratch(SLOT_SEARCH_CAND, (size_t)a.nq * (CAND_CAP + 1) * 4, &status);
    if (!cand) return status;
    int32_t *n_cand = cand + (size_t)a.nq * CAND_CAP;
    CK_CUDA(cudaMemsetAsync(counts, 0, nc * 4, a.st));
    CK_CUDA(cudaMemsetAsync(n_cand, 0, (size_t)a.nq * 4, a.st));
    const int32_t npos = a.max_qlen - a.k + 1;
    int32_t clamp = 32767, top_shift = 8;  // clustkit's int16 hit counters
    if (!a.sub_host) {
        if (npos > 0) {
            int bx = (npos + 7) / 8;  // 8 warps per block
            if (bx > 16) bx = 16;
            dim3 grid((unsigned)bx, (unsigned)a.nq);
            phase_a_count_kernel<<<grid, 256, 0, a.st>>>(a.qflat, a.qflat_len, a.qoff, a.qlen, a.k, a.alpha,
                                                          a.kmer_offsets, a.kmer_entries, a.kmer_targets,
                                                          a.kmer_freqs,
                                                          a.freq_thresh, a.num_db, counts, a.min_hits, cand,
                                                          n_cand, err);
            CK_CUDA(cudaGetLastError());
        }
    } else {
        clamp = INT32_MAX;  // score-weighted int32 sums
        top_shift = 24;
        const int8_t *d_sub = device_sub_matrix(a.sub_host, &status);
        if (!d_sub) return status;
        if (npos > 0) {
            CK_TRY(similar_weights_and_walk(a, d_sub, counts, err));
            // the select scans the whole count row (no candidate list in this mode)
            fill_kernel<<<1, 256, 0, a.st>>>(n_cand, a.nq, CAND_CAP + 1);
            CK_CUDA(cudaGetLastError());
        }
    }
    return select_rows(counts, a.nq, a.num_db, a.min_hits, a.top_k, clamp, top_shift, cand, n_cand,
                       a.out_targets, a.out_scores, a.out_n, a.ordered, a.st);
}

}  // namespace ck

using namespace ck;

extern "C" int32_t ck_kmer_index_build_device(int32_t ctx, const uint8_t *d_flat, int64_t flat_len,
                                              const int64_t *d_offsets, const int32_t *d_lengths,
                                              int64_t n_seqs, int32_t k, int32_t alpha,
                                              int64_t *d_kmer_offsets, int64_t *d_kmer_entries,
                                              int64_t entries_capacity, int32_t *d_kmer_freqs,
                                              int64_t *out_total, void *stream) {
    std::lock_guard<std::mutex> lock(library_mutex());
    reset_thread_status();
    int64_t nk = 1;
    for (int32_t i = 0; i < k && nk < ((int64_t)1 << 31); ++i) nk *= (alpha > 0 ? alpha : 1);
    if (k < 1 || alpha < 1 || nk >= ((int64_t)1 << 31) || n_seqs < 0 || flat_len < 0 || !out_total ||
        !d_kmer_offsets || !d_kmer_freqs || (n_seqs > 0 && (!d_offsets || !d_lengths))) {
        set_error(CK_ERR_INVALID_ARGUMENT, "kmer index: bad arguments (need alpha^k < 2^31)");
        return CK_ERR_INVALID_ARGUMENT;
    }
    IndexBuildArgs a{d_flat, flat_len, d_offsets, d_lengths, n_seqs, k, alpha, d_kmer_offsets,
                     d_kmer_entries, entries_capacity, d_kmer_freqs, out_total, (cudaStream_t)stream};
    return run_in_context(ctx, index_build_impl, &a);
}

extern "C" int32_t ck_kmer_targets_device(int32_t ctx, const int64_t *d_kmer_entries, int64_t n_entries,
                                          int32_t *d_kmer_targets, void *stream) {
    std::lock_guard<std::mutex> lock(library_mutex());
    reset_thread_status();
    if (n_entries < 0 || (n_entries > 0 && (!d_kmer_entries || !d_kmer_targets))) {
        set_error(CK_ERR_INVALID_ARGUMENT, "kmer targets: bad arguments");
        return CK_ERR_INVALID_ARGUMENT;
    }
    struct Args { const int64_t *e; int64_t n; int32_t *t; cudaStream_t st; } a{d_kmer_entries, n_entries,
                                                                                 d_kmer_targets, (cudaStream_t)stream};
    return run_in_context(ctx, [](void *pv) -> int32_t {
        const Args &a = *(const Args *)pv;
        if (a.n == 0) return CK_OK;
        compact_targets_kernel<<<grid_for(a.n, 256), 256, 0, a.st>>>(a.e, a.n, a.t);
        CK_CUDA(cudaGetLastError());
        return CK_OK;
    }, &a);
}

extern "C" int32_t ck_search_pairs_device(int32_t nq, int32_t max_cands, int32_t seq0, int32_t empty_idx,
                                          const int32_t *d_n, const int32_t *d_targets, int32_t *d_pairs,
                                          void *stream) {
    std::lock_guard<std::mutex> lock(library_mutex());
    reset_thread_status();
    if (nq < 0 || max_cands < 0 || (nq > 0 && max_cands > 0 && (!d_n || !d_targets || !d_pairs))) {
        set_error(CK_ERR_INVALID_ARGUMENT, "search pairs: bad arguments");
        return CK_ERR_INVALID_ARGUMENT;
    }
    const int64_t M = (int64_t)nq * max_cands;
    if (M == 0) return CK_OK;
    search_pairs_kernel<<<grid_for(M, 256), 256, 0, (cudaStream_t)stream>>>(nq, max_cands, seq0, empty_idx, d_n,
                                                                             d_targets, (int2 *)d_pairs);
    CK_CUDA(cudaGetLastError());
    return CK_OK;
}

extern "C" int32_t ck_search_phase_a_device(int32_t ctx, const uint8_t *d_qflat, int64_t qflat_len,
                                            const int64_t *d_qoffsets,
                                            const int32_t *d_qlengths, int32_t nq, int32_t max_qlen,
                                            int32_t k, int32_t alpha, const int64_t *d_kmer_offsets,
                                            const int64_t *d_kmer_entries, const int32_t *d_kmer_targets,
                                            const int32_t *d_kmer_freqs, int32_t freq_thresh, int32_t num_db,
                                            int32_t min_total_hits, int32_t top_k, int32_t *d_out_targets,
                                            int32_t *d_out_scores, int32_t *d_out_n, void *stream) {
    std::lock_guard<std::mutex> lock(library_mutex());
    reset_thread_status();
    if (nq < 0 || nq > 65535 || qflat_len < 0 || top_k < 1 || k < 1 || alpha < 1 || num_db < 0 || !d_out_targets || !d_out_n ||
        (nq > 0 && (!d_qflat || !d_qoffsets || !d_qlengths)) || !d_kmer_offsets || !d_kmer_freqs ||
        (!d_kmer_entries && !d_kmer_targets)) {
        set_error(CK_ERR_INVALID_ARGUMENT, "phase A: bad arguments");
        return CK_ERR_INVALID_ARGUMENT;
    }
    PhaseAArgs a{nullptr, 0, d_qflat, qflat_len, d_qoffsets, d_qlengths, nq, max_qlen, k, alpha, d_kmer_offsets, d_kmer_entries,
                 d_kmer_targets, d_kmer_freqs, freq_thresh, num_db, min_total_hits, top_k, d_out_targets, d_out_scores,
                 d_out_n, (cudaStream_t)stream};
    return run_in_context(ctx, phase_a_impl, &a);
}

extern "C" int32_t ck_search_phase_a_similar_device(int32_t ctx, const uint8_t *d_qflat, int64_t qflat_len,
                                                    const int64_t *d_qoffsets, const int32_t *d_qlengths,
                                                    int32_t nq, int32_t max_qlen, const int8_t *sub_matrix_host,
                                                    int32_t kmer_score_thresh, const int64_t *d_kmer_offsets,
                                                    const int64_t *d_kmer_entries, const int32_t *d_kmer_targets,
                                                    const int32_t *d_kmer_freqs, int32_t freq_thresh, int32_t num_db,
                                                    int32_t min_total_hits, int32_t top_k, int32_t *d_out_targets,
                                                    int32_t *d_out_scores, int32_t *d_out_n, int64_t list_capacity,
                                                    void *stream) {
    std::lock_guard<std::mutex> lock(library_mutex());
    reset_thread_status();
    if (nq < 0 || nq > 65535 || qflat_len < 0 || top_k < 1 || num_db < 0 || !sub_matrix_host ||
        kmer_score_thresh < 1 || !d_out_targets || !d_out_n || (nq > 0 && (!d_qflat || !d_qoffsets || !d_qlengths)) ||
        !d_kmer_offsets || !d_kmer_freqs || (!d_kmer_entries && !d_kmer_targets)) {
        set_error(CK_ERR_INVALID_ARGUMENT, "similar k-mer phase A: bad arguments");
        return CK_ERR_INVALID_ARGUMENT;
    }
    PhaseAArgs a{sub_matrix_host, kmer_score_thresh, d_qflat, qflat_len, d_qoffsets, d_qlengths, nq, max_qlen, 5,
                 20, d_kmer_offsets, d_kmer_entries, d_kmer_targets, d_kmer_freqs, freq_thresh, num_db,
                 min_total_hits, top_k, d_out_targets, d_out_scores, d_out_n, (cudaStream_t)stream};
    a.list_capacity = list_capacity;
    return run_in_context(ctx, phase_a_impl, &a);
}

namespace ck {

struct CandArgs {
    PhaseAArgs a;  // Phase A part (sub_host null); top_k there = max_cands
    const int32_t *db_len; int32_t min_diag_hits, width, phase_a_topk; int32_t *out_diags;
    int64_t bins_capacity;  // >= 0: the caller's bound on the bins (no host sync); < 0: sized from the scan
};

static int32_t candidates_impl(void *pv) {
    CandArgs &c = *(CandArgs *)pv;
    PhaseAArgs &a = c.a;
    int32_t status = CK_OK;
    const size_t nq = (size_t)a.nq;
    if (c.min_diag_hits <= 1) {  // Phase A and the cap, hints zero
        CK_TRY(phase_a_impl(&a));
        if (c.out_diags && a.nq > 0) CK_CUDA(cudaMemsetAsync(c.out_diags, 0, nq * a.top_k * 4, a.st));
        return CK_OK;
    }
    int32_t *err = device_error_word(&status);
    if (!err) return status;
    if (a.nq == 0) return CK_OK;
    const int32_t topk = c.phase_a_topk;
    // Phase A with the Phase-B top-K as its cap, into the selection buffers
    int32_t *sel = (int32_t *)scratch(SLOT_SEARCH_TMP2, nq * topk * 4 + nq * 4, &status);
    int64_t *base = (int64_t *)scratch(SLOT_SEARCH_TMP4, (nq * topk + 1) * 8, &status);
    int32_t *hint_sel = (int32_t *)scratch(SLOT_SEARCH_TMP0, nq * topk * 4, &status);
    int32_t *idx_row = (int32_t *)scratch(SLOT_SEARCH_IDX, nq * (size_t)a.num_db * 4 + 4, &status);
    if (!sel || !base || !hint_sel || !idx_row) return status;
    int32_t *sel_n = sel + nq * topk;
    PhaseAArgs a1 = a;
    a1.top_k = topk;
    a1.out_targets = sel;
    a1.out_scores = nullptr;
    a1.out_n = sel_n;
    a1.ordered = false;  // only the selected set matters
    CK_TRY(phase_a_impl(&a1));
    int32_t *counts = (int32_t *)scratch(SLOT_SEARCH_COUNTS, nq * (size_t)a.num_db * 4 + 4, &status);
    if (!counts) return status;
    CK_CUDA(cudaMemsetAsync(idx_row, 0xff, nq * (size_t)a.num_db * 4, a.st));
    const dim3 g1((unsigned)std::min(64, (topk + 255) / 256), (unsigned)a.nq);
    pb_mark_kernel<<<g1, 256, 0, a.st>>>(sel, sel_n, topk, c.db_len, a.qlen, c.width, a.num_db, idx_row, base);
    CK_CUDA(cudaGetLastError());
    // bin offsets: one exclusive scan over every (query, selected target); the
    // trailing entry is the total
    CK_CUDA(cudaMemsetAsync(base + nq * topk, 0, 8, a.st));
    size_t tb = 0;
    CK_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, base, base, (int64_t)(nq * topk + 1), a.st));
    void *tmp = scratch(SLOT_SORT_TEMP, tb, &status);
    if (!tmp) return status;
    CK_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, base, base, (int64_t)(nq * topk + 1), a.st));
    // the bins: a kept-zero buffer of the caller's bounded size (pb_best_kernel
    // resets what it reads; bins past the bound are skipped and flagged), or
    // sized from the scan's total read back here
    int64_t cap = c.bins_capacity;
    int32_t *bins = nullptr;
    if (cap >= 0) {
        bins = (int32_t *)scratch_zeroed(SLOT_SEARCH_BINS, (size_t)(cap > 0 ? cap : 1) * 4, a.st, &status);
    } else {
        CK_CUDA(cudaMemcpyAsync(&cap, base + nq * topk, 8, cudaMemcpyDeviceToHost, a.st));
        CK_CUDA(cudaStreamSynchronize(a.st));
        bins = (int32_t *)scratch(SLOT_SEARCH_TMP1, (size_t)(cap > 0 ? cap : 1) * 4, &status);
        if (bins && cap > 0) CK_CUDA(cudaMemsetAsync(bins, 0, (size_t)cap * 4, a.st));
    }
    if (!bins) return status;
    // from here to pb_best_kernel a failure leaves counts in the kept-zero buffer
    if (c.bins_capacity >= 0) scratch_mark_dirty(SLOT_SEARCH_BINS);
    const int32_t npos = a.max_qlen - a.k + 1;
    if (npos > 0) {
        int bx = (npos + 7) / 8;
        if (bx > 16) bx = 16;
        pb_bin_count_kernel<<<dim3((unsigned)bx, (unsigned)a.nq), 256, 0, a.st>>>(
            a.qflat, a.qflat_len, a.qoff, a.qlen, a.k, a.alpha, a.kmer_offsets, a.kmer_entries, a.kmer_freqs,
            a.freq_thresh, a.num_db, idx_row, topk, base, c.width, bins, cap, err);
        CK_CUDA(cudaGetLastError());
    }
    // final cap over the kept targets: from their list, or a scan of the row
    // when more than CAND_CAP were kept; runs are not clamped (int32 select)
    int32_t *cand = (int32_t *)scratch(SLOT_SEARCH_CAND, nq * (CAND_CAP + 1) * 4, &status);
    if (!cand) return status;
    int32_t *n_cand = cand + nq * CAND_CAP;
    CK_CUDA(cudaMemsetAsync(n_cand, 0, nq * 4, a.st));
    CK_CUDA(cudaMemsetAsync(counts, 0, nq * (size_t)a.num_db * 4, a.st));
    const dim3 g2((unsigned)std::min(64, (topk + 7) / 8), (unsigned)a.nq);
    pb_best_kernel<<<g2, 256, 0, a.st>>>(sel, sel_n, topk, base, bins, cap, a.qlen, c.width, c.min_diag_hits,
                                         a.num_db, counts, hint_sel, cand, n_cand);
    CK_CUDA(cudaGetLastError());
    if (c.bins_capacity >= 0) scratch_clear_dirty(SLOT_SEARCH_BINS);
    CK_TRY(select_rows(counts, a.nq, a.num_db, c.min_diag_hits, a.top_k, INT32_MAX, 24, cand, n_cand,
                       a.out_targets, a.out_scores, a.out_n, true, a.st));
    if (c.out_diags) {
        const dim3 g3((unsigned)std::min(64, (a.top_k + 255) / 256), (unsigned)a.nq);
        pb_hints_kernel<<<g3, 256, 0, a.st>>>(a.out_targets, a.out_n, a.top_k, idx_row, a.num_db, hint_sel, topk,
                                              c.out_diags);
        CK_CUDA(cudaGetLastError());
    }
    return CK_OK;
}

}  // namespace ck

extern "C" int32_t ck_search_kmer_candidates_device(
    int32_t ctx, const uint8_t *d_qflat, int64_t qflat_len, const int64_t *d_qoffsets, const int32_t *d_qlengths,
    int32_t nq, int32_t max_qlen, int32_t k, int32_t alpha, const int64_t *d_kmer_offsets,
    const int64_t *d_kmer_entries, const int32_t *d_kmer_targets, const int32_t *d_kmer_freqs, int32_t freq_thresh,
    int32_t num_db, const int32_t *d_db_lengths, int32_t min_total_hits, int32_t min_diag_hits,
    int32_t diag_bin_width, int32_t max_cands, int32_t phase_a_topk, int32_t *d_out_targets, int32_t *d_out_scores,
    int32_t *d_out_diags, int32_t *d_out_n, int64_t bins_capacity, void *stream) {
    std::lock_guard<std::mutex> lock(library_mutex());
    reset_thread_status();
    if (nq < 0 || nq > 65535 || qflat_len < 0 || max_cands < 1 || k < 1 || alpha < 1 || num_db < 0 ||
        !d_out_targets || !d_out_n || (nq > 0 && (!d_qflat || !d_qoffsets || !d_qlengths)) || !d_kmer_offsets ||
        !d_kmer_freqs || (!d_kmer_entries && !d_kmer_targets) ||
        (min_diag_hits >= 2 && (!d_kmer_entries || !d_db_lengths || diag_bin_width < 1 || phase_a_topk < 1))) {
        set_error(CK_ERR_INVALID_ARGUMENT, "k-mer candidates: bad arguments");
        return CK_ERR_INVALID_ARGUMENT;
    }
    CandArgs c{PhaseAArgs{nullptr, 0, d_qflat, qflat_len, d_qoffsets, d_qlengths, nq, max_qlen, k, alpha,
                          d_kmer_offsets, d_kmer_entries, d_kmer_targets, d_kmer_freqs, freq_thresh, num_db,
                          min_total_hits, max_cands, d_out_targets, d_out_scores, d_out_n, (cudaStream_t)stream},
               d_db_lengths, min_diag_hits, diag_bin_width, phase_a_topk, d_out_diags, bins_capacity};
    return run_in_context(ctx, candidates_impl, &c);
}
