// jaccard.cu -- merge-walk Jaccard of sorted MinHash sketches
// (clustkit/pairwise.py:1564-1612) and the pre-filter mask
// (clustkit/pairwise.py:949-1001).
//
// clustkit walks the two sorted sketches A and B with two heads: equal heads
// are one shared step that advances both, otherwise the smaller head
// advances; it stops after s steps or when both heads are UINT64_MAX, and
// J = shared / steps.  Here one warp evaluates a pair without walking: with
// A and B in shared memory, every element A[i] of value v knows
//   lowB = #B < v, cntB = #B == v, firstA = index of the first v in A,
// it is paired (consumed in the same step as a B element) iff
// v != MAX and i - firstA < cntB, and it is consumed at step
//   i + lowB - P(firstA),  P(x) = number of paired elements among A[0..x),
// because every step before it consumed either an A element before i, a B
// element below v, or both at once (a paired step).  The walk takes
// T = #nonMAX(A) + #nonMAX(B) - #pairs steps in all, so
//   steps  = min(s, T),  shared = #paired A elements consumed at step < s.
// J = shared / steps is the float32 rounding of the quotient, as clustkit's
// float32(shared / union) gives for these small integers.
#include "ck_common.cuh"

namespace ck {

__device__ __forceinline__ int lower_bound_u64(const uint64_t *a, int n, uint64_t v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (a[mid] < v) lo = mid + 1; else hi = mid;
    }
    return lo;
}
__device__ __forceinline__ int upper_bound_u64(const uint64_t *a, int n, uint64_t v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (a[mid] <= v) lo = mid + 1; else hi = mid;
    }
    return lo;
}

__global__ void jaccard_kernel(const int32_t *__restrict__ pairs, int64_t M,
                               const uint64_t *__restrict__ sk, int64_t N, int32_t s, float floor,
                               float *__restrict__ sims, uint8_t *__restrict__ mask, int32_t *err) {
    extern __shared__ uint64_t s_mem[];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    uint64_t *A = s_mem + (size_t)wib * (2 * s + s / 2 + 2);
    uint64_t *B = A + s;
    int32_t *P = (int32_t *)(B + s);  // s + 1 prefix counts
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const uint64_t MAXV = ~0ULL;

    for (int64_t p = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < M; p += warps) {
        const int32_t ia = pairs[2 * p], ib = pairs[2 * p + 1];
        if (ia < 0 || ib < 0 || ia >= N || ib >= N) {
            if (lane == 0) {
                atomicOr(err, ERRBIT_PAIR_INDEX);
                sims[p] = 0.0f;
                if (mask) mask[p] = 0;
            }
            continue;
        }
        const uint64_t *ga = sk + (int64_t)ia * s, *gb = sk + (int64_t)ib * s;
        for (int t = lane; t < s; t += 32) { A[t] = ga[t]; B[t] = gb[t]; }
        __syncwarp();
        // pass 1: paired flags -> exclusive prefix P over A
        int32_t run = 0;
        for (int base = 0; base < s; base += 32) {
            const int i = base + lane;
            int paired = 0;
            if (i < s) {
                const uint64_t v = A[i];
                if (v != MAXV) {
                    const int fa = lower_bound_u64(A, s, v);
                    const int lb = lower_bound_u64(B, s, v);
                    const int ub = upper_bound_u64(B, s, v);
                    paired = (i - fa) < (ub - lb);
                }
            }
            const unsigned bal = __ballot_sync(0xffffffffu, paired);
            if (i < s) P[i] = run + __popc(bal & ((1u << lane) - 1u));
            run += __popc(bal);
        }
        if (lane == 0) P[s] = run;
        __syncwarp();
        // pass 2: shared steps among the first s
        int32_t shared = 0;
        for (int i = lane; i < s; i += 32) {
            const uint64_t v = A[i];
            if (v == MAXV) continue;
            const int fa = lower_bound_u64(A, s, v);
            const int lb = lower_bound_u64(B, s, v);
            const int ub = upper_bound_u64(B, s, v);
            if ((i - fa) < (ub - lb)) {
                const int step = i + lb - P[fa];
                shared += step < s;
            }
        }
        for (int o = 16; o; o >>= 1) shared += __shfl_xor_sync(0xffffffffu, shared, o);
        if (lane == 0) {
            const int nA = lower_bound_u64(A, s, MAXV);
            const int nB = lower_bound_u64(B, s, MAXV);
            const int T = nA + nB - P[s];
            const int steps = T < s ? T : s;
            const float j = steps == 0 ? 0.0f : __fdiv_rn((float)shared, (float)steps);
            sims[p] = j;
            if (mask) mask[p] = j >= floor;
        }
        __syncwarp();
    }
}

// The same closed form from B's side, for s <= 32 E.  Copy m of a value v
// of B (m = j - first index of v in B) is paired iff A[lowA + m] == v with
// lowA = #A < v, and is consumed at step lowA + j - (r - m), r = paired
// elements of B before j.  Most pairs are chance collisions with few shared
// values, so B's elements -- held in registers, 32 k + lane -- are first tested
// against a bitmap of A's low bits (64 bits an element: 2 false hits a pair at
// s = 128), and only hits search A.  A and its bitmap stay in shared memory
// while consecutive pairs of the warp's run share their first sequence, as a
// sorted candidate list's do; the next pair's B is loaded while one is worked
// on.  A lane works through its own hits, so a chance pair costs one binary
// search.  Bound by issue (83 %).  4 M pairs of 100,000 sketches at s = 128:
// 2.92 ms with both sketches staged and every element searched, 1.39 with the
// bitmap and a search for each of a lane's elements, 1.01 now.
constexpr int JACCARD_RUN = 32;  // pairs a warp takes at most (one per lane to load and to write)

template <int E>
__global__ void __launch_bounds__(256)
jaccard_bitmap_kernel(const int32_t *__restrict__ pairs, int64_t M, const uint64_t *__restrict__ sk, int64_t N,
                      int32_t s, int32_t run, float floor, float *__restrict__ sims, uint8_t *__restrict__ mask,
                      int32_t *err) {
    constexpr uint32_t FULL = 0xffffffffu;
    constexpr int WORDS = 64 * E;  // bitmap words: 64 bits for each of 32 E elements
    constexpr uint32_t BITS = 32u * WORDS;
    extern __shared__ uint64_t s_mem[];
    const int lane = threadIdx.x & 31;
    uint64_t *A = s_mem + (size_t)(threadIdx.x >> 5) * (32 * E + WORDS / 2);
    uint32_t *bm = (uint32_t *)(A + 32 * E);
    const uint64_t MAXV = ~0ULL;
    const int64_t p0 = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * run;
    if (p0 >= M) return;
    const int32_t np = M - p0 < run ? (int32_t)(M - p0) : run;

    int32_t ia = -1, ib = -1;
    if (lane < np) { ia = pairs[2 * (p0 + lane)]; ib = pairs[2 * (p0 + lane) + 1]; }
    const bool ok = ia >= 0 && ib >= 0 && ia < N && ib < N;
    if (lane < np && !ok) atomicOr(err, ERRBIT_PAIR_INDEX);
    const uint32_t okb = __ballot_sync(FULL, ok);

    auto load = [&](int32_t i, uint64_t (&v)[E]) {
        const uint64_t *g = sk + (int64_t)i * s;
#pragma unroll
        for (int k = 0; k < E; ++k) v[k] = 32 * k + lane < s ? __ldg(g + 32 * k + lane) : MAXV;
    };
    uint64_t nxt[E];
    if (okb) load(__shfl_sync(FULL, ib, __ffs(okb) - 1), nxt);
    float sim = 0.0f;  // of pair p0 + lane
    int32_t held = -1, n_a = 0;
    for (uint32_t todo = okb; todo; todo &= todo - 1) {
        const int x = __ffs(todo) - 1;
        uint64_t B[E];
#pragma unroll
        for (int k = 0; k < E; ++k) B[k] = nxt[k];
        const uint32_t rest = todo & (todo - 1);
        if (rest) load(__shfl_sync(FULL, ib, __ffs(rest) - 1), nxt);
        const int32_t i_a = __shfl_sync(FULL, ia, x), i_b = __shfl_sync(FULL, ib, x);
        if (i_a != held) {
            held = i_a;
            uint64_t a[E];
            load(i_a, a);
            __syncwarp();
#pragma unroll
            for (int k = 0; k < WORDS / 32; ++k) bm[32 * k + lane] = 0u;
            __syncwarp();
            n_a = 0;
#pragma unroll
            for (int k = 0; k < E; ++k) {
                A[32 * k + lane] = a[k];
                const bool real = a[k] != MAXV;
                const uint32_t h = (uint32_t)a[k] & (BITS - 1);
                if (real) atomicOr(&bm[h >> 5], 1u << (h & 31));
                n_a += __popc(__ballot_sync(FULL, real));
            }
            __syncwarp();
        }
        uint32_t hit = 0;
#pragma unroll
        for (int k = 0; k < E; ++k) {
            const uint32_t h = (uint32_t)B[k] & (BITS - 1);
            if (B[k] != MAXV && ((bm[h >> 5] >> (h & 31)) & 1u)) hit |= 1u << k;
        }
        int32_t shared = 0, total = 0;
        uint32_t paired = 0;
        int32_t at[E];  // of a paired element: its place in A plus its copies before it in B
        // each lane works through its own hits, so a pair costs as many
        // searches as the lane with the most hits has (mostly one)
        while (__any_sync(FULL, hit != 0)) {
            if (hit) {
                const int k = __ffs(hit) - 1;
                hit &= hit - 1;
                uint64_t v = B[0];
#pragma unroll
                for (int i = 1; i < E; ++i)
                    if (k == i) v = B[i];
                int32_t low = 0;  // A is padded with MAX to 32 E, above any v here
#pragma unroll
                for (int step = 16 * E; step; step >>= 1)
                    if (A[low + step - 1] < v) low += step;
                if (A[low] == v) {
                    const uint64_t *gb = sk + (int64_t)i_b * s;
                    const int32_t j = 32 * k + lane;
                    int32_t m = 0;
                    while (m < j && __ldg(gb + j - m - 1) == v) ++m;
                    if (low + m < s && A[low + m] == v) {
                        paired |= 1u << k;
#pragma unroll
                        for (int i = 0; i < E; ++i)
                            if (k == i) at[i] = low + m;
                    }
                }
            }
        }
        if (__any_sync(FULL, paired != 0)) {
#pragma unroll
            for (int k = 0; k < E; ++k) {
                const bool p = (paired >> k) & 1u;
                const uint32_t bal = __ballot_sync(FULL, p);
                const int32_t r = total + __popc(bal & ((1u << lane) - 1u));
                shared += __popc(__ballot_sync(FULL, p && at[k] + 32 * k + lane - r < s));
                total += __popc(bal);
            }
        }
        int32_t steps = s;  // a full sketch alone gives the walk its s steps
        if (n_a < s) {
            int32_t n_b = 0;
#pragma unroll
            for (int k = 0; k < E; ++k) n_b += __popc(__ballot_sync(FULL, B[k] != MAXV));
            const int32_t T = n_a + n_b - total;
            steps = T < s ? T : s;
        }
        if (lane == x) sim = steps == 0 ? 0.0f : __fdiv_rn((float)shared, (float)steps);
    }
    if (lane < np) {
        sims[p0 + lane] = sim;
        if (mask) mask[p0 + lane] = ok && sim >= floor;
    }
}

template <int E>
static int32_t launch_bitmap(const int32_t *pairs, int64_t M, const uint64_t *sk, int64_t N, int32_t s, float floor,
                             float *sims, uint8_t *mask, int32_t *d_err, cudaStream_t st) {
    const size_t per_warp = (size_t)(32 * E + 32 * E) * sizeof(uint64_t);  // A, and 64 bits an element
    const int wpb = 8;
    // runs short enough that a small list still fills the SMs (48 warps each)
    const int64_t fill = (M + 48 * (int64_t)sm_count() - 1) / (48 * (int64_t)sm_count());
    const int32_t run = (int32_t)(fill < 1 ? 1 : fill > JACCARD_RUN ? JACCARD_RUN : fill);
    const int64_t blocks = ((M + run - 1) / run + wpb - 1) / wpb;
    jaccard_bitmap_kernel<E><<<(unsigned)blocks, wpb * 32, per_warp * wpb, st>>>(pairs, M, sk, N, s, run, floor, sims,
                                                                                 mask, d_err);
    CK_CUDA(cudaGetLastError());
    return CK_OK;
}

int32_t jaccard_launch(const int32_t *pairs, int64_t M, const uint64_t *sk, int64_t N, int32_t s,
                       float floor, float *sims, uint8_t *mask, int32_t *d_err, cudaStream_t st) {
    if (s < 1 || s > 4096) {
        set_error(CK_ERR_UNSUPPORTED, "jaccard: need 1 <= s <= 4096");
        return CK_ERR_UNSUPPORTED;
    }
    if (M == 0) return CK_OK;
    if (s <= 32) return launch_bitmap<1>(pairs, M, sk, N, s, floor, sims, mask, d_err, st);
    if (s <= 64) return launch_bitmap<2>(pairs, M, sk, N, s, floor, sims, mask, d_err, st);
    if (s <= 128) return launch_bitmap<4>(pairs, M, sk, N, s, floor, sims, mask, d_err, st);
    if (s <= 256) return launch_bitmap<8>(pairs, M, sk, N, s, floor, sims, mask, d_err, st);
    const size_t per_warp = ((size_t)2 * s + s / 2 + 2) * sizeof(uint64_t);
    int wpb = (int)((48 * 1024) / per_warp);
    if (wpb > 8) wpb = 8;
    if (wpb < 1) {
        wpb = 1;
        CK_CUDA(cudaFuncSetAttribute(jaccard_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)per_warp));
    }
    int64_t want = (M + wpb - 1) / wpb;
    int64_t cap = (int64_t)sm_count() * 32;
    const int blocks = (int)(want < cap ? want : cap);
    jaccard_kernel<<<blocks, wpb * 32, per_warp * wpb, st>>>(pairs, M, sk, N, s, floor, sims, mask, d_err);
    CK_CUDA(cudaGetLastError());
    return CK_OK;
}

}  // namespace ck
