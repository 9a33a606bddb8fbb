// graph.cu -- similarity graph (CSR) and connected components on the device.
//
// Graph (clustkit/graph.py:7-39): the edges (i, j) and (j, i) of every
// passing pair with its identity as weight, in CSR form with the columns of
// each row ascending and repeated (row, column) entries summed -- scipy's
// canonical form after coo_matrix(...).tocsr().  Built by one radix sort of
// (row, column) keys, packed in as many bits as N needs, with their weights, a reduce-by-key for the
// duplicates and a histogram + scan of the rows for the row pointers.
//
// Connected components (clustkit/cluster.py:43-55, scipy's
// connected_components on the undirected graph): union-find over the edge list
// in two passes.  The first links every node to its smallest neighbour below it
// and compresses, which leaves most of a family under one root; in the second
// an edge follows both ends to their roots and hooks the larger under the
// smaller by compare-and-swap, going on from there when another edge has hooked
// that root meanwhile.  A parent is only ever smaller than its child, so
// every component's root is its smallest node.  scipy numbers
// components in order of their smallest node, so a node's label is the number
// of roots below its root.  The host waits once, for the count.  100,000 nodes
// and 250,000 edges: 0.50 -> 0.36 ms with the graph, whose keys lost two sort
// passes (rounds of hooking by atomicMin and pointer jumping, with a host read
// a round, before).  1,000,000 nodes: one chain in any order of its edges 0.27 ms
// (0.84 walking it to its end from every node; by rounds 0.6), a star 0.17 (0.48
// with an atomic for every edge; 0.43).
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_reduce.cuh>
#include <cub/device/device_scan.cuh>

#include "ck_common.cuh"

namespace ck {

struct FAdd {
    __device__ __forceinline__ float operator()(float x, float y) const { return x + y; }
};

static int grid_n(int64_t work, int threads) {
    int64_t b = (work + threads - 1) / threads;
    const int64_t cap = (int64_t)sm_count() * 32;
    if (b > cap) b = cap;
    return (int)(b < 1 ? 1 : b);
}

__global__ void graph_edges_kernel(const int32_t *__restrict__ pairs, const float *__restrict__ sims, int64_t K,
                                   int64_t N, int32_t col_bits, uint64_t *__restrict__ keys,
                                   float *__restrict__ w, int32_t *err) {
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < K; e += (int64_t)gridDim.x * blockDim.x) {
        int64_t i = pairs[2 * e], j = pairs[2 * e + 1];
        if (i < 0 || j < 0 || i >= N || j >= N) {
            atomicOr(err, ERRBIT_PAIR_INDEX);
            i = j = 0;  // harmless placeholder; the call reports the error
        }
        keys[e] = ((uint64_t)i << col_bits) | (uint64_t)j;
        keys[K + e] = ((uint64_t)j << col_bits) | (uint64_t)i;
        const float s = sims ? sims[e] : 1.0f;
        w[e] = s;
        w[K + e] = s;
    }
}

__global__ void graph_rows_kernel(const uint64_t *__restrict__ ukeys, const int64_t *__restrict__ nnz_p,
                                  int32_t col_bits, int32_t *__restrict__ indices, int64_t *__restrict__ row_count) {
    const int64_t nnz = *nnz_p;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t k = ukeys[e];
        indices[e] = (int32_t)(k & (((uint64_t)1 << col_bits) - 1));
        atomicAdd((unsigned long long *)&row_count[k >> col_bits], 1ull);
    }
}

struct GraphArgs {
    const int32_t *pairs; const float *sims; int64_t K, N;
    int64_t *indptr; int32_t *indices; float *data; int64_t *out_nnz; cudaStream_t st;
};

static int32_t graph_impl(void *pv) {
    GraphArgs &a = *(GraphArgs *)pv;
    int32_t status = CK_OK;
    cudaStream_t st = a.st;
    int32_t *err = device_error_word(&status);
    if (!err) return status;
    const int64_t E = 2 * a.K;
    CK_CUDA(cudaMemsetAsync(a.indptr, 0, (size_t)(a.N + 1) * 8, st));
    *a.out_nnz = 0;
    if (E == 0) return CK_OK;
    if (a.N == 0) {  // no row to write an edge to
        set_error(CK_ERR_OUT_OF_RANGE, "graph: pair index outside [0, N)");
        return CK_ERR_OUT_OF_RANGE;
    }
    uint64_t *keys = (uint64_t *)scratch(SLOT_SEARCH_TMP1, (size_t)E * 8 * 2, &status);
    float *w = (float *)scratch(SLOT_SEARCH_TMP2, (size_t)E * 4 * 2, &status);
    int64_t *nnz_d = (int64_t *)scratch(SLOT_MAXLEN, 64, &status);
    if (!keys || !w || !nnz_d) return status;
    int32_t col_bits = 1;  // N < 2^31: a key has at most 62
    while (((int64_t)1 << col_bits) < a.N) ++col_bits;
    const int bits = 2 * col_bits;
    graph_edges_kernel<<<grid_n(a.K, 256), 256, 0, st>>>(a.pairs, a.sims, a.K, a.N, col_bits, keys, w, err);
    CK_CUDA(cudaGetLastError());
    cub::DoubleBuffer<uint64_t> dk(keys, keys + E);
    cub::DoubleBuffer<float> dv(w, w + E);
    size_t t1 = 0, t2 = 0;
    CK_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, t1, dk, dv, E, 0, bits, st));
    CK_CUDA(cub::DeviceReduce::ReduceByKey(nullptr, t2, dk.Current(), dk.Alternate(), dv.Current(), a.data,
                                           nnz_d, FAdd(), E, st));
    void *tmp = scratch(SLOT_SORT_TEMP, std::max(t1, t2), &status);
    if (!tmp) return status;
    CK_CUDA(cub::DeviceRadixSort::SortPairs(tmp, t1, dk, dv, E, 0, bits, st));
    // unique keys into the alternate key buffer, summed weights straight into data
    size_t tt = std::max(t1, t2);
    CK_CUDA(cub::DeviceReduce::ReduceByKey(tmp, tt, dk.Current(), dk.Alternate(), dv.Current(), a.data, nnz_d,
                                           FAdd(), E, st));
    graph_rows_kernel<<<grid_n(E, 256), 256, 0, st>>>(dk.Alternate(), nnz_d, col_bits, a.indices, a.indptr + 1);
    CK_CUDA(cudaGetLastError());
    size_t ts = 0;
    CK_CUDA(cub::DeviceScan::InclusiveSum(nullptr, ts, a.indptr + 1, a.indptr + 1, a.N, st));
    void *tmp2 = scratch(SLOT_SORT_TEMP, std::max(std::max(t1, t2), ts), &status);
    if (!tmp2) return status;
    CK_CUDA(cub::DeviceScan::InclusiveSum(tmp2, ts, a.indptr + 1, a.indptr + 1, a.N, st));
    int32_t h = 0;
    CK_CUDA(cudaMemcpyAsync(a.out_nnz, nnz_d, 8, cudaMemcpyDeviceToHost, st));
    CK_CUDA(cudaMemcpyAsync(&h, err, 4, cudaMemcpyDeviceToHost, st));
    CK_CUDA(cudaMemsetAsync(err, 0, 4, st));
    CK_CUDA(cudaStreamSynchronize(st));
    if (h) {
        set_error(CK_ERR_OUT_OF_RANGE, "graph: pair index outside [0, N)");
        return CK_ERR_OUT_OF_RANGE;
    }
    return CK_OK;
}

// ------------------------------------------------------------ components
__device__ __forceinline__ int32_t uf_find(const int32_t *parent, int32_t x) {
    int32_t p = parent[x];
    while (p != x) {
        x = p;
        p = parent[x];
    }
    return x;
}

// The root of x0, for a thread that alone writes parent[x0]: every UF_OWN steps
// it points there at where the walk has come to, so that a long chain, walked
// from all its nodes at once, halves again and again.  A short walk reads through
// L1, a long one past it, to see what the others have written.
constexpr int UF_OWN = 8;
__device__ __forceinline__ int32_t uf_find_own(int32_t *parent, int32_t x0) {
    int32_t x = x0, p = parent[x];
    for (int n = 1; p != x; ++n) {
        x = p;
        p = n < UF_OWN ? parent[x] : __ldcg(parent + x);
        if (n % UF_OWN == 0) parent[x0] = x;
    }
    return x;
}

__global__ void cc_init_kernel(int32_t *parent, int64_t N) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x)
        parent[i] = (int32_t)i;
}

// Links the larger end of every edge to the smallest such neighbour (parents
// freshly initialised); out-of-range pairs are left to the pass over roots.
__global__ void cc_link_kernel(const int32_t *__restrict__ pairs, int64_t K, int64_t N, int32_t *parent) {
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < K; e += (int64_t)gridDim.x * blockDim.x) {
        const int32_t u = pairs[2 * e], v = pairs[2 * e + 1];
        if (u < 0 || v < 0 || u >= N || v >= N || u == v) continue;
        // a parent read from L1 may be an old one, which is larger: then the atomic
        // finds out.  A node of many edges is spared most of its atomics.
        const int32_t hi = u > v ? u : v, lo = u ^ v ^ hi;
        if (parent[hi] > lo) atomicMin(parent + hi, lo);
    }
}

__global__ void cc_union_kernel(const int32_t *__restrict__ pairs, int64_t K, int64_t N, int32_t *parent,
                                int32_t *err) {
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < K; e += (int64_t)gridDim.x * blockDim.x) {
        int32_t u = pairs[2 * e], v = pairs[2 * e + 1];
        if (u < 0 || v < 0 || u >= N || v >= N) {
            atomicOr(err, ERRBIT_PAIR_INDEX);
            continue;
        }
        // each turn either ends or goes on from a smaller node, so it ends.  A
        // parent read from L1 may be an old one: still an ancestor, or, for what
        // was a root, caught by the compare-and-swap.  (Reads past L1 queued up
        // at the lines of the few roots that most edges share: 152 us.)
        for (;;) {
            u = uf_find(parent, u);
            v = uf_find(parent, v);
            if (u == v) break;
            const int32_t hi = u > v ? u : v, lo = u ^ v ^ hi;
            const int32_t was = atomicCAS(parent + hi, hi, lo);
            if (was == hi) break;
            u = was;  // hooked by another edge meanwhile: under `was` < hi
            v = lo;
        }
    }
}

__global__ void cc_compress_kernel(int32_t *parent, int64_t N) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x)
        parent[i] = uf_find_own(parent, (int32_t)i);
}

__global__ void cc_root_flags_kernel(const int32_t *parent, int64_t N, int32_t *flag) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x)
        flag[i] = parent[i] == (int32_t)i ? 1 : 0;
}

__global__ void cc_label_kernel(const int32_t *parent, const int32_t *rank, int64_t N, int32_t *labels) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x)
        labels[i] = rank[parent[i]];
}

struct CcArgs {
    const int32_t *pairs; int64_t K, N; int32_t *labels; int64_t *out_n; int32_t *out_rounds; cudaStream_t st;
};

static int32_t cc_impl(void *pv) {
    CcArgs &a = *(CcArgs *)pv;
    int32_t status = CK_OK;
    cudaStream_t st = a.st;
    *a.out_n = 0;
    if (a.out_rounds) *a.out_rounds = 0;
    if (a.N == 0) return CK_OK;
    int32_t *err = device_error_word(&status);
    int32_t *parent = (int32_t *)scratch(SLOT_SEARCH_TMP3, (size_t)a.N * 4 * 2 + 8, &status);
    if (!err || !parent) return status;
    int32_t *rank = parent + a.N;
    cc_init_kernel<<<grid_n(a.N, 256), 256, 0, st>>>(parent, a.N);
    CK_CUDA(cudaGetLastError());
    if (a.K > 0) {
        cc_link_kernel<<<grid_n(a.K, 256), 256, 0, st>>>(a.pairs, a.K, a.N, parent);
        CK_CUDA(cudaGetLastError());
        cc_compress_kernel<<<grid_n(a.N, 256), 256, 0, st>>>(parent, a.N);
        CK_CUDA(cudaGetLastError());
        cc_union_kernel<<<grid_n(a.K, 256), 256, 0, st>>>(a.pairs, a.K, a.N, parent, err);
        CK_CUDA(cudaGetLastError());
        cc_compress_kernel<<<grid_n(a.N, 256), 256, 0, st>>>(parent, a.N);
        CK_CUDA(cudaGetLastError());
    }
    cc_root_flags_kernel<<<grid_n(a.N, 256), 256, 0, st>>>(parent, a.N, a.labels);
    CK_CUDA(cudaGetLastError());
    size_t ts = 0;
    CK_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, ts, a.labels, rank, a.N, st));
    void *tmp = scratch(SLOT_SORT_TEMP, ts, &status);
    if (!tmp) return status;
    CK_CUDA(cub::DeviceScan::ExclusiveSum(tmp, ts, a.labels, rank, a.N, st));
    int32_t last_flag = 0, last_rank = 0, e_h = 0;
    CK_CUDA(cudaMemcpyAsync(&last_flag, a.labels + a.N - 1, 4, cudaMemcpyDeviceToHost, st));
    CK_CUDA(cudaMemcpyAsync(&last_rank, rank + a.N - 1, 4, cudaMemcpyDeviceToHost, st));
    CK_CUDA(cudaMemcpyAsync(&e_h, err, 4, cudaMemcpyDeviceToHost, st));
    CK_CUDA(cudaMemsetAsync(err, 0, 4, st));
    cc_label_kernel<<<grid_n(a.N, 256), 256, 0, st>>>(parent, rank, a.N, a.labels);
    CK_CUDA(cudaGetLastError());
    CK_CUDA(cudaStreamSynchronize(st));
    if (e_h) {
        set_error(CK_ERR_OUT_OF_RANGE, "components: pair index outside [0, N)");
        return CK_ERR_OUT_OF_RANGE;
    }
    *a.out_n = (int64_t)last_rank + last_flag;
    if (a.out_rounds) *a.out_rounds = a.K > 0 ? 1 : 0;
    return CK_OK;
}

}  // namespace ck

using namespace ck;

extern "C" int32_t ck_graph_csr_device(int32_t ctx, const int32_t *d_pairs, const float *d_sims, int64_t K,
                                       int64_t N, int64_t *d_indptr, int32_t *d_indices, float *d_data,
                                       int64_t *out_nnz, void *stream) {
    std::lock_guard<std::mutex> lock(library_mutex());
    reset_thread_status();
    if (K < 0 || N < 0 || N >= ((int64_t)1 << 31) || !out_nnz || !d_indptr ||
        (K > 0 && (!d_pairs || !d_indices || !d_data))) {
        set_error(CK_ERR_INVALID_ARGUMENT, "graph: bad arguments");
        return CK_ERR_INVALID_ARGUMENT;
    }
    GraphArgs a{d_pairs, d_sims, K, N, d_indptr, d_indices, d_data, out_nnz, (cudaStream_t)stream};
    return run_in_context(ctx, graph_impl, &a);
}

extern "C" int32_t ck_connected_components_device(int32_t ctx, const int32_t *d_pairs, int64_t K, int64_t N,
                                                  int32_t *d_labels, int64_t *out_n_components,
                                                  int32_t *out_rounds, void *stream) {
    std::lock_guard<std::mutex> lock(library_mutex());
    reset_thread_status();
    if (K < 0 || N < 0 || N >= ((int64_t)1 << 31) || !out_n_components || (N > 0 && !d_labels) ||
        (K > 0 && !d_pairs)) {
        set_error(CK_ERR_INVALID_ARGUMENT, "components: bad arguments");
        return CK_ERR_INVALID_ARGUMENT;
    }
    CcArgs a{d_pairs, K, N, d_labels, out_n_components, out_rounds, (cudaStream_t)stream};
    return run_in_context(ctx, cc_impl, &a);
}
