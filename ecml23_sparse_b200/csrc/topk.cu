// Top-k selection behind ffi_forward_topk (evaluation and serving; PrecisionAtK of sparse/metrics.py:9-70 needs the k best
// labels per sample): the merge of the lists that the forward kernels' epilogues keep, and the selection over the rows of
// y that the small-batch forward writes.  Order of tf.nn.top_k: value descending, lower index first on ties.
#include "ffi_common.cuh"

namespace ffi {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

// Every thread brings a sorted list; the block's best kk go to emit(j, value, row), j ascending.  One round per rank: the
// best head of all lists (shuffles, then one exchange through shared memory), whose owner moves on.
template <class Emit>
__device__ __forceinline__ void block_select(float (&tv)[kTopK], int (&ti)[kTopK], int kk, Emit&& emit) {
    __shared__ float sv[2][kWarps];
    __shared__ int si[2][kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int j = 0; j < kk; ++j) {
        float v = tv[0];
        int i = ti[0];
#pragma unroll
        for (int off = 16; off >= 1; off /= 2) {
            const float v2 = __shfl_xor_sync(0xffffffffu, v, off);
            const int i2 = __shfl_xor_sync(0xffffffffu, i, off);
            if (topk_better(v2, i2, v, i)) v = v2, i = i2;
        }
        if (lane == 0) sv[j & 1][warp] = v, si[j & 1][warp] = i;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < kWarps; ++w)
            if (topk_better(sv[j & 1][w], si[j & 1][w], v, i)) v = sv[j & 1][w], i = si[j & 1][w];
        if (ti[0] == i) {  // rows are distinct: one owner (or only exhausted lists are left)
#pragma unroll
            for (int u = 0; u + 1 < kTopK; ++u) tv[u] = tv[u + 1], ti[u] = ti[u + 1];
            tv[kTopK - 1] = -INFINITY, ti[kTopK - 1] = 0x7fffffff;
        }
        if (threadIdx.x == 0) emit(j, v, i);
    }
}

__device__ __forceinline__ void clear_list(float (&tv)[kTopK], int (&ti)[kTopK]) {
#pragma unroll
    for (int j = 0; j < kTopK; ++j) tv[j] = -INFINITY, ti[j] = 0x7fffffff;
}

// A value that at least kTopK candidates of the block reach: the lowest of its warps' maxima (one warp per rank).  Every
// thread brings the maximum m of candidates of its own; wmax keeps each warp's highest so far, and a bound from values that
// are not all there yet is only a weaker one.
static_assert(kWarps == kTopK, "block_bound takes one candidate per warp");
__device__ __forceinline__ void note_max(int* wmax, float m) {
    const int key = __reduce_max_sync(0xffffffffu, order_key(m));
    if ((threadIdx.x & 31) == 0 && key > wmax[threadIdx.x >> 5]) wmax[threadIdx.x >> 5] = key;
}
__device__ __forceinline__ float block_bound(const int* wmax) {
    int key = 0x7fffffff;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) key = min(key, reinterpret_cast<const volatile int*>(wmax)[w]);
    return order_value(key);
}

// The block's share of n sorted lists, list l at lists + l * stride with `len` entries, into every thread's own list.  Only the
// few entries that reach the bound of the heads are looked at (1,184 lists for each of 128 samples: 15.9 ->
// 9.2 us).
__device__ __forceinline__ void gather_lists(const uint2* lists, int n, size_t stride, int len, float (&tv)[kTopK], int (&ti)[kTopK],
                                             int* wmax) {
    if (threadIdx.x < kWarps) wmax[threadIdx.x] = order_key(-INFINITY);
    float m = -INFINITY;
    for (int l = threadIdx.x; l < n; l += kThreads) m = fmaxf(m, __uint_as_float(__ldcg(lists + l * stride).x));
    __syncthreads();
    note_max(wmax, m);
    __syncthreads();
    const float bound = block_bound(wmax);
    if (m >= bound)
        for (int l = threadIdx.x; l < n; l += kThreads)
            for (int j = 0; j < len; ++j) {
                const uint2 c = __ldcg(lists + l * stride + j);
                if (!(__uint_as_float(c.x) >= bound)) break;
                topk_insert(tv, ti, __uint_as_float(c.x), static_cast<int>(c.y));
            }
}

// One block per batch element: the best kk of all (sorted) lists of its tile, lists[tile][list][BT][kTopK].
__global__ void __launch_bounds__(kThreads) topk_merge_kernel(const uint2* __restrict__ lists, int listsPerTile, int BT,
                                                              int kk, int label_offset, float* __restrict__ out_val,
                                                              int* __restrict__ out_idx) {
    chain_begin();
    const int b = blockIdx.x;
    const int tile = b / BT, bl = b - tile * BT;
    float tv[kTopK];
    int ti[kTopK];
    clear_list(tv, ti);
    __shared__ int wmax[kWarps];
    gather_lists(lists + static_cast<size_t>(tile) * listsPerTile * (BT * kTopK) + bl * kTopK, listsPerTile, BT * kTopK, kTopK, tv, ti,
                 wmax);
    block_select(tv, ti, kk, [&](int j, float v, int i) {
        out_val[static_cast<size_t>(b) * kk + j] = v;
        out_idx[static_cast<size_t>(b) * kk + j] = i == 0x7fffffff ? -1 : i + label_offset;
    });
}

// Block (segment, sample): the best kk of y[sample][segment], as one list of lists[sample][segment][kTopK]; the sample's last
// block to finish (tickets, cleared beforehand) merges them.  A value goes into a thread's list only if it reaches the block's
// bound, which about one in a hundred does; the sorted insertion of all of them was what this kernel spent its time on
// (6 samples of 567,584 rows: 28.9 us and 3.5 for a merge of its own -> 15.8; one of 670,091: 8 + 7 -> 12.2).
__global__ void __launch_bounds__(kThreads) topk_rows_kernel(const float* __restrict__ y, int L, int segRows, int kk, uint2* lists,
                                                             unsigned* tickets, int label_offset, float* __restrict__ out_val,
                                                             int* __restrict__ out_idx) {
    chain_begin();
    __shared__ int wmax[kWarps];
    __shared__ bool last;
    const int o0 = blockIdx.x * segRows, o1 = min(L, o0 + segRows);
    const float* row = y + static_cast<size_t>(blockIdx.y) * L;
    float tv[kTopK];
    int ti[kTopK];
    clear_list(tv, ti);
    if (threadIdx.x < kWarps) wmax[threadIdx.x] = order_key(-INFINITY);
    __syncthreads();
    constexpr int U = 8;
    for (int base = o0; base < o1; base += U * kThreads) {
        const int o = base + threadIdx.x;
        float v[U], m = -INFINITY;
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = o + u * kThreads < o1 ? __ldg(row + o + u * kThreads) : -INFINITY;
#pragma unroll
        for (int u = 0; u < U; ++u) m = fmaxf(m, v[u]);
        note_max(wmax, m);
        if (base == o0) __syncthreads();
        const float bound = block_bound(wmax);
        if (m >= bound) {
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (v[u] >= bound && o + u * kThreads < o1) topk_insert(tv, ti, v[u], o + u * kThreads);
        }
    }
    uint2* mine = lists + (static_cast<size_t>(blockIdx.y) * gridDim.x + blockIdx.x) * kTopK;
    block_select(tv, ti, kk, [&](int j, float v, int i) { mine[j] = make_uint2(__float_as_uint(v), static_cast<unsigned>(i)); });
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(tickets + blockIdx.y, 1u) + 1 == gridDim.x;
        __threadfence();
    }
    __syncthreads();
    if (!last) return;
    clear_list(tv, ti);
    gather_lists(lists + static_cast<size_t>(blockIdx.y) * gridDim.x * kTopK, gridDim.x, kTopK, kk, tv, ti, wmax);
    __syncthreads();
    block_select(tv, ti, kk, [&](int j, float v, int i) {
        out_val[blockIdx.y * kk + j] = v;
        out_idx[blockIdx.y * kk + j] = i == 0x7fffffff ? -1 : i + label_offset;
    });
}

// Segments per sample: about two blocks per SM over the batch, at least 2048 rows each.
int64_t row_segments(int64_t B, int64_t L, const DeviceInfo& dev) {
    const int64_t want = ceil_div(2 * dev.sm_count, B), most = ceil_div(L, 2048);
    return want < most ? want : most;
}

}  // namespace

int launch_topk_merge(const uint2* lists, int lists_per_tile, int bt, int B, int kk, int label_offset, float* top_val,
                      int* top_idx, cudaStream_t stream) {
    FFI_CUDA_CHECK(launch_chained(topk_merge_kernel, dim3(static_cast<unsigned>(B)), dim3(kThreads), 0, stream, lists, lists_per_tile, bt, kk,
                                  label_offset, top_val, top_idx));
    FFI_LAUNCH_CHECK("topk_merge_kernel");
    return FFI_OK;
}

size_t topk_rows_list_bytes(int64_t B, int64_t L) {
    DeviceInfo dev;
    if (get_device_info(&dev) != FFI_OK) return 0;
    return static_cast<size_t>(B) * (row_segments(B, L, dev) * kTopK * sizeof(uint2) + sizeof(unsigned));
}

// the samples' tickets, behind the lists: cleared by whatever writes y
unsigned* topk_rows_tickets(void* lists, int64_t B, int64_t L) {
    return reinterpret_cast<unsigned*>(static_cast<unsigned char*>(lists) + topk_rows_list_bytes(B, L)) - B;
}

// top-k of the rows of y[B][L]; `lists` holds topk_rows_list_bytes, the tickets in it are zero.
int launch_topk_rows(const float* y, int64_t B, int64_t L, uint2* lists, int kk, int label_offset, float* top_val, int* top_idx,
                     cudaStream_t stream) {
    DeviceInfo dev;
    const int rc = get_device_info(&dev);
    if (rc != FFI_OK) return rc;
    const int64_t segs = row_segments(B, L, dev);
    const int segRows = static_cast<int>(ceil_div(L, segs));
    FFI_CUDA_CHECK(launch_chained(topk_rows_kernel, dim3(static_cast<unsigned>(segs), static_cast<unsigned>(B)), dim3(kThreads), 0, stream, y,
                                  static_cast<int>(L), segRows, kk, lists, topk_rows_tickets(lists, B, L), label_offset, top_val, top_idx));
    FFI_LAUNCH_CHECK("topk_rows_kernel");
    return FFI_OK;
}

}  // namespace ffi
