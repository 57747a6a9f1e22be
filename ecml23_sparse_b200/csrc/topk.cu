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

// One block per batch element: the best kk of all (sorted) lists of its tile, lists[tile][list][BT][kTopK].
__global__ void __launch_bounds__(kThreads) topk_merge_kernel(const uint2* __restrict__ lists, int listsPerTile, int BT,
                                                              int kk, int label_offset, float* __restrict__ out_val,
                                                              int* __restrict__ out_idx) {
    const int b = blockIdx.x;
    const int tile = b / BT, bl = b - tile * BT;
    float tv[kTopK];
    int ti[kTopK];
    clear_list(tv, ti);
    for (int l = threadIdx.x; l < listsPerTile; l += kThreads) {
        const uint4* src = reinterpret_cast<const uint4*>(
            lists + (static_cast<size_t>(tile) * listsPerTile + l) * (BT * kTopK) + bl * kTopK);
        uint4 c[kTopK / 2];
#pragma unroll
        for (int j = 0; j < kTopK / 2; ++j) c[j] = __ldg(src + j);
#pragma unroll
        for (int j = 0; j < kTopK / 2; ++j) {
            topk_insert(tv, ti, __uint_as_float(c[j].x), static_cast<int>(c[j].y));
            topk_insert(tv, ti, __uint_as_float(c[j].z), static_cast<int>(c[j].w));
        }
    }
    block_select(tv, ti, kk, [&](int j, float v, int i) {
        out_val[static_cast<size_t>(b) * kk + j] = v;
        out_idx[static_cast<size_t>(b) * kk + j] = i == 0x7fffffff ? -1 : i + label_offset;
    });
}

// Block (segment, sample): the best kTopK of y[sample][segment], as one list of lists[sample][segment][kTopK].
__global__ void __launch_bounds__(kThreads) topk_rows_kernel(const float* __restrict__ y, int L, int segRows, int kk,
                                                             uint2* __restrict__ lists) {
    const int o0 = blockIdx.x * segRows, o1 = min(L, o0 + segRows);
    const float* row = y + static_cast<size_t>(blockIdx.y) * L;
    float tv[kTopK];
    int ti[kTopK];
    clear_list(tv, ti);
    constexpr int U = 8;
    for (int o = o0 + threadIdx.x; o < o1; o += U * kThreads) {
        float v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = o + u * kThreads < o1 ? __ldg(row + o + u * kThreads) : -INFINITY;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (o + u * kThreads < o1) topk_insert(tv, ti, v[u], o + u * kThreads);
    }
    uint2* out = lists + (static_cast<size_t>(blockIdx.y) * gridDim.x + blockIdx.x) * kTopK;
    if (threadIdx.x < kTopK) out[threadIdx.x] = make_uint2(__float_as_uint(-INFINITY), 0x7fffffffu);
    __syncthreads();
    block_select(tv, ti, kk, [&](int j, float v, int i) { out[j] = make_uint2(__float_as_uint(v), static_cast<unsigned>(i)); });
}

// Segments per sample: about two blocks per SM over the batch, at least 2048 rows each.
int64_t row_segments(int64_t B, int64_t L, const DeviceInfo& dev) {
    const int64_t want = ceil_div(2 * dev.sm_count, B), most = ceil_div(L, 2048);
    return want < most ? want : most;
}

}  // namespace

int launch_topk_merge(const uint2* lists, int lists_per_tile, int bt, int B, int kk, int label_offset, float* top_val,
                      int* top_idx, cudaStream_t stream) {
    topk_merge_kernel<<<static_cast<unsigned>(B), kThreads, 0, stream>>>(lists, lists_per_tile, bt, kk, label_offset, top_val,
                                                                         top_idx);
    FFI_LAUNCH_CHECK("topk_merge_kernel");
    return FFI_OK;
}

size_t topk_rows_list_bytes(int64_t B, int64_t L) {
    DeviceInfo dev;
    if (get_device_info(&dev) != FFI_OK) return 0;
    return static_cast<size_t>(B) * row_segments(B, L, dev) * kTopK * sizeof(uint2);
}

// top-k of the rows of y[B][L]; `lists` holds topk_rows_list_bytes.
int launch_topk_rows(const float* y, int64_t B, int64_t L, uint2* lists, int kk, int label_offset, float* top_val, int* top_idx,
                     cudaStream_t stream) {
    DeviceInfo dev;
    const int rc = get_device_info(&dev);
    if (rc != FFI_OK) return rc;
    const int64_t segs = row_segments(B, L, dev);
    const int segRows = static_cast<int>(ceil_div(L, segs));
    topk_rows_kernel<<<dim3(static_cast<unsigned>(segs), static_cast<unsigned>(B)), kThreads, 0, stream>>>(
        y, static_cast<int>(L), segRows, kk, lists);
    FFI_LAUNCH_CHECK("topk_rows_kernel");
    return launch_topk_merge(lists, static_cast<int>(segs), 1, static_cast<int>(B), kk, label_offset, top_val, top_idx, stream);
}

}  // namespace ffi
