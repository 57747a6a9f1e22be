// Forward of the fixed-fan-in sparse layer for a handful of samples (batch <= 8): serving, single queries.
//   y[b,o] = bias[o] + sum_k W[o,k] * x[b, idx[o,k]]
// Replaces the reference's forward_ob_scalar_tp / forward_ib_unrolled (tfsparse/cc/kernels/forward.cu.h:231-264) for
// that range; the batched kernels (forward_stream.cu) put the batch on the lanes and leave most of a warp idle here.
//
// The lanes run along k instead: G lanes share a row, each takes four consecutive entries (one 16-byte load of W and of
// idx), gathers the operands of all samples from shared memory (x_s[N][BP], 4*BP bytes per entry) and the G partial sums
// are added with shuffles.  What bounds it is the stream of W and idx from HBM (8 bytes per entry) up to four samples, and
// the shared-memory gathers (random rows: about 2.6 to 3.5 conflicts per phase) from eight on.  At N=768, L=670,091,
// K=32, fp32, writing y: 34 / 36 / 50 / 90 us for 1 / 2 / 4 / 8 samples (5.0 TB/s at one), against 148 us of the batched
// kernel for any batch up to 32; with 16 samples per entry it took 258 us, so the batched kernel has that.
#include <type_traits>

#include "ffi_common.cuh"

namespace ffi {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

struct SmallParams {
    const void* x;  // element type TX; x[i * x_si + b * x_sb]
    long long x_si, x_sb;
    const int* idx;
    const void* W;
    const float* bias;
    float* y;
    int B, N, L, K;
    int lgG;  // log2 of the lanes per row
    unsigned* tickets;  // nullable, [B]: cleared for the top-k selection that follows
};

// x_s[i][b].  The rows of eight samples swap their halves in every other group of four rows: a phase of a 16-byte gather then
// spreads over all eight bank groups, not over the four that hold the same half of every row (B=8, N=768, L=670,091, K=32: 107 ->
// 90 us).
template <int BP>
__device__ __forceinline__ int sample_at(int i, int b) {
    return BP == 8 ? i * 8 + (b ^ (i & 4)) : i * BP + b;
}

template <int BP>
__device__ __forceinline__ void load_samples(const float* x_s, int i, float (&out)[BP]) {
    const float* src = x_s + sample_at<BP>(i, 0);
    if constexpr (BP == 8) {
        const float4 t = *reinterpret_cast<const float4*>(src);
        const float4 t2 = *reinterpret_cast<const float4*>(x_s + (sample_at<BP>(i, 0) ^ 4));
        out[0] = t.x, out[1] = t.y, out[2] = t.z, out[3] = t.w;
        out[4] = t2.x, out[5] = t2.y, out[6] = t2.z, out[7] = t2.w;
    } else if constexpr (BP == 4) {
        const float4 t = *reinterpret_cast<const float4*>(src);
        out[0] = t.x, out[1] = t.y, out[2] = t.z, out[3] = t.w;
    } else if constexpr (BP == 2) {
        const float2 t = *reinterpret_cast<const float2*>(src);
        out[0] = t.x, out[1] = t.y;
    } else {
        out[0] = *src;
    }
}

template <int BP, typename TX>
__global__ void __launch_bounds__(kThreads) ffi_fwd_small_kernel(SmallParams p) {
    chain_begin();
    constexpr bool kBf16 = !std::is_same<TX, float>::value;
    constexpr int U = BP <= 4 ? 4 : 2;  // rows per lane group in flight
    extern __shared__ __align__(16) float x_s[];  // [N][BP]
    const int lane = threadIdx.x & 31;
    const TX* x = static_cast<const TX*>(p.x);
    const TX* W = static_cast<const TX*>(p.W);
    const int K = p.K, L = p.L, Q = K / 4;
    const int G = 1 << p.lgG, gl = lane & (G - 1), gr = lane >> p.lgG;
    const int rpw = 32 >> p.lgG;  // rows a warp works on at once

    // consecutive threads along the contiguous dimension of x
    const int total = p.N * BP;
    if (p.x_sb == 1) {
#pragma unroll 4
        for (int e = threadIdx.x; e < total; e += kThreads) {
            const int i = e / BP, b = e - i * BP;
            x_s[sample_at<BP>(i, b)] = b < p.B ? widen(x[i * p.x_si + b]) : 0.f;
        }
    } else {
#pragma unroll 4
        for (int e = threadIdx.x; e < total; e += kThreads) {
            const int b = e / p.N, i = e - b * p.N;
            x_s[sample_at<BP>(i, b)] = b < p.B ? widen(x[b * p.x_sb + i]) : 0.f;
        }
    }
    if (p.tickets && blockIdx.x == 0 && threadIdx.x < p.B) p.tickets[threadIdx.x] = 0;
    __syncthreads();

    const int tileRows = U * rpw;
    const int numTiles = (L + tileRows - 1) / tileRows;
    for (int t = blockIdx.x * kWarps + (threadIdx.x >> 5); t < numTiles; t += gridDim.x * kWarps) {
        const int o0 = t * tileRows + gr;
        float acc[U][BP];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int b = 0; b < BP; ++b) acc[u][b] = 0.f;
        for (int q = gl; q < Q; q += G) {
            float w[U][4];
            int4 i4[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const size_t at = static_cast<size_t>(min(o0 + u * rpw, L - 1)) * K + 4 * q;
                i4[u] = __ldg(reinterpret_cast<const int4*>(p.idx + at));
                if constexpr (kBf16) {
                    const uint2 r = __ldg(reinterpret_cast<const uint2*>(W + at));
                    w[u][0] = bf16_lo(r.x), w[u][1] = bf16_hi(r.x), w[u][2] = bf16_lo(r.y), w[u][3] = bf16_hi(r.y);
                } else {
                    const float4 r = __ldg(reinterpret_cast<const float4*>(W + at));
                    w[u][0] = r.x, w[u][1] = r.y, w[u][2] = r.z, w[u][3] = r.w;
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int ii[4] = {i4[u].x, i4[u].y, i4[u].z, i4[u].w};
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float v[BP];
                    load_samples<BP>(x_s, ii[c], v);
#pragma unroll
                    for (int b = 0; b < BP; ++b) acc[u][b] = fmaf(w[u][c], v[b], acc[u][b]);
                }
            }
        }
        for (int off = G >> 1; off >= 1; off >>= 1)
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int b = 0; b < BP; ++b) acc[u][b] += __shfl_xor_sync(0xffffffffu, acc[u][b], off);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int o = o0 + u * rpw;
            const float bias = p.bias && o < L ? __ldg(p.bias + o) : 0.f;
#pragma unroll
            for (int b = 0; b < BP; ++b)
                if (gl == 0 && o < L && b < p.B) p.y[static_cast<size_t>(b) * L + o] = acc[u][b] + bias;
        }
    }
}

template <int BP, typename TX>
int launch_small_t(const SmallParams& p, size_t smem, const DeviceInfo& dev, cudaStream_t stream) {
    auto kern = ffi_fwd_small_kernel<BP, TX>;
    int occ = 0;
    FFI_CUDA_CHECK(prepare_kernel(reinterpret_cast<const void*>(kern), kThreads, smem, &occ));
    if (occ < 1) return fail(FFI_ERR_CUDA, "small-batch forward kernel does not fit on an SM (smem %zu)", smem);
    const int tileRows = (BP <= 4 ? 4 : 2) * (32 >> p.lgG);
    const int64_t want = ceil_div(ceil_div(p.L, tileRows), kWarps), cap = static_cast<int64_t>(dev.sm_count) * occ;
    FFI_CUDA_CHECK(launch_chained(kern, dim3(static_cast<unsigned>(want < cap ? want : cap)), dim3(kThreads), smem, stream, p));
    FFI_LAUNCH_CHECK("ffi_fwd_small_kernel");
    return FFI_OK;
}

template <typename TX>
int launch_small_b(const SmallParams& p, int bp, size_t smem, const DeviceInfo& dev, cudaStream_t stream) {
    if (bp == 1) return launch_small_t<1, TX>(p, smem, dev, stream);
    if (bp == 2) return launch_small_t<2, TX>(p, smem, dev, stream);
    if (bp == 4) return launch_small_t<4, TX>(p, smem, dev, stream);
    return launch_small_t<8, TX>(p, smem, dev, stream);
}

}  // namespace

constexpr int kSmallMaxB = 8;

bool forward_small_applicable(int64_t B, int64_t N, int64_t K) {
    DeviceInfo dev;
    if (get_device_info(&dev) != FFI_OK || B > kSmallMaxB || K % 4 != 0) return false;
    int bp = 1;
    while (bp < B) bp *= 2;
    return static_cast<size_t>(N) * bp * 4 <= static_cast<size_t>(dev.max_smem_optin);
}

// y for a batch of at most kSmallMaxB, x in either layout and storage type; *handled = false where another kernel has to run
// (fan-in not a multiple of four, unaligned rows, x too wide for shared memory).
int launch_forward_small(const void* x, int x_transposed, const int32_t* idx, const void* W, bool bf16, const float* bias,
                         float* y, int64_t B, int64_t N, int64_t L, int64_t K, unsigned* tickets, cudaStream_t stream, bool* handled) {
    *handled = false;
    if (!forward_small_applicable(B, N, K) || reinterpret_cast<uintptr_t>(W) % (bf16 ? 8 : 16) != 0 ||
        reinterpret_cast<uintptr_t>(idx) % 16 != 0)
        return FFI_OK;
    DeviceInfo dev;
    const int rc = get_device_info(&dev);
    if (rc != FFI_OK) return rc;
    *handled = true;
    SmallParams p;
    p.x = x;
    p.x_si = x_transposed ? B : 1;
    p.x_sb = x_transposed ? 1 : N;
    p.idx = idx;
    p.W = W;
    p.bias = bias;
    p.y = y;
    p.tickets = tickets;
    p.B = static_cast<int>(B);
    p.N = static_cast<int>(N);
    p.L = static_cast<int>(L);
    p.K = static_cast<int>(K);
    int bp = 1;
    while (bp < B) bp *= 2;
    // lanes per row: the fewest idle lanes over the row's K/4 quads; of equals eight (two 64-byte runs of a K=32 row and
    // four rows per warp), then more, then fewer
    const int64_t Q = K / 4;
    int64_t best = -1;
    for (int lg : {3, 4, 5, 2, 1, 0}) {
        const int64_t slots = round_up(Q, 1 << lg);
        if (best < 0 || slots < best) best = slots, p.lgG = lg;
    }
    const size_t smem = static_cast<size_t>(N) * bp * 4;
    return bf16 ? launch_small_b<__nv_bfloat16>(p, bp, smem, dev, stream) : launch_small_b<float>(p, bp, smem, dev, stream);
}

}  // namespace ffi
