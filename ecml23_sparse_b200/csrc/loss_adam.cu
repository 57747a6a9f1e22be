// Sigmoid-BCE gradient against sparse multi-hot targets, and the fused Adam step.
//
// ffi_bce_grad replaces the loss graph SparseBinaryCrossEntropyLoss builds
// (sparse/metrics.py:132-139,167-173; sparse/utils.py:15-21: a dense
// sigmoid_cross_entropy_with_logits over all B*L logits with zero targets, positives
// patched in by scatter, mean over labels, then the Keras mean over the batch) together
// with its gradient, in one dense pass plus a pass over the few positives.
// ffi_adam_step replaces the per-variable elementwise kernels of keras.optimizers.Adam
// (the base class of SparseAdam, sparse/optimizer.py:9-12).
// Both reductions run in a fixed order: results are bit-reproducible.
#include "ffi_common.cuh"

namespace ffi {
namespace {

constexpr int kBceBlocks = 1184;  // 8 per SM on a 148-SM part; fixed so the sum order is fixed
constexpr int kBceThreads = 256;

__device__ __forceinline__ float softplus_f(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }
__device__ __forceinline__ float sigmoid_f(float z) { return 1.f / (1.f + expf(-z)); }

__device__ __forceinline__ double block_sum(double v, double* sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int off = 16; off >= 1; off /= 2) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (blockDim.x >> 5); ++w) t += sh[w];
    return t;  // valid in thread 0
}

// ws[0] = sum of z over the positives that fall in this shard.
__global__ void bce_positive_sum_kernel(const float* __restrict__ z, const int* __restrict__ row_ptr,
                                        const int* __restrict__ labels, int B, long long L,
                                        long long label_offset, double* __restrict__ ws) {
    __shared__ double sh[32];
    double s = 0.0;
    for (int b = 0; b < B; ++b) {
        const int lo = row_ptr[b], hi = row_ptr[b + 1];
        for (int e = lo + threadIdx.x; e < hi; e += blockDim.x) {
            const long long o = static_cast<long long>(labels[e]) - label_offset;
            if (o >= 0 && o < L) s += static_cast<double>(z[static_cast<size_t>(b) * L + o]);
        }
    }
    const double t = block_sum(s, sh);
    if (threadIdx.x == 0) ws[0] = t;
}

// g = scale * sigmoid(z) over the flat array; ws[1 + block] = sum softplus(z) of the block.
__global__ void __launch_bounds__(kBceThreads) bce_dense_kernel(const float* z, float* g, long long n,
                                                                float scale, double* __restrict__ ws,
                                                                int vec4) {
    __shared__ double sh[32];
    float local = 0.f;
    const long long tid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    if (vec4) {
        const long long n4 = n / 4;
        const float4* z4 = reinterpret_cast<const float4*>(z);
        float4* g4 = reinterpret_cast<float4*>(g);
        for (long long e = tid; e < n4; e += stride) {
            const float4 v = z4[e];
            local += (softplus_f(v.x) + softplus_f(v.y)) + (softplus_f(v.z) + softplus_f(v.w));
            g4[e] = make_float4(scale * sigmoid_f(v.x), scale * sigmoid_f(v.y), scale * sigmoid_f(v.z),
                                scale * sigmoid_f(v.w));
        }
        for (long long e = n4 * 4 + tid; e < n; e += stride) {
            const float v = z[e];
            local += softplus_f(v);
            g[e] = scale * sigmoid_f(v);
        }
    } else {
        for (long long e = tid; e < n; e += stride) {
            const float v = z[e];
            local += softplus_f(v);
            g[e] = scale * sigmoid_f(v);
        }
    }
    const double t = block_sum(static_cast<double>(local), sh);
    if (threadIdx.x == 0) ws[1 + blockIdx.x] = t;
}

// loss = scale * (sum of block partials - positive sum); g[b,label] -= scale at the positives.
__global__ void bce_finalize_kernel(const int* __restrict__ row_ptr, const int* __restrict__ labels,
                                    float* __restrict__ g, float* __restrict__ loss, int B, long long L,
                                    long long label_offset, float scale, const double* __restrict__ ws,
                                    int nPartials) {
    __shared__ double sh[32];
    for (int b = 0; b < B; ++b) {
        const int lo = row_ptr[b], hi = row_ptr[b + 1];
        for (int e = lo + threadIdx.x; e < hi; e += blockDim.x) {
            const long long o = static_cast<long long>(labels[e]) - label_offset;
            if (o >= 0 && o < L) g[static_cast<size_t>(b) * L + o] -= scale;
        }
    }
    if (loss) {
        double s = 0.0;
        for (int j = threadIdx.x; j < nPartials; j += blockDim.x) s += ws[1 + j];
        const double t = block_sum(s, sh);
        if (threadIdx.x == 0) *loss = static_cast<float>((t - ws[0]) * static_cast<double>(scale));
    }
}

// After the forward kernel with the fused loss epilogue, which took every target as 0: corrects gT at
// the positives (BCE: scale * (sigmoid(z) - 1); squared hinge: -2 * scale * max(0, 1 - z); hinge: -scale
// where z < 1), recomputing z of the few positive (b,o) pairs.  One block per sample; pos_partials[b] = the sample's sum of
// loss(z, target 1) - loss(z, target 0) over its positives (fixed order).  The last block to finish adds up
// loss = scale * (the forward kernel's CTA partials (all targets taken as 0) + the positives' corrections).
__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T>
__global__ void __launch_bounds__(256) bce_positive_fix_kernel(
    const T* __restrict__ xT, long long ldx, const int* __restrict__ idx, const T* __restrict__ W,
    const float* __restrict__ bias, const int* __restrict__ row_ptr, const int* __restrict__ labels,
    float* __restrict__ gT, long long ldg, double* pos_partials, float scale, long long L, int K,
    long long label_offset, int loss_kind, const double* __restrict__ partials, int nPartials, unsigned* ticket,
    float* __restrict__ loss) {
    chain_begin();
    __shared__ double sh[32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int b = blockIdx.x;
    double possum = 0.0;  // kept by lane 0 of each warp
    const int lo = row_ptr[b], hi = row_ptr[b + 1];
    for (int e = lo + warp; e < hi; e += nwarps) {
        const long long o = static_cast<long long>(labels[e]) - label_offset;
        if (o < 0 || o >= L) continue;
        // what the end needs is requested with the row: this kernel is a chain of trips to memory
        float* cell = gT + static_cast<size_t>(o) * ldg + b;
        const float bias_o = bias ? __ldg(bias + o) : 0.f, negative = loss_kind == 0 ? *cell : 0.f;
        float z = 0.f;
        for (int k = lane; k < K; k += 32) {
            const int i = idx[o * K + k];
            z = fmaf(to_f32(W[o * K + k]), to_f32(xT[static_cast<size_t>(i) * ldx + b]), z);
        }
#pragma unroll
        for (int off = 16; off >= 1; off /= 2) z += __shfl_xor_sync(0xffffffffu, z, off);
        if (lane == 0) {
            z += bias_o;
            // possum collects loss(target 1) - loss(target 0) of this logit
            if (loss_kind == 0) {
                possum -= static_cast<double>(z);
                *cell = negative - scale;
            } else {
                const float hp = fmaxf(1.f - z, 0.f), hn = fmaxf(1.f + z, 0.f);
                if (loss_kind == 1) {
                    possum += static_cast<double>(hp * hp) - static_cast<double>(hn * hn);
                    *cell = -2.f * hp * scale;
                } else {
                    possum += static_cast<double>(hp) - static_cast<double>(hn);
                    *cell = hp > 0.f ? -scale : 0.f;
                }
            }
        }
    }
    if (lane == 0) sh[warp] = possum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < nwarps; ++w) t += sh[w];
        pos_partials[b] = t;
        // the forward kernel cleared the ticket; the block that draws the last one adds everything up, in a fixed order
        __threadfence();
        last = loss && atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double s = 0.0;
    for (int j = threadIdx.x; j < nPartials; j += blockDim.x) s += partials[j];
    for (int j = threadIdx.x; j < static_cast<int>(gridDim.x); j += blockDim.x) s += __ldcg(pos_partials + j);
    const double t = block_sum(s, sh);
    if (threadIdx.x == 0) *loss = static_cast<float>(t * static_cast<double>(scale));
}

// grad_bias[o] = sum_b gT[o][b]: one warp per row of the transposed gradient, fixed lane tree.
__global__ void __launch_bounds__(256) bias_grad_rows_kernel(const float* __restrict__ gT, long long ldg,
                                                             long long L, float* __restrict__ gbias) {
    const int lane = threadIdx.x & 31;
    const long long o = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (o >= L) return;
    float s = 0.f;
    for (long long b = lane; b < ldg; b += 32) s += gT[static_cast<size_t>(o) * ldg + b];
#pragma unroll
    for (int off = 16; off >= 1; off /= 2) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) gbias[o] = s;
}

// Up to kAdamTensors parameters in one launch (a layer's weights and bias; a launch each, and another for the last n % 4
// elements, added 4 to 6 us to the step of a small layer).  HBM-bound: 28 (24 with bf16 weights) bytes per element,
// 16-byte accesses (8-byte to bf16 weights), 94 % of the measured copy bandwidth at 21.4 M elements.
constexpr int kAdamTensors = 8;
struct AdamTensor {
    void* w;
    float* m;
    float* v;
    const float* grad;
    long long n, n4;  // elements; groups of four with aligned accesses (0: none)
    int bf16;
    int blocks;       // blocks of the grid that work on it
};
struct AdamParams {
    AdamTensor t[kAdamTensors];
    float alpha, omb1, omb2, eps;
};

__device__ __forceinline__ float adam_update(float g, float& m, float& v, const AdamParams& p) {
    m += (g - m) * p.omb1;
    v += (g * g - v) * p.omb2;
    return p.alpha * m / (sqrtf(v) + p.eps);
}

__global__ void __launch_bounds__(256) adam_kernel(const __grid_constant__ AdamParams p) {
    chain_begin();
    int block = blockIdx.x, j = 0;
    while (block >= p.t[j].blocks) block -= p.t[j].blocks, ++j;
    const AdamTensor& t = p.t[j];
    const long long tid = static_cast<long long>(block) * 256 + threadIdx.x, stride = static_cast<long long>(t.blocks) * 256;
    float4* m4 = reinterpret_cast<float4*>(t.m);
    float4* v4 = reinterpret_cast<float4*>(t.v);
    const float4* g4 = reinterpret_cast<const float4*>(t.grad);
    for (long long e = tid; e < t.n4; e += stride) {
        const float4 g = g4[e];
        float4 m = m4[e], v = v4[e], w;
        if (t.bf16) {
            const uint2 r = static_cast<const uint2*>(t.w)[e];
            w = make_float4(bf16_lo(r.x), bf16_hi(r.x), bf16_lo(r.y), bf16_hi(r.y));
        } else {
            w = static_cast<const float4*>(t.w)[e];
        }
        w.x -= adam_update(g.x, m.x, v.x, p);
        w.y -= adam_update(g.y, m.y, v.y, p);
        w.z -= adam_update(g.z, m.z, v.z, p);
        w.w -= adam_update(g.w, m.w, v.w, p);
        m4[e] = m;
        v4[e] = v;
        if (t.bf16) {
            auto pack = [](float lo, float hi) {
                return __bfloat16_as_ushort(__float2bfloat16_rn(lo)) |
                       (static_cast<unsigned>(__bfloat16_as_ushort(__float2bfloat16_rn(hi))) << 16);
            };
            static_cast<uint2*>(t.w)[e] = make_uint2(pack(w.x, w.y), pack(w.z, w.w));
        } else {
            static_cast<float4*>(t.w)[e] = w;
        }
    }
    for (long long e = 4 * t.n4 + tid; e < t.n; e += stride) {
        const float upd = adam_update(t.grad[e], t.m[e], t.v[e], p);
        if (t.bf16) {
            __nv_bfloat16* w = static_cast<__nv_bfloat16*>(t.w) + e;
            *w = __float2bfloat16_rn(__bfloat162float(*w) - upd);
        } else {
            static_cast<float*>(t.w)[e] -= upd;
        }
    }
}

}  // namespace
}  // namespace ffi

namespace ffi {
namespace {
__global__ void __launch_bounds__(256) widen_bf16_kernel(const __nv_bfloat16* __restrict__ src, float* __restrict__ dst,
                                                         long long n) {
    chain_begin();
    const long long tid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    for (long long e = tid; e < n; e += stride) dst[e] = __bfloat162float(src[e]);
}
}  // namespace

// bf16 -> fp32 (exact).
int launch_widen_bf16(const void* src, float* dst, int64_t n, cudaStream_t stream) {
    const long long blocks = (n + 255) / 256;
    const dim3 grid(static_cast<unsigned>(blocks < 1184 * 4 ? (blocks < 1 ? 1 : blocks) : 1184 * 4));
    FFI_CUDA_CHECK(launch_chained(widen_bf16_kernel, grid, dim3(256), 0, stream, static_cast<const __nv_bfloat16*>(src), dst,
                                  static_cast<long long>(n)));
    FFI_LAUNCH_CHECK("widen_bf16_kernel");
    return FFI_OK;
}

// xT and W are fp32, or bf16 when `bf16` is set.
int launch_bce_positive_fix(const void* xT, int64_t ldx, const int* idx, const void* W, const float* bias,
                            const int* row_ptr, const int* labels, float* gT, int64_t ldg, float* loss,
                            const double* partials, int nPartials, double* pos_partials, float scale, int B,
                            int64_t L, int K, int64_t label_offset, int loss_kind, bool bf16, cudaStream_t stream) {
    unsigned* ticket = loss_ticket(const_cast<double*>(partials));
    auto launch = [&](auto kern, const auto* x, const auto* w) {
        return launch_chained(kern, dim3(static_cast<unsigned>(B)), dim3(256), 0, stream, x, static_cast<long long>(ldx), idx, w, bias, row_ptr,
                              labels, gT, static_cast<long long>(ldg), pos_partials, scale, static_cast<long long>(L), K,
                              static_cast<long long>(label_offset), loss_kind, partials, nPartials, ticket, loss);
    };
    FFI_CUDA_CHECK(bf16 ? launch(bce_positive_fix_kernel<__nv_bfloat16>, static_cast<const __nv_bfloat16*>(xT), static_cast<const __nv_bfloat16*>(W))
                        : launch(bce_positive_fix_kernel<float>, static_cast<const float*>(xT), static_cast<const float*>(W)));
    FFI_LAUNCH_CHECK("bce_positive_fix_kernel");
    return FFI_OK;
}

int launch_bias_grad_rows(const float* gT, int64_t ldg, int64_t L, float* gbias, cudaStream_t stream) {
    bias_grad_rows_kernel<<<static_cast<unsigned>(ceil_div(L, 8)), 256, 0, stream>>>(gT, ldg, L, gbias);
    FFI_LAUNCH_CHECK("bias_grad_rows_kernel");
    return FFI_OK;
}
}  // namespace ffi

using namespace ffi;

extern "C" size_t ffi_bce_workspace_bytes(int64_t, int64_t) { return (1 + kBceBlocks) * sizeof(double); }

extern "C" int ffi_bce_grad(const float* z, const int32_t* row_ptr, const int32_t* labels, float* g,
                            float* loss, int64_t B, int64_t L, int64_t L_total, int64_t label_offset,
                            void* workspace, size_t workspace_bytes, void* stream_v) {
    FFI_TRACE("ffi_bce_grad");
    if (!z || !row_ptr || !labels || !g) return fail(FFI_ERR_INVALID_ARGUMENT, "NULL argument to ffi_bce_grad");
    if (B <= 0 || L <= 0 || L_total < L || B >= (1LL << 31))
        return fail(FFI_ERR_INVALID_ARGUMENT, "bad shape B=%lld L=%lld L_total=%lld", (long long)B,
                    (long long)L, (long long)L_total);
    if (!workspace || workspace_bytes < ffi_bce_workspace_bytes(B, L) ||
        reinterpret_cast<uintptr_t>(workspace) % 8 != 0)
        return fail(FFI_ERR_WORKSPACE, "ffi_bce_grad needs %zu bytes of 8-byte aligned workspace",
                    ffi_bce_workspace_bytes(B, L));
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    double* ws = static_cast<double*>(workspace);
    const float scale = static_cast<float>(1.0 / (static_cast<double>(B) * static_cast<double>(L_total)));
    const long long n = B * L;
    bce_positive_sum_kernel<<<1, 256, 0, stream>>>(z, row_ptr, labels, static_cast<int>(B), L, label_offset, ws);
    const int vec4 = reinterpret_cast<uintptr_t>(z) % 16 == 0 && reinterpret_cast<uintptr_t>(g) % 16 == 0;
    bce_dense_kernel<<<kBceBlocks, kBceThreads, 0, stream>>>(z, g, n, scale, ws, vec4);
    bce_finalize_kernel<<<1, 256, 0, stream>>>(row_ptr, labels, g, loss, static_cast<int>(B), L, label_offset,
                                               scale, ws, kBceBlocks);
    FFI_LAUNCH_CHECK("bce kernels");
    return FFI_OK;
}

extern "C" int ffi_adam_step_group(const ffi_adam_tensor* tensors, int count, float lr, float beta1, float beta2, float eps,
                                   int64_t step, void* stream_v) {
    FFI_TRACE("ffi_adam_step_group");
    if (!tensors) return fail(FFI_ERR_INVALID_ARGUMENT, "NULL argument to ffi_adam_step_group");
    if (count < 1 || step < 1) return fail(FFI_ERR_INVALID_ARGUMENT, "count and step must be >= 1");
    for (int j = 0; j < count; ++j) {
        const ffi_adam_tensor& t = tensors[j];
        if (!t.w || !t.m || !t.v || !t.grad) return fail(FFI_ERR_INVALID_ARGUMENT, "NULL tensor passed to the Adam step");
        if (t.n <= 0) return fail(FFI_ERR_INVALID_ARGUMENT, "n must be positive");
        if (t.dtype != FFI_F32 && t.dtype != FFI_BF16) return fail(FFI_ERR_UNSUPPORTED, "unknown dtype %d", t.dtype);
    }
    DeviceInfo dev;
    const int rc = get_device_info(&dev);
    if (rc != FFI_OK) return rc;
    AdamParams p;
    const double t = static_cast<double>(step);
    p.alpha = static_cast<float>(static_cast<double>(lr) * sqrt(1.0 - pow(static_cast<double>(beta2), t)) /
                                 (1.0 - pow(static_cast<double>(beta1), t)));
    p.omb1 = 1.f - beta1;
    p.omb2 = 1.f - beta2;
    p.eps = eps;
    for (int first = 0; first < count; first += kAdamTensors) {
        const int n = count - first < kAdamTensors ? count - first : kAdamTensors;
        int64_t elements = 0;
        for (int j = 0; j < n; ++j) elements += tensors[first + j].n;
        // eight blocks per SM over all tensors, in proportion to their sizes; no more than one block per 1024 elements
        int64_t grid = 0;
        for (int j = 0; j < n; ++j) {
            const ffi_adam_tensor& in = tensors[first + j];
            AdamTensor& out = p.t[j];
            const uintptr_t a16 = reinterpret_cast<uintptr_t>(in.m) | reinterpret_cast<uintptr_t>(in.v) |
                                  reinterpret_cast<uintptr_t>(in.grad);
            const bool aligned = a16 % 16 == 0 && reinterpret_cast<uintptr_t>(in.w) % (in.dtype == FFI_BF16 ? 8 : 16) == 0;
            out.w = in.w;
            out.m = in.m;
            out.v = in.v;
            out.grad = in.grad;
            out.n = in.n;
            out.n4 = aligned ? in.n / 4 : 0;
            out.bf16 = in.dtype == FFI_BF16;
            const int64_t share = ceil_div(static_cast<int64_t>(dev.sm_count) * 8 * (in.n / 1024 + 1), elements / 1024 + 1);
            const int64_t most = ceil_div(in.n, 1024);
            out.blocks = static_cast<int>(share < most ? share : most);
            grid += out.blocks;
        }
        FFI_CUDA_CHECK(launch_chained(adam_kernel, dim3(static_cast<unsigned>(grid)), dim3(256), 0, static_cast<cudaStream_t>(stream_v), p));
        FFI_LAUNCH_CHECK("adam_kernel");
    }
    return FFI_OK;
}

extern "C" int ffi_adam_step(void* w, float* m, float* v, const float* grad, int64_t n, float lr, float beta1,
                             float beta2, float eps, int64_t step, int dtype, void* stream_v) {
    FFI_TRACE("ffi_adam_step");
    if (!w || !m || !v || !grad) return fail(FFI_ERR_INVALID_ARGUMENT, "NULL argument to ffi_adam_step");
    if (n <= 0 || step < 1) return fail(FFI_ERR_INVALID_ARGUMENT, "n must be positive and step >= 1");
    const ffi_adam_tensor t{w, m, v, grad, n, dtype};
    return ffi_adam_step_group(&t, 1, lr, beta1, beta2, eps, step, stream_v);
}
