// Forward of the fixed-fan-in sparse layer, barrier-free variant for the common case
// (fp32 storage, x tile resident in shared memory).
//
// Same arithmetic as ffi_fwd_kernel (forward.cu), but every warp is its own pipeline: it owns a private double buffer for the W/idx rows of
// the next row pair (filled by the warp's own cp.async: 2 rows x (W + idx) of K=32 are
// exactly one 16-byte copy per lane) and a private 4-row result tile, so the steady state
// has no CTA-wide barrier at all and the shared-memory pipe never drains at tile edges.
// Warps take row quads round-robin over the whole grid.  Results leave through the
// private tile as 16-byte runs along o (4 consecutive outputs per batch row).
#include "ffi_common.cuh"

namespace ffi {
namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;

struct FwdStreamParams {
    const float* xT;
    long long ldx;
    const int* idx;
    const float* W;
    const float* bias;
    float* y;
    int B, N, L, K;
    int Kp;  // K rounded up to a multiple of 4: row stride in the warps' buffers
    // fused sigmoid-BCE epilogue (BCE variant): instead of y the kernel writes the loss gradient,
    // already transposed, gT[o][b] = scale * sigmoid(z[b,o]) (positives are corrected afterwards),
    // and one partial sum of softplus(z) per CTA
    float* gT;
    long long ldg;
    float scale;
    double* loss_partials;
    int loss_kind;  // ffi_loss_kind: BCE, squared hinge or hinge (for target 0; positives are corrected afterwards)
    // top-k epilogue: every warp keeps, per batch element of the tile, the kTopK best logits of the
    // rows it computed; lists [tile][cta][warp][batch][kTopK] of (value, row) go to `topk_lists`
    uint2* topk_lists;
    // per batch column and group of warps (one in kTopK), the highest logit seen so far (order_key).  The lowest of a column's
    // kTopK groups is a bound: that many logits reach it, so a row pair whose logits all lie below it is done with.  Without
    // it every warp sorts its own few hundred rows (0.60 ms at B=128, N=768, L=670,091, K=32); with the best kTopK-th value
    // of any warp as the bound, which two logits in a thousand still pass, 0.51 ms; with this one, passed by about twenty per
    // column in all, 0.48 ms.  nullptr: few rows per warp, no sharing.
    int* topk_floor;
    int topk_stride;  // columns per group
};

// Bounds are kept as order_key; the memset value kFloorNone decodes to "no bound yet".
constexpr int kFloorNone = static_cast<int>(0x80808080u);
__device__ __forceinline__ float floor_value(int k) {
    return k == kFloorNone ? -INFINITY : order_value(k);
}

// A HALF warp covers the batch tile (16 lanes x VPL batch elements) and the two halves of a warp
// work on the two rows of a row pair at once.  The fetch of a row's W and idx values is then one
// shared-memory access for both rows (two addresses, one per half) instead of a warp-uniform access
// per row; against a whole warp per row this took a fifth off the traffic of the shared-memory pipe,
// the unit this kernel is bound by (0.56 -> 0.48 ms at B=128, N=768, L=670,091, K=32).
// x tile in natural order: x_s[i][b].
template <int VPL>
__device__ __forceinline__ int pair_column(int q, int j) {
    if constexpr (VPL == 8) return j < 4 ? 4 * q + j : 64 + 4 * q + (j - 4);
    else return VPL * q + j;
}

// (Keeping the indices as 16-bit values in the warp's buffer, four per 8-byte access, was measured:
// the repacking on the way in costs more than the narrower fetch saves, 0.50 vs 0.48 ms.)
//
// ODD: K is not a multiple of 4, or W or idx not 16-byte aligned.  The rows are then copied with 4-byte cp.async into the same
// 16-byte aligned rows of the buffer (K/8 copies per lane and row pair, a tenth of the instructions of a pair), so the loop
// reads them four entries at a time all the same; the K % 4 last ones singly, for a padding entry of weight 0 would still
// turn an infinite x into a NaN.  Such shapes went to the kernel with CTA-wide tiles before.
template <int VPL, int MODE, bool ODD>
__global__ void __launch_bounds__(kThreads, 1) ffi_fwd_pair_kernel(FwdStreamParams p) {
    chain_wait();
    constexpr bool BCE = MODE == 1;  // 0: write y; 1: loss epilogue; 2: running top-k of the logits
    constexpr int BT = 16 * VPL;
    constexpr int S = BT + 8;  // result-tile row stride: 16-byte rows, conflict-free for both access patterns
    extern __shared__ __align__(16) unsigned char smem_raw[];

    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int h = lane >> 4;  // which row of a pair
    const int q = lane & 15;
    const int b0 = blockIdx.y * BT;
    const int K = p.K, L = p.L, Kp = ODD ? p.Kp : p.K;

    float* x_s = reinterpret_cast<float*>(smem_raw);
    const int regionWords = 8 * Kp + 4 * S;
    float* region = x_s + static_cast<size_t>(p.N) * BT + static_cast<size_t>(warp) * regionWords;
    float* wi = region;
    float* ys = region + 8 * Kp;

    const float* xs_lane = x_s + (VPL == 8 ? 4 : VPL) * q;
    const long long numQuads = (static_cast<long long>(L) + 3) / 4;
    const long long gw = static_cast<long long>(blockIdx.x) * kWarps + warp;
    const long long GW = static_cast<long long>(gridDim.x) * kWarps;
    const int chunksPerRow = K / 2;
    const int nChunks = 2 * chunksPerRow;

    auto issue = [&](long long pr, int buf) {
        float* dstbuf = wi + buf * 4 * Kp;
        if constexpr (ODD) {
            const long long e0 = 2 * pr * K;
            const int n = 2 * pr + 1 < L ? 2 * K : K;  // both rows, or the one row left of an odd L
            for (int c = lane; c < n; c += 32) {
                float* dst = dstbuf + c + (c >= K ? 2 * Kp - K : 0);
                __pipeline_memcpy_async(dst, p.W + e0 + c, 4);
                __pipeline_memcpy_async(dst + Kp, p.idx + e0 + c, 4);
            }
        } else {
            for (int c = lane; c < nChunks; c += 32) {
                const int row = c / chunksPerRow;
                const int within = c - row * chunksPerRow;
                const bool isIdx = within >= K / 4;
                const int kc = isIdx ? within - K / 4 : within;
                const long long o = 2 * pr + row;
                if (o < L) {
                    const void* src = isIdx ? static_cast<const void*>(p.idx + o * K + 4 * kc)
                                            : static_cast<const void*>(p.W + o * K + 4 * kc);
                    __pipeline_memcpy_async(dstbuf + row * 2 * K + (isIdx ? K : 0) + 4 * kc, src, 16);
                }
            }
        }
        __pipeline_commit();
    };

    // the warp's first W/idx rows are requested before the x tile is filled: both trips to memory overlap
    long long qd = gw;
    if (qd < numQuads) issue(2 * qd, 0);

    if (p.ldx % 4 == 0 && b0 + BT <= p.B && reinterpret_cast<uintptr_t>(p.xT) % 16 == 0) {
        // whole tile inside the batch, rows 16-byte aligned: 16-byte loads and stores
        constexpr int VR = BT / 4;
        const int total = p.N * VR;
#pragma unroll 12
        for (int e = tid; e < total; e += kThreads) {
            const int i = e / VR;
            const int v = e - i * VR;
            reinterpret_cast<float4*>(x_s)[e] =
                __ldg(reinterpret_cast<const float4*>(p.xT + static_cast<size_t>(i) * p.ldx + b0) + v);
        }
    } else {
        // ragged rows: 4-byte asynchronous copies, all of a thread's in flight at once (the zero-filled ones read nothing)
        const int total = p.N * BT;
        for (int e = tid; e < total; e += kThreads) {
            const int i = e / BT;
            const int b = b0 + e - i * BT;
            const bool in = b < p.B;
            __pipeline_memcpy_async(x_s + e, in ? p.xT + static_cast<size_t>(i) * p.ldx + b : p.xT, 4, in ? 0 : 4);
        }
        __pipeline_commit();
        __pipeline_wait_prior(0);
    }
    __syncthreads();

    int s = 0;
    float loss_local = 0.f;
    // top-k mode: lane keeps the lists of batch columns lane, lane + 32, ... of the tile
    constexpr int TM = MODE == 2 ? (BT + 31) / 32 : 1;
    float tv[TM][kTopK];
    int ti[TM][kTopK];
#pragma unroll
    for (int m = 0; m < TM; ++m)
#pragma unroll
        for (int j = 0; j < kTopK; ++j) tv[m][j] = -INFINITY, ti[m][j] = 0x7fffffff;
    int fq[VPL];  // MODE 2: bounds of the columns this lane computes
#pragma unroll
    for (int j = 0; j < VPL; ++j) fq[j] = kFloorNone;
    int turn = 0;
    for (; qd < numQuads; qd += GW) {
        if constexpr (MODE == 2) {
            if (p.topk_floor && (turn++ & 7) == 0) {  // the shared bounds of this lane's columns, now and then
#pragma unroll
                for (int j = 0; j < VPL; ++j) fq[j] = 0x7fffffff;
#pragma unroll
                for (int g = 0; g < kTopK; ++g) {
                    const int* src = p.topk_floor + g * p.topk_stride + b0;
#pragma unroll
                    for (int j = 0; j < VPL; j += 2) {
                        const int2 t = __ldcg(reinterpret_cast<const int2*>(src + pair_column<VPL>(q, j)));
                        fq[j] = min(fq[j], t.x), fq[j + 1] = min(fq[j + 1], t.y);
                    }
                }
#pragma unroll
                for (int j = 0; j < VPL; ++j)  // nothing passes in the padded columns
                    if (b0 + pair_column<VPL>(q, j) >= p.B) fq[j] = order_key(INFINITY);
            }
        }
#pragma unroll
        for (int half = 0; half < 2; ++half, ++s) {
            const int buf = s & 1;
            const long long pr = 2 * qd + half;
            const long long nextPr = half == 0 ? pr + 1 : 2 * (qd + GW);
            const bool haveNext = half == 0 ? (2 * nextPr < L) : (qd + GW < numQuads);
            if (haveNext) {
                issue(nextPr, buf ^ 1);
                __pipeline_wait_prior(1);
            } else {
                __pipeline_wait_prior(0);
            }
            __syncwarp();

            const long long oA = 2 * pr;
            if (oA < L) {
                const bool mine = oA + h < L;       // false only for the missing second row of an odd L
                const long long o = mine ? oA + h : oA;
                const float* row = wi + buf * 4 * Kp + (mine ? h : 0) * 2 * Kp;
                const float4* wr = reinterpret_cast<const float4*>(row);
                const int4* ir = reinterpret_cast<const int4*>(row + Kp);
                const float bias = p.bias ? __ldg(p.bias + o) : 0.f;
                float acc[VPL];
#pragma unroll
                for (int j = 0; j < VPL; ++j) acc[j] = 0.f;
#pragma unroll 2
                for (int k4 = 0; k4 < K / 4; ++k4) {
                    const int4 i4 = ir[k4];
                    const float4 w4 = wr[k4];
                    const int ii[4] = {i4.x, i4.y, i4.z, i4.w};
                    const float ww[4] = {w4.x, w4.y, w4.z, w4.w};
                    float a[4][VPL];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const float* src = xs_lane + ii[u] * BT;
                        if constexpr (VPL == 2) {
                            const float2 t = *reinterpret_cast<const float2*>(src);
                            a[u][0] = t.x, a[u][1] = t.y;
                        } else {
                            const float4 t = *reinterpret_cast<const float4*>(src);
                            a[u][0] = t.x, a[u][1] = t.y, a[u][2] = t.z, a[u][3] = t.w;
                            if constexpr (VPL == 8) {
                                const float4 t2 = *reinterpret_cast<const float4*>(src + 64);
                                a[u][4] = t2.x, a[u][5] = t2.y, a[u][6] = t2.z, a[u][7] = t2.w;
                            }
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u)
#pragma unroll
                        for (int j = 0; j < VPL; ++j) acc[j] = fmaf(ww[u], a[u][j], acc[j]);
                }
                if constexpr (ODD) {
                    for (int k = K & ~3; k < K; ++k) {
                        const float w = row[k];
                        const float* src = xs_lane + __float_as_int(row[Kp + k]) * BT;
                        if constexpr (VPL == 2) {
                            const float2 t = *reinterpret_cast<const float2*>(src);
                            acc[0] = fmaf(w, t.x, acc[0]), acc[1] = fmaf(w, t.y, acc[1]);
                        } else {
#pragma unroll
                            for (int v = 0; v < VPL / 4; ++v) {
                                const float4 t = *reinterpret_cast<const float4*>(src + 64 * v);
                                acc[4 * v] = fmaf(w, t.x, acc[4 * v]), acc[4 * v + 1] = fmaf(w, t.y, acc[4 * v + 1]);
                                acc[4 * v + 2] = fmaf(w, t.z, acc[4 * v + 2]), acc[4 * v + 3] = fmaf(w, t.w, acc[4 * v + 3]);
                            }
                        }
                    }
                }
                if constexpr (BCE) {
                    // a lane holds runs of 4 (or 2) consecutive batch elements of its row: vector stores
#pragma unroll
                    for (int j0 = 0; j0 < VPL; j0 += (VPL == 2 ? 2 : 4)) {
                        constexpr int W4 = VPL == 2 ? 2 : 4;
                        const int b = b0 + pair_column<VPL>(q, j0);
                        float gv[W4];
#pragma unroll
                        for (int j = 0; j < W4; ++j) {
                            const bool live = b + j < p.B;
                            float v, g;
                            loss_for_negative(p.loss_kind, acc[j0 + j] + bias, v, g);
                            if (live && mine) loss_local += v;
                            gv[j] = live ? p.scale * g : 0.f;
                        }
                        if (mine && b < p.ldg) {
                            float* dst = p.gT + static_cast<size_t>(o) * p.ldg + b;
                            if constexpr (W4 == 4) *reinterpret_cast<float4*>(dst) = make_float4(gv[0], gv[1], gv[2], gv[3]);
                            else *reinterpret_cast<float2*>(dst) = make_float2(gv[0], gv[1]);
                        }
                    }
                    if (mine && blockIdx.y + 1 == gridDim.y)  // the last tile clears the columns past it, too
                        for (long long b = b0 + BT + 4 * q; b < p.ldg; b += 64)
                            *reinterpret_cast<float4*>(p.gT + static_cast<size_t>(o) * p.ldg + b) = make_float4(0.f, 0.f, 0.f, 0.f);
                } else if constexpr (MODE == 2) {
                    bool hit = p.topk_floor == nullptr;
#pragma unroll
                    for (int j = 0; j < VPL; ++j) hit |= acc[j] + bias >= floor_value(fq[j]);
                    if (__any_sync(0xffffffffu, hit)) {
                        float* yrow = ys + h * S;
#pragma unroll
                        for (int j = 0; j < VPL; ++j) yrow[pair_column<VPL>(q, j)] = acc[j] + bias;
                        __syncwarp();
#pragma unroll
                        for (int m = 0; m < TM; ++m) {
                            const int bl = lane + 32 * m;
                            if (bl < BT && b0 + bl < p.B) {
                                const float best = tv[m][0];
#pragma unroll
                                for (int oo = 0; oo < 2; ++oo)
                                    if (oA + oo < L) topk_insert(tv[m], ti[m], ys[oo * S + bl], static_cast<int>(oA) + oo);
                                if (p.topk_floor && tv[m][0] > best)
                                    atomicMax(p.topk_floor + (gw % kTopK) * p.topk_stride + b0 + bl, order_key(tv[m][0]));
                            }
                        }
                    }
                } else {
                    float* yrow = ys + (2 * half + h) * S;
#pragma unroll
                    for (int j = 0; j < VPL; ++j) yrow[pair_column<VPL>(q, j)] = acc[j] + bias;
                }
            }
            __syncwarp();
        }
        if constexpr (MODE == 0) {
            const long long oq = 4 * qd;
#pragma unroll
            for (int it = 0; it < BT * 4 / 32; ++it) {
                const int id = it * 32 + lane;
                const int bl = id >> 2, oo = id & 3;
                if (b0 + bl < p.B && oq + oo < L)
                    p.y[static_cast<size_t>(b0 + bl) * L + oq + oo] = ys[oo * S + bl];
            }
            __syncwarp();
        }
    }
    __pipeline_wait_prior(0);

    if constexpr (MODE == 2) {
        uint2* out = p.topk_lists +
                     ((static_cast<size_t>(blockIdx.y) * gridDim.x + blockIdx.x) * kWarps + warp) * (BT * kTopK);
#pragma unroll
        for (int m = 0; m < TM; ++m) {
            const int bl = lane + 32 * m;
            if (bl < BT)
#pragma unroll
                for (int j = 0; j < kTopK; ++j)
                    out[bl * kTopK + j] = make_uint2(__float_as_uint(tv[m][j]), static_cast<unsigned>(ti[m][j]));
        }
    }

    if constexpr (BCE) {
        double v = static_cast<double>(loss_local);
#pragma unroll
        for (int off = 16; off >= 1; off /= 2) v += __shfl_xor_sync(0xffffffffu, v, off);
        __syncthreads();
        double* red = reinterpret_cast<double*>(smem_raw);
        if (lane == 0) red[warp] = v;
        __syncthreads();
        clear_loss_ticket(p.loss_partials);
        if (tid == 0) {
            double t = 0.0;
            for (int w = 0; w < kWarps; ++w) t += red[w];
            p.loss_partials[static_cast<size_t>(blockIdx.y) * gridDim.x + blockIdx.x] = t;
        }
    }
}

template <int VPL, int MODE, bool ODD>
int launch_pair_t(const FwdStreamParams& p, size_t smem, int nBT, const DeviceInfo& dev, cudaStream_t stream,
                  int* ctas_out) {
    auto kern = ffi_fwd_pair_kernel<VPL, MODE, ODD>;
    int occ = 0;
    FFI_CUDA_CHECK(prepare_kernel(reinterpret_cast<const void*>(kern), kThreads, smem, &occ));
    if (occ < 1) return fail(FFI_ERR_CUDA, "streaming forward kernel does not fit on an SM (smem %zu)", smem);
    // The epilogue variants write one record per CTA (loss partial, top-k lists) into scratch that is
    // sized for one CTA per SM, whatever occupancy the kernel would allow.
    if (MODE != 0) occ = 1;
    int per_bt = dev.sm_count * occ / nBT;
    if (per_bt < 1) per_bt = 1;
    const long long numQuads = (static_cast<long long>(p.L) + 3) / 4;
    const long long want = (numQuads + kWarps - 1) / kWarps;
    dim3 grid(static_cast<unsigned>(want < per_bt ? want : per_bt), static_cast<unsigned>(nBT));
    if (MODE == 1 && static_cast<size_t>(grid.x) * grid.y > static_cast<size_t>(kMaxLossPartials))
        return fail(FFI_ERR_UNSUPPORTED, "the fused loss keeps at most %d per-CTA partials; this batch needs %u",
                    kMaxLossPartials, grid.x * grid.y);
    if (ctas_out) *ctas_out = static_cast<int>(grid.x * grid.y);
    FFI_CUDA_CHECK(launch_chained(kern, grid, dim3(kThreads), smem, stream, p));
    FFI_LAUNCH_CHECK("ffi_fwd_pair_kernel");
    return FFI_OK;
}

template <int MODE, bool ODD>
int launch_pair(const FwdStreamParams& p, size_t smem, int nBT, int bpl, const DeviceInfo& dev, cudaStream_t stream, int* ctas_out) {
    if (bpl == 4) return launch_pair_t<8, MODE, ODD>(p, smem, nBT, dev, stream, ctas_out);
    if (bpl == 2) return launch_pair_t<4, MODE, ODD>(p, smem, nBT, dev, stream, ctas_out);
    return launch_pair_t<2, MODE, ODD>(p, smem, nBT, dev, stream, ctas_out);
}

}  // namespace

// Shared launcher: BCE epilogue when bce != nullptr.
struct BceEpilogue {
    float* gT;
    long long ldg;
    float scale;
    double* loss_partials;
    int* ctas;  // out: number of CTAs = number of loss partials written
    int loss_kind;
};
struct TopkEpilogue {
    uint2* lists;  // scratch from forward_topk_workspace_bytes
    int* ctas_x;   // out: CTAs per batch tile
    int* bt;       // out: batch tile width
    int* floor;    // [kTopK][batch padded to whole tiles] shared bounds, cleared by the launcher
};

static int launch_forward_stream_impl(const FwdArgs& a, const BceEpilogue* bce, const TopkEpilogue* topk,
                                      cudaStream_t stream, bool* handled) {
    *handled = false;
    DeviceInfo dev;
    int rc = get_device_info(&dev);
    if (rc != FFI_OK) return rc;
    if (a.bf16) return FFI_OK;  // this kernel reads fp32 only
    const int Kp = static_cast<int>(round_up(a.K, 4));
    const bool odd = a.K % 4 != 0 || reinterpret_cast<uintptr_t>(a.W) % 16 != 0 || reinterpret_cast<uintptr_t>(a.idx) % 16 != 0;
    // Width of the batch tiles: the one with the least work for the busiest warp, counted in accesses of the shared-memory
    // pipe per row pair (per four entries the gathers, W and idx and their copies; the results; about 20 for the rest) times
    // its rounds over the table.  A long table takes the widest tile that fits; a short one, whose row quads do not fill the
    // warps, narrower ones: B=127, N=254, L=513, K=73 had 9 CTAs of 128 columns (13.8 us with CTA-wide tiles), now 36 of 32
    // (7.7 us); B=418, N=228, L=2,578, K=16 15.3 -> 8.7 us in tiles of 64.  A narrower tile has to promise a tenth, for it
    // fetches W and idx more often (B=152, L=31,964, K=8: promised 5 %, 22 -> 25 us).
    int bpl = 0;
    size_t smem = 0;
    double least = 0;
    for (int c = a.B <= 32 ? 1 : (a.B <= 64 ? 2 : 4); c >= 1; c /= 2) {
        const size_t BT = 32 * c;
        const size_t need = static_cast<size_t>(a.N) * BT * 4 + static_cast<size_t>(kWarps) * (8 * Kp + 4 * (BT + 8)) * 4;
        if (need > static_cast<size_t>(dev.max_smem_optin)) continue;
        const int64_t per_bt = dev.sm_count / ceil_div(a.B, BT) > 0 ? dev.sm_count / ceil_div(a.B, BT) : 1;
        const double cost = ((BT / 4 + 2.5) * Kp / 4 + BT / 4 + 20) * static_cast<double>(ceil_div(ceil_div(a.L, 4), per_bt * kWarps) * ceil_div(ceil_div(a.B, BT) * per_bt, dev.sm_count));
        if (bpl == 0 || cost < 0.9 * least) bpl = c, smem = need, least = cost;
    }
    if (bpl < 1) return FFI_OK;
    FwdStreamParams p;
    p.xT = static_cast<const float*>(a.xT);
    p.ldx = a.ldx;
    p.idx = a.idx;
    p.W = static_cast<const float*>(a.W);
    p.bias = a.bias;
    p.y = a.y;
    p.B = a.B;
    p.N = a.N;
    p.L = a.L;
    p.K = a.K;
    p.Kp = Kp;
    p.gT = bce ? bce->gT : nullptr;
    p.ldg = bce ? bce->ldg : 0;
    p.scale = bce ? bce->scale : 0.f;
    p.loss_partials = bce ? bce->loss_partials : nullptr;
    p.loss_kind = bce ? bce->loss_kind : 0;
    p.topk_lists = topk ? topk->lists : nullptr;
    p.topk_floor = nullptr;
    p.topk_stride = 0;
    const int nBT = static_cast<int>(ceil_div(a.B, 32 * bpl));
    *handled = true;
    // same tile sizes and shared-memory footprint: BT = 32 * bpl = 16 * VPL
    if (topk) {
        int ctas = 0;
        // sharing pays once a warp sees more rows than its list has room for a few times over
        if (a.L >= 8 * kTopK * kWarps * dev.sm_count / nBT) {
            p.topk_stride = nBT * 32 * bpl;
            FFI_CUDA_CHECK(cudaMemsetAsync(topk->floor, 0x80, kTopK * static_cast<size_t>(p.topk_stride) * sizeof(int), stream));
            p.topk_floor = topk->floor;
        }
        rc = odd ? launch_pair<2, true>(p, smem, nBT, bpl, dev, stream, &ctas) : launch_pair<2, false>(p, smem, nBT, bpl, dev, stream, &ctas);
        *topk->ctas_x = ctas / nBT;
        *topk->bt = 32 * bpl;
        return rc;
    }
    if (bce)
        return odd ? launch_pair<1, true>(p, smem, nBT, bpl, dev, stream, bce->ctas) : launch_pair<1, false>(p, smem, nBT, bpl, dev, stream, bce->ctas);
    return odd ? launch_pair<0, true>(p, smem, nBT, bpl, dev, stream, nullptr) : launch_pair<0, false>(p, smem, nBT, bpl, dev, stream, nullptr);
}

// Launches the barrier-free kernel when the shape allows it; *handled tells the caller.
int launch_forward_stream(const FwdArgs& a, cudaStream_t stream, bool* handled) {
    return launch_forward_stream_impl(a, nullptr, nullptr, stream, handled);
}

// Forward with the fused sigmoid-BCE epilogue: writes gT[o][b] = scale * sigmoid(z[b,o]) (zero in the
// padded batch columns) and one partial of sum softplus(z) per CTA; *ctas receives their number
// (at most 2 * SM count).  *handled is false when the shape needs the unfused path.
int launch_forward_bce_stream(const FwdArgs& a, float* gT, int64_t ldg, float scale, double* loss_partials, int* ctas,
                              int loss_kind, cudaStream_t stream, bool* handled) {
    BceEpilogue e{gT, ldg, scale, loss_partials, ctas, loss_kind};
    return launch_forward_stream_impl(a, &e, nullptr, stream, handled);
}

int launch_forward_topk_tile(const FwdArgs& a, void* lists, int* lists_per_tile, int* bt, cudaStream_t stream);

int launch_topk_merge(const uint2* lists, int lists_per_tile, int bt, int B, int kk, int label_offset, float* top_val,
                      int* top_idx, cudaStream_t stream);

// Scratch for forward_topk: the warp lists (an upper bound over the grids the launcher may choose), then the shared bounds.
static size_t topk_list_bytes(int64_t B) {
    DeviceInfo dev;
    if (get_device_info(&dev) != FFI_OK) return 0;
    // tiles * CTAs per tile <= SM count (one CTA per SM), BT <= 128
    const size_t lists = static_cast<size_t>(dev.sm_count + ceil_div(B, 32)) * kWarps;
    return lists * 128 * kTopK * sizeof(uint2);
}
size_t forward_topk_workspace_bytes(int64_t B) { return topk_list_bytes(B) + kTopK * round_up(B, 128) * sizeof(int); }

// Forward whose epilogue keeps the best logits per batch element instead of writing y; top_val/top_idx
// [B][kk] receive them in tf.nn.top_k order (row + label_offset as the index).  *handled as above.
int launch_forward_topk_stream(const FwdArgs& a, void* scratch, float* top_val, int* top_idx, int kk, int label_offset,
                               cudaStream_t stream, bool* handled) {
    if (kk < 1 || kk > kTopK) return fail(FFI_ERR_UNSUPPORTED, "top-k supports 1 <= k <= %d", kTopK);
    int ctas_x = 0, bt = 0;
    int* floor = reinterpret_cast<int*>(static_cast<unsigned char*>(scratch) + topk_list_bytes(a.B));
    TopkEpilogue e{static_cast<uint2*>(scratch), &ctas_x, &bt, floor};
    int rc = launch_forward_stream_impl(a, nullptr, &e, stream, handled);
    if (rc != FFI_OK) return rc;
    int lists_per_tile = ctas_x * kWarps;
    if (!*handled) {  // wide inputs, bf16 storage: the CTA-tile kernel's top-k epilogue
        rc = launch_forward_topk_tile(a, scratch, &lists_per_tile, &bt, stream);
        if (rc != FFI_OK) return rc;
        *handled = true;
    }
    return launch_topk_merge(static_cast<const uint2*>(scratch), lists_per_tile, bt, a.B, kk, label_offset, top_val, top_idx,
                             stream);
}

}  // namespace ffi
