// grad_x and grad_W (and grad_bias) of the fixed-fan-in sparse layer in ONE pass over the transposed index, for wide
// inputs (x does not fit shared memory, an input has too few entries per chunk for the kernel of backward_fused.cu):
//   grad_x[b,i] = sum over entries (o,k) with idx[o,k]==i of W[o,k] * g[b,o]
//   grad_W[o,k] = sum_b g[b,o] * x[b, idx[o,k]],   grad_bias[o] = sum_b g[b,o]
//
// Replaces, for the output layers of the stacked configurations (hidden widths of 32,768 ... 100,000), both halves of the
// reference's grad functor (tfsparse/cc/kernels/backward.cu:112-133).
//
// What bounds these shapes is the bytes that cross the L2-to-SM fabric (64 bytes a clock into each SM) and the L1 data pipe they
// pass through: two separate kernels gather a row of g per entry for grad_x and a row of x per entry for grad_W.  A warp that
// walks the entries of ONE input keeps x[:, i] in registers, so the row of g it gathers serves both.
//
// What makes that pay:
//  - The order.  The outputs are cut into chunks whose rows of gT fit L2 (one launch each, which keeps the warps together): the
//    gathers hit L2, and the 4-byte stores of grad_W, which scatter over the chunk's rows, meet in L2 until their sectors are
//    complete.  A launch finds its entries of an input where the one before stopped (a cursor per input: the entries are sorted
//    by output), and adds its part of grad_x by reductions in L2; an input belongs to one warp of a launch, so the order of
//    additions is fixed.
//  - Registers and L1.  32 warps per SM with two steps' rows in flight each saturate the fabric; 24 warps, spills or less L1 for the
//    rows in flight cost 10 to 50 %.  See WarpScratch.
//  - The data pipe.  With up to 128 columns a group of lanes narrower than a warp covers an entry's row, 8 columns per lane: fewer
//    partial dots to store and add, fewer reads of outputs and weights (7.7 wavefronts an entry against 10.2 with a warp per entry
//    and 4 columns per lane: 842 against 982 us at B=128).
//
// Backward with grad_bias from the transposed gradient, before (two kernels) -> now, us: B=128, N=32,768, L=670,091, K=32 fp32
// 1,340 -> 844; B=256, N=65,536, L=501,070, K=32 bf16 1,630 -> 1,313; B=512, N=100,000, L=83,762, K=72 bf16 1,185 -> 960.
// (The gathers alone at 19 TB/s, what a loop of nothing else reaches: 571, 855 and 645 us.)
//
// Tried and slower at these shapes: one launch that walks all chunks (the warps drift apart: +0 to 50 %); no chunks, all warps in a
// moving window (965, 2,077 and 1,239 us); rows asked for two steps ahead in a ring of registers instead of two at a time (1,003,
// 1,554, 1,133); outputs and weights of both steps read before the gathers (858, 1,553, 1,127); bulk copies of the rows to shared
// memory (3 to 6 TB/s).
#include <algorithm>
#include <climits>
#include <type_traits>

#include "ffi_common.cuh"
#include "packed.cuh"

namespace ffi {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
// A chunk's rows of gT, of the tile's columns, take at most kChunkBytes (whole steps, us, with 32, 40, 48, 56, 64 MB at the three shapes
// above: 1,476, 1,455, 1,456, 1,513, 1,589; 2,061, 1,953, 1,946, 1,971, 2,043; 1,425, 1,421, 1,404, 1,438, 1,447), and together with the
// chunk's W, positions and grad_W, which pass through L2 besides, at most kChunkAll: with 64 columns and fewer those are the larger
// part (without that limit, with 112 MB, with 88 MB: B=64, N=78,400, L=558,266, K=48 bf16 1,831, 1,521, 1,453; B=32, N=30,000, L=600,000,
// K=32 fp32 848, 772, 770; B=20, N=20,000, L=700,000, K=72 fp32 1,915, 1,847, 1,852).
constexpr long long kChunkBytes = 48ll << 20, kChunkAll = 96ll << 20;
constexpr int kRow = 36;  // floats per buffered step: 32 partial dots + padding (16-byte rows, conflict-free both ways)

struct BwdWideParams {
    const void* W;
    const float* gT;  // [L][ldg], this launch's batch tile
    const void* xT;   // [N][ldx], element type of W, this launch's batch tile
    float* gx;        // [N][ldgx], likewise
    const int* rowptr;
    const int* perm;
    const int* starts;  // [N] first entry of each input that the chunks before have not walked
    int* cursor;        // [N] the same after this chunk, or nullptr (more batch tiles to come)
    float* gW;
    float* gbias;  // or nullptr
    long long ldg, ldx, ldgx;
    long long o0, o1;  // outputs of this chunk
    int endPos;        // o1 * K
    unsigned ldgBytes;
    int B, N, K;      // B: columns from this tile on
    bool xVec, gxVec; // rows of x / grad_x are aligned and hold the whole tile
    bool addW, addX;  // a batch tile / a chunk after the first
};

// The 8 batch columns one lane of a group holds, as pairs: 4q..4q+3 of each half of the tile (HALF columns apart).
template <int HALF>
struct Cols8 {
    u64 v[4];
    __device__ __forceinline__ void zero() { v[0] = v[1] = v[2] = v[3] = 0ull; }
    // at: this lane's first column
    __device__ __forceinline__ void gather(const unsigned char* at) {
        const ulonglong2 a = __ldg(reinterpret_cast<const ulonglong2*>(at));
        const ulonglong2 b = __ldg(reinterpret_cast<const ulonglong2*>(at + 4 * HALF));
        v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
    }
    __device__ __forceinline__ void load_shared(const float* at) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(at), b = *reinterpret_cast<const ulonglong2*>(at + HALF);
        v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
    }
    __device__ __forceinline__ void load_shared(const __nv_bfloat16* at) {
        const uint2 a = *reinterpret_cast<const uint2*>(at), b = *reinterpret_cast<const uint2*>(at + HALF);
        v[0] = pack2(bf16_lo(a.x), bf16_hi(a.x)), v[1] = pack2(bf16_lo(a.y), bf16_hi(a.y));
        v[2] = pack2(bf16_lo(b.x), bf16_hi(b.x)), v[3] = pack2(bf16_lo(b.y), bf16_hi(b.y));
    }
    // element by element; `left` columns exist from `at` on
    template <typename T>
    __device__ __forceinline__ void load_ragged(const T* at, int left) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int col = (j >> 1) * HALF + (j & 1) * 2;
            v[j] = pack2(col < left ? widen(at[col]) : 0.f, col + 1 < left ? widen(at[col + 1]) : 0.f);
        }
    }
    __device__ __forceinline__ void axpy(float w, const Cols8& g) {
        const u64 ww = pack2(w, w);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = fma2(ww, g.v[j], v[j]);
    }
    __device__ __forceinline__ float dot(const Cols8& g) const {
        float lo, hi;
        unpack2(fma2(g.v[3], v[3], fma2(g.v[2], v[2], fma2(g.v[1], v[1], mul2(g.v[0], v[0])))), lo, hi);
        return lo + hi;
    }
};

// A weight, past L1: a line of L1 for each of these small scattered reads would push out gathered rows on their way.
__device__ __forceinline__ float load_weight(const float* at) { return __ldcg(at); }
__device__ __forceinline__ float load_weight(const __nv_bfloat16* at) {
    return bf16_lo(__ldcg(reinterpret_cast<const unsigned short*>(at)));
}

// Shared memory of a warp.  What a warp knows about the batches ahead lives here and arrives by asynchronous copies: the gathers
// need the registers (a spilled value costs a round trip to L2, because the gathered rows push it out of L1) and L1 (of which this
// takes its part: rows in flight occupy it).
template <int BT>
struct WarpScratch {
    float x[BT];            // x of the next run's input, in its storage type
    float dots[16 * kRow];  // the lanes' partial dots of up to 16 steps
    uint2 ent[32];          // (output, weight) of this batch's entries
    int pos[3][32];         // positions of this batch, the next and the one after
    int next[4];            // (2 used) the bounds of the run after the newest batch's
};

template <int GROUPS, typename TX>
__global__ void __launch_bounds__(kThreads, 4) ffi_bwd_wide_kernel(const __grid_constant__ BwdWideParams p) {
    constexpr int LG = 32 / GROUPS, BT = 8 * LG, HALF = BT / 2;
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int FE = GROUPS == 1 ? 16 : 32;  // entries whose partial dots are added up together
    constexpr int LPE = 32 / FE;               // by as many lanes each
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, grp = lane / LG, q = lane % LG;
    WarpScratch<BT>& ws = reinterpret_cast<WarpScratch<BT>*>(smem_raw)[threadIdx.x >> 5];
    const int stride = gridDim.x * kWarps;
    // neighbouring inputs go to different CTAs, so that all SMs hold the same number of inputs to within one
    int i0 = blockIdx.x + gridDim.x * (threadIdx.x >> 5);

    // The launch after this one may start its CTAs while this one's last warps finish: grad_bias needs nothing of the chunks
    // before, and reading the chunk's rows for it brings them into L2.  This comes before the wait, so gT has to be complete when the
    // first launch of the sequence starts: that one is a plain launch (launch_wide), which starts after all that precedes it.
    chain_release();
    if (p.gbias) {  // four rows at a time
        for (long long o = p.o0 + i0; o < p.o1; o += 4ll * stride) {
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
            for (int b = 4 * lane; b < p.ldg; b += 128)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (o + j * stride < p.o1) {
                        const float4 v = __ldg(reinterpret_cast<const float4*>(p.gT + (o + j * stride) * p.ldg + b));
                        sum[j] += (v.x + v.y) + (v.z + v.w);
                    }
#pragma unroll
            for (int off = 16; off >= 1; off /= 2)
#pragma unroll
                for (int j = 0; j < 4; ++j) sum[j] += __shfl_xor_sync(kAll, sum[j], off);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (lane == 0 && o + j * stride < p.o1) p.gbias[o + j * stride] = sum[j];
        }
    }
    chain_wait();
    if (i0 >= p.N) return;

    // A batch is up to 32 entries of one run.  While one is worked on, the weights of the next and the positions of the one
    // after that are on their way, and so are the bounds of the run after those.
    auto fetch_bounds = [&](int i) {
        if (lane < 2) {
            if (i < p.N) __pipeline_memcpy_async(&ws.next[lane], lane == 0 ? p.starts + i : p.rowptr + i + 1, 4);
            else ws.next[lane] = 0;
        }
    };
    auto fetch_pos = [&](int slot, int e, int t) {
        if (e + lane < t) __pipeline_memcpy_async(&ws.pos[slot][lane], p.perm + e + lane, 4);
        else ws.pos[slot][lane] = INT_MAX;
    };
    auto fetch_weight = [&](int pos) -> float { return pos < p.endPos ? load_weight(static_cast<const TX*>(p.W) + pos) : 0.f; };
    // x of a run's input: copied to shared memory a batch ahead where its rows are aligned
    auto fetch_x = [&](int i) {
        if (p.xVec && i < p.N) {
            const unsigned char* src = reinterpret_cast<const unsigned char*>(static_cast<const TX*>(p.xT) + static_cast<size_t>(i) * p.ldx);
            constexpr int kBytes = BT * sizeof(TX);
#pragma unroll
            for (int o = 0; o < kBytes; o += 512)
                if (o + 512 <= kBytes || o + lane * 16 < kBytes)
                    __pipeline_memcpy_async(reinterpret_cast<unsigned char*>(ws.x) + o + lane * 16, src + o + lane * 16, 16);
        }
    };
    auto arrived = [&]() {
        __pipeline_commit();
        __pipeline_wait_prior(0);
        __syncwarp();
    };
    Cols8<HALF> acc, x;
    auto begin_run = [&](int i) {
        acc.zero();
        if (p.xVec) x.load_shared(reinterpret_cast<const TX*>(ws.x) + 4 * q);
        else x.load_ragged(static_cast<const TX*>(p.xT) + static_cast<size_t>(i) * p.ldx + 4 * q, p.B - 4 * q);
    };
    int e1 = p.starts[i0], t1 = p.rowptr[i0 + 1];  // first entry of the newest batch, its run's end
    // from the newest batch, of input i and cnt entries, to the one after it
    auto advance = [&](int i, int cnt) {
        if (cnt < 32) {
            if (p.cursor && lane == 0 && i < p.N) p.cursor[i] = e1 + cnt;
            e1 = ws.next[0], t1 = ws.next[1];
            __syncwarp();
            fetch_bounds(i + 2 * stride);
        } else {
            e1 += 32;
        }
    };
    fetch_pos(0, e1, t1);
    fetch_bounds(i0 + stride);
    fetch_x(i0);
    arrived();
    const int first_pos = ws.pos[0][lane];
    int cnt0 = __popc(__ballot_sync(kAll, first_pos < p.endPos));  // entries of this batch (positions ascend along a run)
    float w0 = fetch_weight(first_pos);
    advance(i0, cnt0);
    fetch_pos(1, e1, t1);
    begin_run(i0);
    __syncwarp();
    if (cnt0 < 32) fetch_x(i0 + stride);
    int slot = 0;  // of this batch's positions
    while (true) {
        arrived();
        int cnt1;  // entries of the next batch
        {
            ws.ent[lane] = make_uint2(static_cast<unsigned>(ws.pos[slot][lane]) / static_cast<unsigned>(p.K), __float_as_uint(w0));
            const int slot1 = slot == 2 ? 0 : slot + 1;
            const int pos1 = ws.pos[slot1][lane];
            cnt1 = __popc(__ballot_sync(kAll, pos1 < p.endPos));
            w0 = fetch_weight(pos1);
            advance(cnt0 < 32 ? i0 + stride : i0, cnt1);
            fetch_pos(slot1 == 2 ? 0 : slot1 + 1, e1, t1);
            __syncwarp();
        }
        const unsigned char* gLane = reinterpret_cast<const unsigned char*>(p.gT + 4 * q);
#pragma unroll 1
        for (int h = 0; h < cnt0; h += FE) {
            const int n = FE == 32 ? cnt0 : min(FE, cnt0 - h);
            const uint2* en = ws.ent + h + grp;
            float* d = ws.dots + lane;
            int u = 0;
            // two steps' rows in flight: 32 warps per SM with 2 KB each keep the fabric busy, more per warp gains nothing
#pragma unroll 1
            for (; u + 2 * GROUPS <= n; u += 2 * GROUPS) {
                Cols8<HALF> v0, v1;
                v0.gather(gLane + static_cast<unsigned long long>(en[u].x) * p.ldgBytes);
                v1.gather(gLane + static_cast<unsigned long long>(en[u + GROUPS].x) * p.ldgBytes);
                acc.axpy(__uint_as_float(en[u].y), v0);
                d[(u / GROUPS) * kRow] = x.dot(v0);
                acc.axpy(__uint_as_float(en[u + GROUPS].y), v1);
                d[(u / GROUPS + 1) * kRow] = x.dot(v1);
            }
            for (; u < n; u += GROUPS) {  // the last steps have entries for the first n - u groups only
                Cols8<HALF> v;
                float w = 0.f;
                v.zero();
                if (u + grp < n) {
                    const uint2 e = en[u];
                    w = __uint_as_float(e.y);
                    v.gather(gLane + static_cast<unsigned long long>(e.x) * p.ldgBytes);
                }
                acc.axpy(w, v);
                d[(u / GROUPS) * kRow] = x.dot(v);
            }
            __syncwarp();
            // lane LPE * e adds the partial dots of entry h + e (with its neighbour's help where LPE = 2), in a fixed order
            const int el = lane / LPE;
            const float4* row = reinterpret_cast<const float4*>(ws.dots + (el / GROUPS) * kRow + (el % GROUPS) * LG + (lane % LPE) * (LG / LPE));
            float s[LG / LPE / 4];
#pragma unroll
            for (int k = 0; k < LG / LPE / 4; ++k) s[k] = (row[k].x + row[k].y) + (row[k].z + row[k].w);
#pragma unroll
            for (int k = LG / LPE / 8; k >= 1; k /= 2)
#pragma unroll
                for (int j = 0; j < k; ++j) s[j] += s[j + k];
            if (LPE == 2) s[0] += __shfl_xor_sync(kAll, s[0], 1);
            if (lane % LPE == 0 && el < n) {
                float* dst = p.gW + ws.pos[slot][h + el];
                // (a batch tile after the first adds to what the one before stored, once per element: a reduction in L2 that nobody waits
                // for; loading the old value took 158 to 187 % of the time at B=300, N=3,000 ... 4,000)
                if (p.addW) atomicAdd(dst, s[0]);
                else *dst = s[0];
            }
            __syncwarp();
        }
        if (cnt0 < 32) {
            // This chunk's part of grad_x joins what the chunks before left, by reductions in L2 that nobody waits for: a row is
            // only ever added to by one warp per launch.
            float out[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) unpack2(acc.v[j], out[2 * j], out[2 * j + 1]);
#pragma unroll
            for (int j = 0; j < 8; ++j)
#pragma unroll
                for (int off = 16; off >= LG; off /= 2) out[j] += __shfl_xor_sync(kAll, out[j], off);
            if (grp == 0) {
                float* dst = p.gx + static_cast<size_t>(i0) * p.ldgx + 4 * q;
#pragma unroll
                for (int j = 0; j < 8; j += 4) {
                    float* at = dst + (j / 4) * HALF;
                    if (p.gxVec) {
                        if (p.addX)
                            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(at), "f"(out[j]), "f"(out[j + 1]),
                                         "f"(out[j + 2]), "f"(out[j + 3])
                                         : "memory");
                        else
                            *reinterpret_cast<float4*>(at) = make_float4(out[j], out[j + 1], out[j + 2], out[j + 3]);
                    } else {
#pragma unroll
                        for (int m = 0; m < 4; ++m)
                            if ((j / 4) * HALF + m < p.B - 4 * q) {
                                if (p.addX) atomicAdd(at + m, out[j + m]);
                                else at[m] = out[j + m];
                            }
                    }
                }
            }
            i0 += stride;
            if (i0 >= p.N) break;
            begin_run(i0);
        }
        __syncwarp();
        if (cnt1 < 32) fetch_x(i0 + stride);  // the next batch is its run's last
        cnt0 = cnt1;
        slot = slot == 2 ? 0 : slot + 1;
    }
    __pipeline_wait_prior(0);
}

template <int GROUPS, typename TX>
int launch_wide(BwdWideParams p, long long L, const DeviceInfo& dev, cudaStream_t stream) {
    auto kern = ffi_bwd_wide_kernel<GROUPS, TX>;
    constexpr int BT = 256 / GROUPS;
    constexpr size_t smem = kWarps * sizeof(WarpScratch<BT>);
    int occ = 0;
    FFI_CUDA_CHECK(prepare_kernel(reinterpret_cast<const void*>(kern), kThreads, smem, &occ));
    if (occ < 1) return fail(FFI_ERR_CUDA, "one-pass backward for wide inputs does not fit on an SM");
    const int B = p.B, tiles = static_cast<int>(ceil_div(B, BT));
    const long long perRow = BT * 4 + static_cast<long long>(p.K) * (4 + 4 + sizeof(TX));
    long long rows = std::min(kChunkBytes / (BT * 4), kChunkAll / perRow);
    if (rows < 1) rows = 1;
    const long long nChunks = ceil_div(L, rows), T = ceil_div(L, nChunks);
    // as many warps as give each the same number of inputs, and as many CTAs on every SM: with 257 CTAs for 2,049 inputs some SMs had
    // two and others one (B=300, L=200,000, K=32 1,334 -> 987 us; N=5,000 1,224 -> 1,007; from 16,384 inputs on no difference)
    const long long cap = static_cast<long long>(dev.sm_count) * occ * kWarps;
    const long long ctas = round_up(ceil_div(ceil_div(p.N, ceil_div(p.N, cap)), kWarps), dev.sm_count);
    int* cursor = p.cursor;
    const float* gT = p.gT;
    const TX* xT = static_cast<const TX*>(p.xT);
    float *gx = p.gx, *gbias = p.gbias;
    for (long long o0 = 0; o0 < L; o0 += T) {
        p.o0 = o0, p.o1 = L < o0 + T ? L : o0 + T;
        p.endPos = static_cast<int>(p.o1 * p.K);
        p.starts = o0 == 0 ? p.rowptr : cursor;
        p.addX = o0 > 0;
        for (int t = 0; t < tiles; ++t) {
            p.gT = gT + t * BT, p.xT = xT + t * BT, p.gx = gx + t * BT, p.B = B - t * BT;
            p.xVec = p.ldx % 8 == 0 && p.ldx >= static_cast<long long>(tiles) * BT && reinterpret_cast<uintptr_t>(xT) % 16 == 0;
            p.gxVec = p.ldgx % 4 == 0 && p.B >= BT && reinterpret_cast<uintptr_t>(gx) % 16 == 0;
            p.addW = t > 0;
            p.cursor = t + 1 == tiles && p.o1 < L ? cursor : nullptr;
            p.gbias = t == 0 ? gbias : nullptr;
            if (o0 > 0 || t > 0) FFI_CUDA_CHECK(launch_chained(kern, dim3(static_cast<unsigned>(ctas)), dim3(kThreads), smem, stream, p));
            else kern<<<static_cast<unsigned>(ctas), kThreads, smem, stream>>>(p);  // not chained: the kernel reads gT and writes grad_bias before it waits
        }
    }
    FFI_LAUNCH_CHECK("ffi_bwd_wide_kernel");
    return FFI_OK;
}

}  // namespace

// Plans without chunked lists (wide inputs).  Against a kernel each for grad_x and grad_W, at K=16 ... 64, L=20,000 and 200,000, by
// number of inputs: 2,049 1.1 (B=390 bf16, two tiles of which the second is half empty) to 3.8 times as fast (B=20), 5,000 1.1 to
// 2.4, 12,000 1.35 to 2.6, 65,536 1.2 to 2.1.
bool backward_wide_applicable(const ffi_plan* plan) { return plan && !plan->has_chunks && plan->N > 2048; }

namespace {
// Columns of the batch tiles.
int tile_columns(int64_t ldg) { return ldg % 256 == 0 ? 256 : ldg % 128 == 0 ? 128 : ldg % 64 == 0 ? 64 : 32; }
}  // namespace

// An input belongs to one warp, here and in the kernel for grad_x alone, so an input with very many entries holds up everything else.
// Here the batch tiles come one after another, in kChain us an entry and tile; there all tiles are walked at once, in about 0.2 us an
// entry (0.13 to 0.28).  So several tiles pay for what the hottest input has beyond the others as long as that stays below what one
// gather less gains, 0.1 (bf16) or 0.2 (fp32) us for a million entries and columns, and 10 us for a kernel less.  Measured, both kernels against one, us, for the inputs drawn
// by Zipf's law of the exponents 0, 0.2, 0.3, 0.4, 0.6: B=512, N=16,384, L=50,000, K=32 bf16 334, 369, 520, 886, 2,732 against 254, 374,
// 588, 1,043, 4,003 (line at 0.3), fp32 425, 469, 620, 1,001, 2,974 against 256, 371, 575, 1,016, 3,912 (line between 0.3 and 0.4);
// B=1,024, N=32,768, L=60,000, K=32 bf16 788, 816, 929, 1,276, 3,695 against 597, 705, 998, 1,753, 7,343 (line between 0.2 and 0.3);
// B=384 fp32 line between 0.4 and 0.5.  One tile pays always: B=256, N=65,536, L=200,000 bf16 681, 784, 1,057, 1,874, 8,353 against 520,
// 575, 737, 1,168, 4,963.
bool backward_wide_pays(const ffi_plan* plan, int64_t B, int64_t ldg, bool bf16) {
    const int columns = tile_columns(ldg);
    const double kChain = columns == 256 ? 0.14 : columns == 128 ? 0.077 : columns == 64 ? 0.054 : 0.035;
    const double more = ceil_div(B, columns) * kChain - 0.2;
    const double entries = static_cast<double>(plan->L) * plan->K, beyond = plan->longest_input - 2.0 * entries / plan->N;
    return more <= 0.0 || beyond * more <= (bf16 ? 1e-7 : 2e-7) * entries * B + 10.0;
}

// grad_x as [N][B] (always), grad_W and, when gbias != nullptr, grad_bias, from gT; xT is x as [N][ldx]; cursor: N ints.
int launch_backward_wide(const GradXArgs& a, const void* xT, int64_t ldx, float* gxT, float* gW, float* gbias, int* cursor,
                         cudaStream_t stream) {
    DeviceInfo dev;
    const int rc = get_device_info(&dev);
    if (rc != FFI_OK) return rc;
    BwdWideParams p{};
    p.W = a.W, p.gT = a.gT, p.xT = xT, p.gx = gxT, p.gW = gW, p.gbias = gbias;
    p.rowptr = a.plan->rowptr, p.perm = a.plan->perm, p.cursor = cursor;
    p.ldg = a.ldg, p.ldx = ldx, p.ldgx = a.B, p.ldgBytes = static_cast<unsigned>(a.ldg * 4);
    p.B = a.B, p.N = a.N, p.K = a.K;
    auto typed = [&](auto tx) -> int {
        using TX = decltype(tx);
        switch (tile_columns(a.ldg)) {
            case 256: return launch_wide<1, TX>(p, a.L, dev, stream);
            case 128: return launch_wide<2, TX>(p, a.L, dev, stream);
            case 64: return launch_wide<4, TX>(p, a.L, dev, stream);
            default: return launch_wide<8, TX>(p, a.L, dev, stream);
        }
    };
    return a.w_bf16 ? typed(__nv_bfloat16{}) : typed(float{});
}

}  // namespace ffi
