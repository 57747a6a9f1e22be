// Forward of the fixed-fan-in sparse layer for bf16 storage on the tensor cores, narrow inputs (N <= 768):
//   y[b,o] = bias[o] + sum_i Wd[o,i] * x[i,b],   Wd = the rows of W scattered into zeros.
// Replaces the reference's forward_ob_scalar_tp (tfsparse/cc/kernels/forward.cu.h:231-264) for the configurations that keep
// x and W in bf16.
//
// Why densify: the gather kernels move one operand per multiplication through shared memory (2.7 GFMA x 2 bytes at the
// headline shape, 0.28 ms), while a row of 32 entries among 768 inputs costs the tensor core 24 times the multiplications
// at 60 times the rate.  The products of bf16 values are exact in fp32 and the accumulator is fp32, so nothing is lost
// against the gather; zeros add nothing to finite inputs.  An infinite or NaN x[i,b] would turn them into NaN in every row,
// so the tensor core is given +-1 in its place, and the rows that read input i get w * x[i,b] added in fp32 (the sum then
// holds +-|w| and the infinity or NaN itself: what a plain sum over the row's entries holds).
//
// Dataflow (one persistent CTA per SM and batch tile of 128):
//   * the batch tile of x is the A operand and stays in tensor memory, lane = sample, 32-bit column = two inputs
//     (N / 2 <= 384 columns); D is [128 samples][64 outputs] fp32, two buffers of 64 columns;
//   * B is a tile of 64 rows of Wd, [64][N] bf16 in shared memory (128-byte swizzled panels of 64 inputs), two buffers.  It
//     is never cleared as a whole: a warp owns eight rows (four with K > 32), remembers where it wrote and puts zeros back there,
//     so a row of K entries costs 2K two-byte stores instead of a row of N;
//   * entries of a row with the same input cannot share a cell (their sum is no bf16): one of them is written, the others
//     go to a list per 16 rows that is added to the results with fp32 FMAs, x read back from tensor memory; what does not fit
//     the list waits for another round of the same tile that accumulates.  Tables without repeated inputs never do either;
//   * the warps specialise: 8 build tiles, one issues the N / 16 MMAs of a tile (M = 128, N = 64, K = 16), 16 turn D into y
//     or the loss gradient (16 and 8 with K > 32: building, two entries a lane, is the longest stage there); mbarriers hand the
//     buffers on, so the three stages of consecutive tiles overlap.  (With all warps building and emitting in turn, one CTA
//     barrier per tile, the stages' latencies added up: 214 us for y, 310 with the BCE epilogue.)
// What bounds it, by the share of the time that a stage does not wait for another (N = 768, distinct inputs / with replacement): at
// K = 32 the thread that issues the MMAs 0.88 / 0.86 (the tensor core's part is active for 0.46 / 0.42; tiles of 64 rows are
// what fits beside x), the building warps 0.84 / 0.95, the emitting ones 0.43 / 0.56; at K = 64 the thread 0.90 / 0.59, building
// 0.82 / 0.68, emitting 0.59 / 0.97 (about 80 clocks per repeated input: its sum is read, added to and written in shared memory).
// Measured at B = 128, L = 670,091, tables of distinct inputs / drawn with replacement, against the gather kernel:
// N = 768, K = 32: y 232/261 (379) us, loss gradient 245/288 (289) us; K = 64: 274/430 (594) and 294/493 (474) us;
// B = 256, N = 512, L = 65,536, K = 64: y 62/113 (113) us.  With the lists read by 16 warps from L2, one entry after the other, and
// 8 building warps: y 239/299 and 331/905, loss gradient 253/327 and 364/986, 71/220 us.
#include <type_traits>

#include "tcgen05.cuh"

namespace ffi {
namespace {

__device__ int g_dense_timeouts = 0;                // bounded waits of this kernel that gave up
__device__ long long g_dense_limit = 4000000000ll;  // clock64 ticks a wait may last (about two seconds)
constexpr long long kDrainLimit = 4000000000ll;     // ... and the last one, for MMAs that are under way, whatever that is set to

constexpr int kMmaWarp = 24;                  // the warps before it write results or build tiles, this one issues the MMAs
constexpr int kThreads = 32 * (kMmaWarp + 1);
constexpr int kMaxBuildWarps = 16;
constexpr int kRows = 64;                     // outputs per tile
constexpr int kMaxPanels = 12;                // 12 * 32 columns of x + 2 * 64 of D fill the tensor memory
constexpr unsigned kPanelBytes = kRows * 128;

struct DenseFwdParams {
    const __nv_bfloat16* xT;  // [N][ldx]
    long long ldx;
    const int* idx;
    const unsigned short* W;
    const float* bias;
    float* y;
    int B, N, L, K;
    int panels;  // ceil(N / 64)
    int cap;     // entries a building warp may add to a list of repeated inputs, a multiple of 4
    // loss epilogue (MODE 1), as in forward_stream.cu
    float* gT;
    long long ldg;
    float scale;
    double* loss_partials;
    int loss_kind;
};

// sigmoid-BCE for target 0 on 16 logits of one sample: gradients in place, the loss values' sum returned.  The formulas of
// loss_for_negative; the logarithms of 1 + exp(-|z|) <= 2 are taken once over their product.
__device__ __forceinline__ float bce_negative16(float (&z)[16]) {
    float sum = 0.f, prod = 1.f;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        float s, r;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(fabsf(z[j]) * -1.4426950408889634f));
        const float d = 1.f + s;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
        prod *= d;
        sum += fmaxf(z[j], 0.f);
        z[j] = z[j] >= 0.f ? r : s * r;
    }
    return sum + __logf(prod);
}

constexpr unsigned kBf16One = 0x3f80u;
__device__ __forceinline__ bool bf16_finite(unsigned low_half) { return (low_half & 0x7f80u) != 0x7f80u; }
__device__ __forceinline__ __nv_bfloat162 as_bf162(unsigned w) { return *reinterpret_cast<const __nv_bfloat162*>(&w); }
__device__ __forceinline__ unsigned as_word(__nv_bfloat162 v) { return *reinterpret_cast<const unsigned*>(&v); }

struct DenseBarriers {
    unsigned long long full[2];    // a tile is built (one arrival per building warp)
    unsigned long long done[2];    // its MMAs are done: the tile buffer is free
    unsigned long long ready[2];   // ... and no further round follows: D is complete
    unsigned long long dfree[2];   // D has been read (one arrival per emitting warp)
    unsigned long long idle;       // all MMAs of the CTA are done
    unsigned tmem;
    int more[2];                   // another round of this tile follows
    int listed[2][kMaxBuildWarps]; // entries each building warp has in the lists of repeated inputs
    int bad;                       // a wait gave up: everybody runs through without waiting, the results are void
    unsigned nonfinite[2 * kMaxPanels];  // inputs with a sample of this tile that is infinite or NaN
};
// Behind the barriers: the lists of repeated inputs, one per buffer and 16 rows.  An entry is laid out so that the emitting warps
// need few instructions for it: the weight in the half of a word that its input has in a column of x, and
// column << 23 | square_row(row of the 16).
constexpr size_t kListsAt = (sizeof(DenseBarriers) + 15) / 16 * 16;

// Offset of output j's row in an emitting warp's square of [16 outputs][32 samples], with the key of its samples' order
// (sample s stands at place s ^ 2j: conflict-free by rows and by columns).
__host__ __device__ constexpr unsigned square_row(unsigned j) { return j << 7 | j << 3; }

// z + x.lo * w.lo + x.hi * w.hi, exact products of bf16
__device__ __forceinline__ float fma_pair(unsigned x, unsigned w, float z) {
    unsigned short xl, xh, wl, wh;
    asm("mov.b32 {%0, %1}, %2;" : "=h"(xl), "=h"(xh) : "r"(x));
    asm("mov.b32 {%0, %1}, %2;" : "=h"(wl), "=h"(wh) : "r"(w));
    asm("fma.rn.f32.bf16 %0, %1, %2, %0;" : "+f"(z) : "h"(xl), "h"(wl));
    asm("fma.rn.f32.bf16 %0, %1, %2, %0;" : "+f"(z) : "h"(xh), "h"(wh));
    return z;
}

// z plus the products of row o with the infinite and NaN inputs of sample b.  Called by whole warps, where a tile has any.
__device__ __forceinline__ float add_nonfinite(const DenseFwdParams& p, const unsigned* flags, long long o, int b, float z) {
    const int lane = threadIdx.x & 31;
    for (int k0 = 0; k0 < p.K; k0 += 32) {
        const int k = k0 + lane;
        const unsigned i = k < p.K ? static_cast<unsigned>(__ldg(p.idx + o * p.K + k)) : 0xffffffffu;
        const unsigned w = k < p.K ? static_cast<unsigned>(__ldg(p.W + o * p.K + k)) << 16 : 0u;
        unsigned todo = __ballot_sync(0xffffffffu, i < static_cast<unsigned>(p.N) && (flags[i >> 5] >> (i & 31) & 1u));
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1;
            const unsigned ib = __shfl_sync(0xffffffffu, i, src);
            const float wb = __uint_as_float(__shfl_sync(0xffffffffu, w, src));
            const float x = b < p.B ? widen(p.xT[static_cast<size_t>(ib) * p.ldx + b]) : 0.f;
            if (!isfinite(x)) z = fmaf(wb, x, z);
        }
    }
    return z;
}

// MODE 0 writes y, 1 the loss gradient.  KG: entries of a row per lane (K <= 32 * KG).  EMIT: warps that write results (8 or 16).
template <int MODE, int KG, int EMIT>
__global__ void __launch_bounds__(kThreads, 1) ffi_fwd_dense_kernel(DenseFwdParams p) {
    chain_wait();
    constexpr int kEmitWarps = EMIT, kBuildWarps = kMmaWarp - EMIT;
    constexpr int kWarpRows = kRows / kBuildWarps;  // rows of a tile that a building warp has
    constexpr int kListWarps = 16 / kWarpRows;      // building warps that share a list
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b0 = blockIdx.y * 128;
    const int K = p.K, L = p.L;
    const unsigned tileBytes = p.panels * kPanelBytes;
    unsigned char* squares = smem + 2 * tileBytes;  // one of 2 KB per emitting warp
    DenseBarriers* bars = reinterpret_cast<DenseBarriers*>(smem + 2 * tileBytes + kEmitWarps * 2048);
    uint2* lists = reinterpret_cast<uint2*>(reinterpret_cast<unsigned char*>(bars) + kListsAt);
    volatile int* bad = &bars->bad;

    if (warp == kMmaWarp) tc::alloc(&bars->tmem);
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            tc::bar_init(bars->full + i, kBuildWarps);
            tc::bar_init(bars->done + i, 1);
            tc::bar_init(bars->ready + i, 1);
            tc::bar_init(bars->dfree + i, kEmitWarps);
        }
        tc::bar_init(&bars->idle, 1);
        *bad = 0;
    }
    // After a wait that gave up the lists are read before or while they are written: what stands there is always a list.
    for (int e = tid; e < 2 * kBuildWarps * p.cap; e += kThreads) lists[e] = make_uint2(0u, 0u);
    if (tid < 2 * kMaxBuildWarps) (&bars->listed[0][0])[tid] = 0;
    if (tid < 2) bars->more[tid] = 0;
    if (tid < 2 * kMaxPanels) bars->nonfinite[tid] = 0;
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const unsigned tmem = bars->tmem;
    const unsigned tmem_d = tmem + p.panels * (tc::kPanelK / 2);
    const unsigned lane_base = static_cast<unsigned>((warp & 3) * 32) << 16;

    // ---- x into tensor memory, through the (still unused) tile buffers: rows of 128 samples, then lane = sample ----------
    {
        unsigned short* xs = reinterpret_cast<unsigned short*>(smem);
        const int rows = p.panels * tc::kPanelK;
        const bool vec = p.ldx % 8 == 0 && b0 + 128 <= p.B && reinterpret_cast<uintptr_t>(p.xT) % 16 == 0;
        const unsigned short* xg = reinterpret_cast<const unsigned short*>(p.xT) + b0;
        if (vec) {
            for (int e = tid; e < rows * 16; e += kThreads) {
                const int i = e >> 4, v = e & 15;
                if (i < p.N) __pipeline_memcpy_async(xs + i * 128 + 8 * v, xg + static_cast<size_t>(i) * p.ldx + 8 * v, 16);
                else *reinterpret_cast<uint4*>(xs + i * 128 + 8 * v) = make_uint4(0u, 0u, 0u, 0u);
            }
            __pipeline_commit();
            __pipeline_wait_prior(0);
        } else {
#pragma unroll 8
            for (int e = tid; e < rows * 128; e += kThreads) {
                const int i = e >> 7, b = e & 127;
                xs[e] = i < p.N && b0 + b < p.B ? __ldg(xg + static_cast<size_t>(i) * p.ldx + b) : static_cast<unsigned short>(0);
            }
        }
        __syncthreads();
        if (warp < kMmaWarp) {
            const unsigned short* xl = xs + (warp & 3) * 32 + lane;
            for (int c = (warp >> 2) * 8; c < rows / 2; c += 8 * (kMmaWarp / 4)) {
                unsigned r[8];
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    r[j] = xl[(2 * (c + j)) * 128] | (static_cast<unsigned>(xl[(2 * (c + j) + 1) * 128]) << 16);
                // zero times an infinity or a NaN is NaN: one sum tells whether any of the sixteen values is not finite
                __nv_bfloat162 zeros = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
                for (int j = 0; j < 8; ++j) zeros = __hfma2(as_bf162(r[j]), __floats2bfloat162_rn(0.f, 0.f), zeros);
                if ((as_word(zeros) & 0x7fff7fffu) != 0) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const bool lo = !bf16_finite(r[j]), hi = !bf16_finite(r[j] >> 16);
                        const int i = 2 * (c + j);
                        if (lo | hi) atomicOr(bars->nonfinite + (i >> 5), (static_cast<unsigned>(lo) | static_cast<unsigned>(hi) << 1) << (i & 31));
                        if (lo) r[j] = (r[j] & 0xffff8000u) | kBf16One;
                        if (hi) r[j] = (r[j] & 0x8000ffffu) | kBf16One << 16;
                    }
                }
                tc::store8(tmem + lane_base + c, r);
            }
            tc::wait_store();
        }
        __syncthreads();
        for (unsigned e = tid; e < tileBytes / 8; e += kThreads) reinterpret_cast<uint4*>(smem)[e] = make_uint4(0u, 0u, 0u, 0u);
        tc::fence_smem();
        tc::fence_before_sync();
        __syncthreads();
    }

    const int tiles = (L + kRows - 1) / kRows;
    const long long limit = g_dense_limit;
    auto await = [&](unsigned long long* bar, unsigned parity) {
        if (!*bad && !tc::bar_wait(bar, parity, limit)) {
            atomicAdd(&g_dense_timeouts, 1);
            *bad = 1;
        }
        __syncwarp();  // a lane may have given up by itself
    };
    float loss_local = 0.f;

    if (warp == kMmaWarp) {
        // ---- the MMAs ----------------------------------------------------------------------------------------------------
        unsigned full_ph[2] = {0u, 0u};
        int it = 0;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++it) {
            const int buf = it & 1;
            for (bool first = true;; first = false) {
                await(bars->full + buf, full_ph[buf]);
                full_ph[buf] ^= 1u;
                if (first && it >= 2) await(bars->dfree + buf, ((it >> 1) - 1) & 1);
                const bool more = __shfl_sync(0xffffffffu, *static_cast<volatile int*>(&bars->more[buf]) != 0 && !*bad, 0);
                if (lane == 0) {
                    tc::fence_after_sync();
                    // (a descriptor from scratch for each MMA took this thread 113 clocks a step)
                    const unsigned long long b = tc::panel_desc(tc::smem_addr(smem) + buf * tileBytes);
                    const unsigned d = tmem_d + buf * kRows;
                    for (int panel = 0; panel < p.panels; ++panel)
#pragma unroll
                        for (int m = 0; m < 4; ++m)
                            tc::mma(d, tmem + panel * 32 + m * 8, tc::desc_at(b, panel * kPanelBytes + m * 32), tc::instr_desc(kRows),
                                    !first || panel + m > 0);
                    tc::commit(bars->done + buf);
                    if (!more) tc::commit(bars->ready + buf);
                }
                __syncwarp();
                if (!more) break;
            }
        }
        // the CTA's memory is given back only after the last MMAs have read it, also when some wait has given up
        if (lane == 0) tc::commit(&bars->idle);
        __syncwarp();
        if (!tc::bar_wait(&bars->idle, 0, kDrainLimit)) atomicAdd(&g_dense_timeouts, 1);
    } else if (warp >= kEmitWarps) {
        // ---- tiles of Wd -------------------------------------------------------------------------------------------------
        const int bw = warp - kEmitWarps;
        int ir[kWarpRows][KG];
        unsigned short wr[kWarpRows][KG];
        // half the offset of the cells this lane has written in each buffer, two rows per word
        unsigned cells[2][kWarpRows / 2][KG];
        constexpr unsigned kNone = 0xffffu;
#pragma unroll
        for (int r = 0; r < kWarpRows / 2; ++r)
#pragma unroll
            for (int g = 0; g < KG; ++g) cells[0][r][g] = cells[1][r][g] = ~0u;
        auto fetch = [&](int t) {
#pragma unroll
            for (int r = 0; r < kWarpRows; ++r) {
                const long long o = static_cast<long long>(t) * kRows + bw * kWarpRows + r;
#pragma unroll
                for (int g = 0; g < KG; ++g) {
                    const int k = 32 * g + lane;
                    const bool in = o < L && k < K;
                    ir[r][g] = in ? __ldg(p.idx + o * K + k) : 0;
                    wr[r][g] = in ? __ldg(p.W + o * K + k) : static_cast<unsigned short>(0);
                }
            }
        };
        unsigned done_ph[2] = {0u, 0u};
        auto build = [&](auto bufc, int t, int use) {  // the use-th tile in buffer bufc
            constexpr int buf = decltype(bufc)::value;
            unsigned char* tile = smem + buf * tileBytes;
            auto at = [&](unsigned c) { return reinterpret_cast<volatile unsigned short*>(tile + 2u * c); };
            auto cell = [&](int r, int g) { return (cells[buf][r / 2][g] >> (16 * (r & 1))) & 0xffffu; };
            auto set_cell = [&](int r, int g, unsigned c) {
                cells[buf][r / 2][g] = (r & 1) ? ((cells[buf][r / 2][g] & 0xffffu) | (c << 16)) : ((cells[buf][r / 2][g] & 0xffff0000u) | c);
            };
            for (bool wait = use > 0, first = true;; wait = true, first = false) {
                if (wait) {  // the last MMAs on this buffer
                    await(bars->done + buf, done_ph[buf]);
                    done_ph[buf] ^= 1u;
                }
#pragma unroll
                for (int r = 0; r < kWarpRows; ++r)
#pragma unroll
                    for (int g = 0; g < KG; ++g)
                        if (cell(r, g) != kNone) *at(cell(r, g)) = 0;
                __syncwarp();
                // Every entry puts its number into its cell and reads it back: the one that finds it is the cell's.
                // (__match_any_sync per row took about 60 clocks of the SM each, 100 us at the headline shape.)
#pragma unroll
                for (int r = 0; r < kWarpRows; ++r)
#pragma unroll
                    for (int g = 0; g < KG; ++g) {
                        const unsigned i = static_cast<unsigned>(ir[r][g]);
                        const bool active = (wr[r][g] & 0x7fffu) != 0 && i < static_cast<unsigned>(p.N);
                        const unsigned c = ((i >> 6) * kPanelBytes + tc::panel_offset(bw * kWarpRows + r, i & 63u)) >> 1;
                        set_cell(r, g, active ? c : kNone);
                        if (active) *at(c) = static_cast<unsigned short>(32 * g + lane);
                    }
                __syncwarp();
                unsigned mine = 0, lost = 0;
#pragma unroll
                for (int r = 0; r < kWarpRows; ++r)
#pragma unroll
                    for (int g = 0; g < KG; ++g)
                        if (cell(r, g) != kNone) {
                            if (*at(cell(r, g)) == 32 * g + lane) mine |= 1u << (r * KG + g);
                            else lost |= 1u << (r * KG + g);
                        }
                __syncwarp();
#pragma unroll
                for (int r = 0; r < kWarpRows; ++r)
#pragma unroll
                    for (int g = 0; g < KG; ++g) {
                        if (mine >> (r * KG + g) & 1u) {
                            *at(cell(r, g)) = wr[r][g];
                            wr[r][g] = 0;
                        } else {
                            set_cell(r, g, kNone);
                        }
                    }
                // The entries that found another's number go to the list of their sixteen rows, in a fixed order: the warps that
                // share it tell each other their counts across the barrier.  What a warp has no room for waits for another
                // round, in which nothing is listed any more.
                unsigned who[kWarpRows * KG];
                int found = 0;
                bool left = lost != 0;
                if (first) {
                    if (use > 0) await(bars->dfree + buf, (use - 1) & 1);  // the lists of this buffer's tile before have been read
                    if (__any_sync(0xffffffffu, lost != 0)) {
#pragma unroll
                        for (int j = 0; j < kWarpRows * KG; ++j) {
                            who[j] = __ballot_sync(0xffffffffu, lost >> j & 1u);
                            found += __popc(who[j]);
                        }
                        left = lost != 0 && found > p.cap;
                    }
                    if (lane == 0) bars->listed[buf][bw] = min(found, p.cap);
                }
                tc::fence_smem();
                unsigned again;
                asm volatile(
                    "{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\n"
                    "barrier.cta.red.or.pred q, 1, %2, p;\nselp.u32 %0, 1, 0, q;\n}"
                    : "=r"(again)
                    : "r"(static_cast<unsigned>(left && !*bad)), "n"(32 * kBuildWarps)
                    : "memory");
                if (first) {
                    const int part = bw % kListWarps;
                    int at = 0, total = 0;
#pragma unroll
                    for (int w = 0; w < kListWarps; ++w) {
                        const int n = *static_cast<volatile int*>(&bars->listed[buf][bw - part + w]);
                        if (w < part) at += n;
                        total += n;
                    }
                    uint2* list = lists + (buf * kBuildWarps + bw - part) * p.cap;
                    if (found > 0) {
                        int before = 0;
#pragma unroll
                        for (int j = 0; j < kWarpRows * KG; ++j) {
                            const int slot = before + __popc(who[j] & ((1u << lane) - 1u));
                            before += __popc(who[j]);
                            if ((lost >> j & 1u) && slot < p.cap) {
                                const unsigned i = static_cast<unsigned>(ir[j / KG][j % KG]), w = wr[j / KG][j % KG];
                                list[at + slot] = make_uint2(i & 1u ? w << 16 : w, (i >> 1) << 23 | square_row(part * kWarpRows + j / KG));
                                wr[j / KG][j % KG] = 0;
                            }
                        }
                    }
                    // a step of the emitting warps takes four entries
                    if (part == kListWarps - 1 && lane < (-total & 3)) list[total + lane] = make_uint2(0u, 0u);
                    __syncwarp();
                }
                if (lane == 0) {
                    if (bw == 0) *static_cast<volatile int*>(&bars->more[buf]) = static_cast<int>(again);
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_addr(bars->full + buf)) : "memory");
                }
                if (!again) break;  // one answer for the building warps, which meet at the barrier above
            }
            const int next = t + static_cast<int>(gridDim.x);
            if (next < tiles) fetch(next);
        };
        int t = blockIdx.x;
        fetch(t);
        for (int it = 0; t < tiles; ++it) {
            build(std::integral_constant<int, 0>{}, t, it);
            t += gridDim.x;
            if (t >= tiles) break;
            build(std::integral_constant<int, 1>{}, t, it);
            t += gridDim.x;
        }
    } else {
        // ---- results -----------------------------------------------------------------------------------------------------
        const int q = warp & 3, col = lane & 15;  // this warp's samples are 32 q ...; its outputs the 64 / EMIT groups of 16 below
        const int b = b0 + q * 32 + lane;
        unsigned char* sq = squares + warp * 2048;
        auto sq_at = [&](int j, int sample) -> float& { return *reinterpret_cast<float*>(sq + ((4 * sample) ^ square_row(j))); };
        const bool nonfinite = __any_sync(0xffffffffu, lane < 2 * kMaxPanels && bars->nonfinite[lane] != 0);
        auto emit = [&](int t, int buf, int c0, bool last) {  // outputs c0 .. c0 + 15 of tile t
            const long long o0 = static_cast<long long>(t) * kRows + c0;
            const float bias_l = p.bias && o0 + col < L ? __ldg(p.bias + o0 + col) : 0.f;
            tc::fence_after_sync();
            float v[16];
            tc::load16(tmem_d + buf * kRows + c0 + lane_base, v);
            int total = 0;  // repeated inputs of these outputs
#pragma unroll
            for (int w = 0; w < kListWarps; ++w) total += bars->listed[buf][c0 / kWarpRows + w];
            total = min(total, kListWarps * p.cap);
            const bool extra = total > 0 || nonfinite;
            if (MODE == 0 || extra) {
#pragma unroll
                for (int j = 0; j < 16; ++j) sq_at(j, lane) = v[j];
            }
            if (extra) {
                // x of the input is in tensor memory, in this warp's lanes
                const uint4* list = reinterpret_cast<const uint4*>(lists + (buf * kBuildWarps + c0 / kWarpRows) * p.cap);
#pragma unroll 1
                for (int e = 0; e < total; e += 4) {
                    const uint4 lo = list[e / 2], hi = list[e / 2 + 1];
                    const unsigned w[4] = {lo.x, lo.z, hi.x, hi.z}, at[4] = {lo.y, lo.w, hi.y, hi.w};
                    unsigned x[4];
                    tc::load_columns(tmem + lane_base, at[0] >> 23, at[1] >> 23, at[2] >> 23, at[3] >> 23, x);
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        float& z = *reinterpret_cast<float*>(sq + ((4 * lane) ^ (at[u] & 0x7f8u)));
                        z = fma_pair(x[u], w[u], z);
                    }
                }
                if (nonfinite) {
#pragma unroll 1
                    for (int j = 0; j < 16 && o0 + j < L; ++j)
                        sq_at(j, lane) = add_nonfinite(p, bars->nonfinite, o0 + j, b, sq_at(j, lane));
                }
            }
            tc::fence_before_sync();
            __syncwarp();
            if (last && lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_addr(bars->dfree + buf)) : "memory");
            if constexpr (MODE == 1) {
                if (extra) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = sq_at(j, lane);
                }
                const float scale = b < p.B ? p.scale : 0.f;
                const int rows = static_cast<int>(L - o0 < 16 ? (L - o0 < 0 ? 0 : L - o0) : 16);
                float* dst = p.gT + o0 * p.ldg + b;
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] += __shfl_sync(0xffffffffu, bias_l, j);
                if (p.loss_kind == FFI_LOSS_BCE && rows == 16) {
                    loss_local += bce_negative16(v);
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        float val, g;
                        loss_for_negative(p.loss_kind, v[j], val, g);
                        if (j < rows) loss_local += val;
                        v[j] = g;
                    }
                }
                if (b < p.ldg) {
                    if (rows == 16 && p.ldg == 128) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) dst[j * 128] = scale * v[j];
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (j < rows) dst[j * p.ldg] = scale * v[j];
                    }
                }
            } else {
                // the square is read back turned round, so that 16 lanes write a run of y
                const long long o = o0 + col;
                float* dst = p.y + static_cast<size_t>(b0 + q * 32 + (lane >> 4)) * L + o;
                const int left = o < L ? p.B - (b0 + q * 32 + (lane >> 4)) : 0;
#pragma unroll
                for (int rr = 0; rr < 16; ++rr) {
                    const float z = sq_at(col, 2 * rr + (lane >> 4)) + bias_l;
                    if (2 * rr < left) *dst = z;
                    dst += 2 * static_cast<long long>(L);
                }
                __syncwarp();
            }
        };
        int it = 0;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++it) {
            await(bars->ready + (it & 1), (it >> 1) & 1);
#pragma unroll 1
            for (int part = 0; part < 16 / EMIT; ++part) emit(t, it & 1, (warp >> 2) * (256 / EMIT) + part * 16, part == 16 / EMIT - 1);
        }
        if (MODE == 1 && b >= p.B) loss_local = 0.f;
    }

    if constexpr (MODE == 1) {
        double v = static_cast<double>(loss_local);
#pragma unroll
        for (int off = 16; off >= 1; off /= 2) v += __shfl_xor_sync(0xffffffffu, v, off);
        __syncthreads();
        double* red = reinterpret_cast<double*>(smem);
        if (lane == 0) red[warp] = v;
        __syncthreads();
        clear_loss_ticket(p.loss_partials);
        if (tid == 0) {
            double s = 0.0;
            for (int w = 0; w < kEmitWarps; ++w) s += red[w];
            p.loss_partials[static_cast<size_t>(blockIdx.y) * gridDim.x + blockIdx.x] = s;
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == kMmaWarp) tc::dealloc(tmem);
}

}  // namespace

// Where launch_forward_dense is the faster kernel.  Its time hardly depends on the batch or, in steps of 32, on K, that of the gather
// kernel (forward_bf16.cu) is proportional to K and, in tiles of 32, 64 or 128 columns, to the batch.  How often a row repeats
// an input is not known here: a table drawn with replacement (as FFILayer draws it and ffi_rewire edits it) has K*K / 2N
// repeats a row, one of distinct inputs none, and a line is drawn where both kinds are served.  Times are
// distinct / with replacement against the gather kernel, us:
//   * more than 64 samples (64: y 87 against 58 at N=768, L=670,091, K=32; 72 at L=300,000: 121/133 against 147);
//   * a fan-in of at most 64 (registers of the building warps) and a quarter of the inputs;
//   * at least 16 for y, 24 for the loss gradient (16: 53/59 against 60 and 62 against 62 at B=256, N=512, L=65,536);
//   * where the gather kernel cannot run (a fan-in off the multiples of 8, rows off the 16-byte boundaries) nothing else: the
//     alternatives widen x and W first (N=512, L=200,000, K=36: y 88/109 against 196; N=256, L=100,000, K=60: loss 62/136 against 142);
//   * else y up to a fan-in of an eighth of the inputs (B=256, N=512, L=65,536, K=64: 62/113 against 113; N=384, L=300,000, K=48: 117/201
//     against 192; beyond, N=256, L=100,000, K=48: 47/92 against 74),
//   * and the loss gradient, whose epilogue already fills the emitting warps, up to a twelfth, with K at 32 or not far below 64
//     (N=768, L=670,091: K=32 245/288 against 289, K=64 294/493 against 474, but K=24 245/278 against 251 and K=48 292/407 against
//     385; N=512, L=200,000: K=32 83/101 against 105, but K=40 103/140 against 118).
bool forward_dense_applicable(int64_t B, int64_t N, int64_t L, int64_t K, const void* W, const int32_t* idx, bool loss) {
    if (N > 64 * kMaxPanels || K > 64 || 4 * K > N || B <= 64 || K < (loss ? 24 : 16) || L <= 0) return false;
    if (K % 8 != 0 || reinterpret_cast<uintptr_t>(W) % 16 != 0 || reinterpret_cast<uintptr_t>(idx) % 16 != 0) return true;
    return loss ? 12 * K <= N && K >= 32 && round_up(K, 32) - K <= 8 : 8 * K <= N;
}

// y (or, with `loss`, the loss gradient and one loss partial per CTA) from bf16 x as [N][ldx] and bf16 W.
int launch_forward_dense(const void* xT, int64_t ldx, const int32_t* idx, const void* W, const float* bias, float* y, int64_t B,
                         int64_t N, int64_t L, int64_t K, const Bf16LossEpilogue* loss, cudaStream_t stream) {
    DeviceInfo dev;
    const int rc = get_device_info(&dev);
    if (rc != FFI_OK) return rc;
    DenseFwdParams p;
    p.xT = static_cast<const __nv_bfloat16*>(xT);
    p.ldx = ldx;
    p.idx = idx;
    p.W = static_cast<const unsigned short*>(W);
    p.bias = bias;
    p.y = y;
    p.B = static_cast<int>(B);
    p.N = static_cast<int>(N);
    p.L = static_cast<int>(L);
    p.K = static_cast<int>(K);
    p.panels = static_cast<int>(ceil_div(N, tc::kPanelK));
    p.gT = loss ? loss->gT : nullptr;
    p.ldg = loss ? loss->ldg : 0;
    p.scale = loss ? loss->scale : 0.f;
    p.loss_partials = loss ? loss->loss_partials : nullptr;
    p.loss_kind = loss ? loss->loss_kind : 0;
    const int64_t nBT = ceil_div(B, 128), tiles = ceil_div(L, kRows);
    const int64_t per_bt = dev.sm_count / nBT > 0 ? dev.sm_count / nBT : 1;
    const dim3 grid(static_cast<unsigned>(tiles < per_bt ? tiles : per_bt), static_cast<unsigned>(nBT));
    if (loss) *loss->ctas = static_cast<int>(grid.x * grid.y);
    auto go = [&](auto kern, int emit) -> int {
        // lists as long as a building warp's rows could need, or what is left of the shared memory
        const int build = kMmaWarp - emit;
        const size_t used = 2 * static_cast<size_t>(p.panels) * kPanelBytes + emit * 2048 + kListsAt;
        const int64_t longest = round_up(kRows / build * K, 4), room = (dev.max_smem_optin - static_cast<int64_t>(used)) / (2 * build * 32) * 4;
        p.cap = static_cast<int>(longest < room ? longest : room);
        const size_t smem = used + 2 * build * 8 * static_cast<size_t>(p.cap);
        FFI_CUDA_CHECK(prepare_kernel(reinterpret_cast<const void*>(kern), 0, smem, nullptr));
        FFI_CUDA_CHECK(launch_chained(kern, grid, dim3(kThreads), smem, stream, p));
        FFI_LAUNCH_CHECK("ffi_fwd_dense_kernel");
        return FFI_OK;
    };
    if (loss) return K <= 32 ? go(ffi_fwd_dense_kernel<1, 1, 16>, 16) : go(ffi_fwd_dense_kernel<1, 2, 8>, 8);
    return K <= 32 ? go(ffi_fwd_dense_kernel<0, 1, 16>, 16) : go(ffi_fwd_dense_kernel<0, 2, 8>, 8);
}

int dense_forward_timeouts(int* out) {
    FFI_CUDA_CHECK(cudaMemcpyFromSymbol(out, g_dense_timeouts, sizeof(int)));
    return FFI_OK;
}
int set_dense_forward_wait_limit(long long ticks) {
    FFI_CUDA_CHECK(cudaMemcpyToSymbol(g_dense_limit, &ticks, sizeof(ticks)));
    return FFI_OK;
}

}  // namespace ffi
