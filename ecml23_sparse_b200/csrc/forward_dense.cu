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
//     is never cleared as a whole: a warp owns four rows, remembers where it wrote and puts zeros back there, so a row of
//     K entries costs 2K two-byte stores instead of a row of N;
//   * entries of a row with the same input cannot share a cell (their sum is no bf16): one of them is written, the others
//     go to a short list that is added to the results with fp32 FMAs (x read from L2); what does not fit the list waits
//     for another round of the same tile that accumulates.  Tables without repeated inputs never do either;
//   * the warps specialise: 8 build tiles, one issues the N / 16 MMAs of a tile (M = 128, N = 64, K = 16), 8 turn D into y
//     or the loss gradient; mbarriers hand the buffers on, so the three stages of consecutive tiles overlap.  (With all
//     warps building and emitting in turn, one CTA barrier per tile, the stages' latencies added up: 214 us for y, 310 with
//     the BCE epilogue.)
// What bounds it: an MMA of M = 128 takes 62 clocks for any N up to 128 (measured), so the N = 64 that fits beside x costs
// 48 x 62 clocks per tile at N = 768 (110 us at L = 670,091); the building warps' chain of stores and the results' stores
// are about as long and overlap only in part.  Measured at B = 128, L = 670,091, against the gather kernels:
// N = 768, K = 32: y 234 (408) us, loss gradient 249 (284) us; K = 64: 325 (590) and 360 (468) us; inputs drawn with
// replacement: 296 (403) and 325 (286) us; B = 256, N = 512, L = 65,536, K = 64: y 66 (196) us.
#include <type_traits>

#include "tcgen05.cuh"

namespace ffi {
namespace {

__device__ int g_dense_timeouts = 0;                // bounded waits of this kernel that gave up
__device__ long long g_dense_limit = 4000000000ll;  // clock64 ticks a wait may last (about two seconds)
constexpr long long kDrainLimit = 4000000000ll;     // ... and the last one, for MMAs that are under way, whatever that is set to

constexpr int kEmitWarps = 16, kBuildWarps = 8;  // warps 0..15 write results, 16..23 build tiles, 24 issues the MMAs
constexpr int kMmaWarp = kEmitWarps + kBuildWarps;
constexpr int kThreads = 32 * (kMmaWarp + 1);
constexpr int kRows = 64;                     // outputs per tile
constexpr int kWarpRows = kRows / kBuildWarps;
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

constexpr int kExtras = 19;  // per building warp and tile (8 rows): the shared memory that N = 768 leaves

struct DenseBarriers {
    unsigned long long full[2];    // a tile is built (one arrival per building warp)
    unsigned long long done[2];    // its MMAs are done: the tile buffer is free
    unsigned long long ready[2];   // ... and no further round follows: D is complete
    unsigned long long dfree[2];   // D has been read (one arrival per emitting warp)
    unsigned long long idle;       // all MMAs of the CTA are done
    unsigned tmem;
    int more[2];                   // another round of this tile follows
    int extras[2][kBuildWarps];    // entries in the lists below
    uint2 extra[2][kBuildWarps][kExtras];  // (input | row of the tile << 16, weight) of repeated inputs
    int bad;                       // a wait gave up: everybody runs through without waiting, the results are void
    unsigned nonfinite[2 * kMaxPanels];  // inputs with a sample of this tile that is infinite or NaN
};

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

// MODE 0 writes y, 1 the loss gradient.  KG: entries of a row per lane (K <= 32 * KG).
template <int MODE, int KG>
__global__ void __launch_bounds__(kThreads, 1) ffi_fwd_dense_kernel(DenseFwdParams p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b0 = blockIdx.y * 128;
    const int K = p.K, L = p.L;
    const unsigned tileBytes = p.panels * kPanelBytes;
    float* ys = reinterpret_cast<float*>(smem + 2 * tileBytes);  // [warp][32 samples][16 outputs]
    DenseBarriers* bars = reinterpret_cast<DenseBarriers*>(smem + 2 * tileBytes + kEmitWarps * 2048);
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
    for (unsigned e = tid; e < sizeof(bars->extra) / 4; e += kThreads) reinterpret_cast<unsigned*>(bars->extra)[e] = 0;
    if (tid < 2 * kBuildWarps) bars->extras[0][tid] = 0;
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
                    const unsigned base = tc::smem_addr(smem) + buf * tileBytes;
                    for (int m = 0; m < 4 * p.panels; ++m)
                        tc::mma(tmem_d + buf * kRows, tmem + m * 8, tc::panel_desc(base + (m >> 2) * kPanelBytes + (m & 3) * 32),
                                tc::instr_desc(kRows), !first || m > 0);
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
            int extras = 0;
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
                bool left = false;
                // the list of this buffer's tile before has been read
                if (first && use > 0) await(bars->dfree + buf, (use - 1) & 1);
                if (__any_sync(0xffffffffu, lost != 0)) {
#pragma unroll
                    for (int r = 0; r < kWarpRows; ++r)
#pragma unroll
                        for (int g = 0; g < KG; ++g) {
                            const bool mine_lost = lost >> (r * KG + g) & 1u;
                            const unsigned who = __ballot_sync(0xffffffffu, mine_lost);
                            const int slot = extras + __popc(who & ((1u << lane) - 1u));
                            if (mine_lost && slot < kExtras) {
                                bars->extra[buf][bw][slot] = make_uint2(static_cast<unsigned>(ir[r][g]) | (bw * kWarpRows + r) << 16,
                                                                        static_cast<unsigned>(wr[r][g]) << 16);
                                wr[r][g] = 0;
                            } else if (mine_lost) {
                                left = true;
                            }
                            extras = min(kExtras, extras + __popc(who));
                        }
                }
                if (lane == 0) bars->extras[buf][bw] = extras;
                tc::fence_smem();
                unsigned again;
                asm volatile(
                    "{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\n"
                    "barrier.cta.red.or.pred q, 1, %2, p;\nselp.u32 %0, 1, 0, q;\n}"
                    : "=r"(again)
                    : "r"(static_cast<unsigned>(left && !*bad)), "n"(32 * kBuildWarps)
                    : "memory");
                if (lane == 0) {
                    if (bw == 0) *static_cast<volatile int*>(&bars->more[buf]) = static_cast<int>(again);
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_addr(bars->full + buf)) : "memory");
                }
                if (!again) break;  // one answer for the eight warps, which meet at the barrier above
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
        const int q = warp & 3, c0 = (warp >> 2) * 16;  // this warp's samples and outputs within the tile
        const int b = b0 + q * 32 + lane;
        float* sq = ys + warp * 512;  // its [32 samples][16 outputs] square, rows rotated (conflict-free both ways)
        auto sq_at = [&](int row, int col) -> float& { return sq[row * 16 + ((col + (row >> 1)) & 15)]; };
        const bool nonfinite = __any_sync(0xffffffffu, lane < 2 * kMaxPanels && bars->nonfinite[lane] != 0);
        int it = 0;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++it) {
            const int buf = it & 1;
            const long long o0 = static_cast<long long>(t) * kRows + c0;
            const int col = lane & 15;
            const float bias_l = p.bias && o0 + col < L ? __ldg(p.bias + o0 + col) : 0.f;
            await(bars->ready + buf, (it >> 1) & 1);
            tc::fence_after_sync();
            float v[16];
            tc::load16(tmem_d + buf * kRows + c0 + lane_base, v);
            tc::fence_before_sync();
            // repeated inputs of these 16 outputs (two building warps)
            const int n0 = bars->extras[buf][(c0 >> 3)], n1 = bars->extras[buf][(c0 >> 3) + 1];
            const bool extra = n0 + n1 > 0 || nonfinite;
            if (MODE == 0 || extra) {
#pragma unroll
                for (int j = 0; j < 16; ++j) sq_at(lane, j) = v[j];
            }
            if (extra) {
                for (int e = 0; e < n0 + n1; ++e) {
                    const uint2 x = e < n0 ? bars->extra[buf][c0 >> 3][e] : bars->extra[buf][(c0 >> 3) + 1][e - n0];
                    const float xv = b < p.B ? widen(p.xT[static_cast<size_t>(x.x & 0xffffu) * p.ldx + b]) : 0.f;
                    float& z = sq_at(lane, static_cast<int>(x.x >> 16) - c0);
                    z = fmaf(__uint_as_float(x.y), xv, z);
                }
                if (nonfinite) {
#pragma unroll 1
                    for (int j = 0; j < 16 && o0 + j < L; ++j)
                        sq_at(lane, j) = add_nonfinite(p, bars->nonfinite, o0 + j, b, sq_at(lane, j));
                }
            }
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_addr(bars->dfree + buf)) : "memory");
            if constexpr (MODE == 1) {
                if (extra) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = sq_at(lane, j);
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
                    const float z = sq_at(2 * rr + (lane >> 4), col) + bias_l;
                    if (2 * rr < left) *dst = z;
                    dst += 2 * static_cast<long long>(L);
                }
                __syncwarp();
            }
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

// Where launch_forward_dense is the faster kernel.  Its time hardly depends on K or the batch, the gather kernel's
// (forward_bf16.cu) is proportional to K and, in tiles of 32, 64 or 128 columns, to the batch:
//   * more than 64 samples (128: y 236 against 370 us and loss gradient 242 against 272 at N=768, L=670,091, K=32, y 30 against
//     53 at N=256, L=100,000; 64: 87 against 58 and 31 against 32);
//   * a fan-in of at least 16 for y and 24 for the loss gradient (16: 43 against 51 and 50 against 47 us at B=256, N=512,
//     L=65,536; 8: y 45 against 41);
//   * a fan-in of at most 64 (registers of the building warps) and a quarter of the inputs: beyond, repeated inputs in a row
//     are so frequent that their list overflows (N=150, K=40 drawn with replacement: 602 against 215 us).
bool forward_dense_applicable(int64_t B, int64_t N, int64_t L, int64_t K, bool loss) {
    return N <= 64 * kMaxPanels && K <= 64 && 4 * K <= N && B > 64 && K >= (loss ? 24 : 16) && L > 0;
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
    const size_t smem = 2 * static_cast<size_t>(p.panels) * kPanelBytes + kEmitWarps * 2048 + sizeof(DenseBarriers);
    const int64_t nBT = ceil_div(B, 128), tiles = ceil_div(L, kRows);
    const int64_t per_bt = dev.sm_count / nBT > 0 ? dev.sm_count / nBT : 1;
    const dim3 grid(static_cast<unsigned>(tiles < per_bt ? tiles : per_bt), static_cast<unsigned>(nBT));
    if (loss) *loss->ctas = static_cast<int>(grid.x * grid.y);
    auto go = [&](auto kern) -> int {
        FFI_CUDA_CHECK(prepare_kernel(reinterpret_cast<const void*>(kern), 0, smem, nullptr));
        kern<<<grid, kThreads, smem, stream>>>(p);
        FFI_LAUNCH_CHECK("ffi_fwd_dense_kernel");
        return FFI_OK;
    };
    if (loss) return K <= 32 ? go(ffi_fwd_dense_kernel<1, 1>) : go(ffi_fwd_dense_kernel<1, 2>);
    return K <= 32 ? go(ffi_fwd_dense_kernel<0, 1>) : go(ffi_fwd_dense_kernel<0, 2>);
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
