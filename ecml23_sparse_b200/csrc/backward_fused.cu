// grad_x and grad_W of the fixed-fan-in sparse layer in ONE pass over the transposed index (narrow inputs):
//   grad_x[b,i] = sum over entries (o,k) with idx[o,k]==i of W[o,k] * g[b,o]
//   grad_W[o,k] = sum_b g[b,o] * x[b, idx[o,k]]
//
// Replaces, for that case, both halves of the reference's grad functor
// (tfsparse/cc/kernels/backward.cu.h:112-133: feature_grad_launch_vector_tp + the
// weight_grad launch).  Walking the entries grouped by input i means x[:, i] is the same for a
// whole run of entries, so grad_W needs NO gather of its own: the
// g[:, o] vector gathered for grad_x is multiplied by x[:, i] and reduced over the lanes.  This
// removes the B*L*K shared-memory gathers of a separate grad_W pass.
//
// A launch covers up to 128 batch columns; larger batches run one launch per tile of 128 (grad_W of a later tile adds to
// what the tile before stored: one addition per element and launch, in tile order).
//
// Structure (per CTA = range of chunks x slice of 16*ni inputs; warp = ni inputs): see the comment at
// ffi_bwd_runs_kernel.  grad_x partials are flushed every few chunks, one per range, and the ranges are added in fp64 in
// a fixed order.  Results are bit-reproducible.
#include <cuda.h>

#include <type_traits>

#include "packed.cuh"
#include "tcgen05.cuh"

namespace ffi {
int peer_wait_timeouts(int* out);  // peer_reduce.cu
int set_peer_wait_limit(long long ticks);
int dense_forward_timeouts(int* out);  // forward_dense.cu
int set_dense_forward_wait_limit(long long ticks);
namespace {
__device__ int g_wait_timeouts = 0;  // bounded waits of this file's kernels that gave up
__device__ long long g_wait_limit = 4000000000ll;  // clock64 ticks a wait may last (about two seconds)
constexpr long long kDrainLimit = 4000000000ll;    // ... and one for a copy that has to end before the CTA does

constexpr int kWarps = 16;                  // warps that walk
constexpr int kThreads = 32 * kWarps + 32;  // ... and one that fetches the g tiles and sums grad_bias
constexpr int kDRow = 36;                   // row stride of the per-warp dot buffer (32 dots): 16-byte rows, conflict-free
constexpr int kPosRegs = 8;                 // positions per lane kept in registers ahead of their staging
constexpr int kKShift = 18;                 // entry code = byte offset of the g row in its tile | position in the chunk << 18
constexpr int kBounds = 36;                 // ints per warp and staging buffer: where its runs (or their halves) start
// The kernel of uneven tables: in a chunk where the longest run of a bundle has more than twice the average and kLongRun entries, what
// it has more than the others is walked by all lane groups.  No run walked side by side exceeds kSideBySide: a group whose run has
// ended fetches on, unused, and must stay inside shared memory (see dbuf and bounds, which follow the entries).
constexpr int kLongRun = 16, kSideBySide = kFusedLongestRun;
static_assert(kFusedNI * 2 + 1 < kBounds && kFusedWarps == kWarps, "bounds of the halves of a warp's runs");

struct BwdFusedParams {
    const void* W;   // fp32 or bf16 (TX)
    const float* gT;
    long long ldg;
    const void* xT;  // same element type as W
    long long ldx;
    const int* cperm;
    const int* cptr;
    const int* order;  // UNEVEN: the input at each place of the chunked lists, or nullptr: in order
    float* partial;  // [R][N][Bpad]
    float* gW;
    float* gbias;  // grad_bias[o] = sum_b gT[o][b], from the g tiles at hand anyway; or nullptr
    int B, N, L, K;
    int kShift;  // log2(K) when K is a power of two, else -1
    int T;       // rows per chunk
    long long nChunks;
    int R;
    int Bpad;
    int segChunks;  // chunks per flushed partial
    int ni;         // inputs per warp
    int longRun;    // UNEVEN: kLongRun, or 0 where the lane groups share all runs (shares_runs)
    int boxes;      // TMA boxes per tile (at most 256 rows each)
    int lastHalf;   // bf16 W of an odd number of elements: position of the last one, which has no whole word; else -1
    bool xVec;      // rows of x start on 8 bytes; what lies behind an odd B in them is zero
    int entOff[kWarps + 1];  // where each warp's entries start in a staging buffer
};

// ---- mbarrier + TMA (tiled bulk copies of g tiles, no multicast) ------------------------------

__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc::smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_addr(bar)) : "memory");
}
// Box of the 2-D tensor `map` with first element (x, y) -> dst; completion is signalled on `bar`.
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            tc::smem_addr(dst)),
        "l"(map), "r"(x), "r"(y), "r"(tc::smem_addr(bar))
        : "memory");
}
// Waits for the phase with the given parity, at most g_wait_limit ticks or until another thread of the CTA has given up.
__device__ __forceinline__ bool mbar_wait_or_dead(unsigned long long* bar, unsigned parity, volatile int* dead) {
    if (tc::bar_try_wait(bar, parity)) return true;
    const long long start = clock64(), limit = g_wait_limit;
    while (!tc::bar_try_wait(bar, parity)) {
        if (*dead) return false;
        if (clock64() - start > limit) {
            atomicAdd(&g_wait_timeouts, 1);
            *dead = 1;
            return false;
        }
    }
    return true;
}

// The VPL batch columns one lane of a group of LG lanes holds: pieces of 4 at columns 4q + m * 4 * LG.
template <int VPL, int LG>
struct LaneVec {
    static constexpr int kPairs = VPL / 2;
    u64 v[kPairs];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int j = 0; j < kPairs; ++j) v[j] = 0ull;
    }
    // ptr: this lane's first column
    __device__ __forceinline__ void load_shared(const unsigned char* ptr) {
#pragma unroll
        for (int m = 0; m < VPL / 4; ++m) {
            const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(ptr + m * (16 * LG));
            v[2 * m] = t.x, v[2 * m + 1] = t.y;
        }
    }
    __device__ __forceinline__ void axpy(float w, const LaneVec& g) {
        const u64 ww = pack2(w, w);
#pragma unroll
        for (int j = 0; j < kPairs; ++j) v[j] = fma2(ww, g.v[j], v[j]);
    }
    __device__ __forceinline__ float dot(const LaneVec& g) const {
        float lo, hi;
        if constexpr (kPairs >= 8) {  // two chains
            u64 s = mul2(g.v[0], v[0]), t = mul2(g.v[1], v[1]);
#pragma unroll
            for (int j = 2; j < kPairs; j += 2) s = fma2(g.v[j], v[j], s), t = fma2(g.v[j + 1], v[j + 1], t);
            unpack2(fma2(pack2(1.f, 1.f), s, t), lo, hi);
        } else {
            u64 s = mul2(g.v[0], v[0]);
#pragma unroll
            for (int j = 1; j < kPairs; ++j) s = fma2(g.v[j], v[j], s);
            unpack2(s, lo, hi);
        }
        return lo + hi;
    }
    // what lane `src` holds
    __device__ __forceinline__ void from_lane(int src) {
#pragma unroll
        for (int j = 0; j < kPairs; ++j) v[j] = __shfl_sync(0xffffffffu, v[j], src);
    }
    // the sum over the lane groups, in all of them
    __device__ __forceinline__ void add_groups() {
#pragma unroll
        for (int j = 0; j < kPairs; ++j)
#pragma unroll
            for (int off = LG; off < 32; off *= 2) v[j] = fma2(pack2(1.f, 1.f), v[j], __shfl_xor_sync(0xffffffffu, v[j], off));
    }
    __device__ __forceinline__ float sum() const {
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < kPairs; j += 2) {
            float f[4];
            unpack2(v[j], f[0], f[1]), unpack2(v[j + 1], f[2], f[3]);
            s += (f[0] + f[1]) + (f[2] + f[3]);
        }
        return s;
    }
};

// 2 * VPL columns of this thread's TMEM lane -> (sums, x) of its group's input, complete on return.  The 32-bit halves are paired
// inside the asm blocks so that the loaded registers ARE the pairs.
template <int LG>
__device__ __forceinline__ void tmem_load_input(unsigned taddr, LaneVec<16, LG>& a, LaneVec<16, LG>& x) {
    asm volatile(
        "{\n"
        ".reg .b32 t<32>;\n"
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {t0, t1, t2, t3, t4, t5, t6, t7, t8, t9, t10, t11, t12, t13, t14, t15,\n"
        " t16, t17, t18, t19, t20, t21, t22, t23, t24, t25, t26, t27, t28, t29, t30, t31}, [%16];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        "mov.b64 %0, {t0, t1};\n mov.b64 %1, {t2, t3};\n mov.b64 %2, {t4, t5};\n mov.b64 %3, {t6, t7};\n"
        "mov.b64 %4, {t8, t9};\n mov.b64 %5, {t10, t11};\n mov.b64 %6, {t12, t13};\n mov.b64 %7, {t14, t15};\n"
        "mov.b64 %8, {t16, t17};\n mov.b64 %9, {t18, t19};\n mov.b64 %10, {t20, t21};\n mov.b64 %11, {t22, t23};\n"
        "mov.b64 %12, {t24, t25};\n mov.b64 %13, {t26, t27};\n mov.b64 %14, {t28, t29};\n mov.b64 %15, {t30, t31};\n"
        "}"
        : "=l"(a.v[0]), "=l"(a.v[1]), "=l"(a.v[2]), "=l"(a.v[3]), "=l"(a.v[4]), "=l"(a.v[5]), "=l"(a.v[6]), "=l"(a.v[7]),
          "=l"(x.v[0]), "=l"(x.v[1]), "=l"(x.v[2]), "=l"(x.v[3]), "=l"(x.v[4]), "=l"(x.v[5]), "=l"(x.v[6]), "=l"(x.v[7])
        : "r"(taddr)
        : "memory");
}
template <int LG>
__device__ __forceinline__ void tmem_load_input(unsigned taddr, LaneVec<8, LG>& a, LaneVec<8, LG>& x) {
    asm volatile(
        "{\n"
        ".reg .b32 t<16>;\n"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {t0, t1, t2, t3, t4, t5, t6, t7, t8, t9, t10, t11, t12, t13, t14, t15}, [%8];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        "mov.b64 %0, {t0, t1};\n mov.b64 %1, {t2, t3};\n mov.b64 %2, {t4, t5};\n mov.b64 %3, {t6, t7};\n"
        "mov.b64 %4, {t8, t9};\n mov.b64 %5, {t10, t11};\n mov.b64 %6, {t12, t13};\n mov.b64 %7, {t14, t15};\n"
        "}"
        : "=l"(a.v[0]), "=l"(a.v[1]), "=l"(a.v[2]), "=l"(a.v[3]), "=l"(x.v[0]), "=l"(x.v[1]), "=l"(x.v[2]), "=l"(x.v[3])
        : "r"(taddr)
        : "memory");
}
template <int LG>
__device__ __forceinline__ void tmem_load_input(unsigned taddr, LaneVec<4, LG>& a, LaneVec<4, LG>& x) {
    asm volatile(
        "{\n"
        ".reg .b32 t<8>;\n"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {t0, t1, t2, t3, t4, t5, t6, t7}, [%4];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        "mov.b64 %0, {t0, t1};\n mov.b64 %1, {t2, t3};\n mov.b64 %2, {t4, t5};\n mov.b64 %3, {t6, t7};\n"
        "}"
        : "=l"(a.v[0]), "=l"(a.v[1]), "=l"(x.v[0]), "=l"(x.v[1])
        : "r"(taddr)
        : "memory");
}
// VPL columns of this thread's TMEM lane, four at a time
template <int VPL, int LG>
__device__ __forceinline__ void tmem_store(unsigned taddr, const LaneVec<VPL, LG>& a) {
#pragma unroll
    for (int j = 0; j < VPL / 2; j += 2)
        asm volatile(
            "{\n"
            ".reg .b32 t<4>;\n"
            "mov.b64 {t0, t1}, %1;\n mov.b64 {t2, t3}, %2;\n"
            "tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {t0, t1, t2, t3};\n"
            "}" ::"r"(taddr + 2 * j),
            "l"(a.v[j]), "l"(a.v[j + 1])
            : "memory");
}

// =====================================================================================
// G lane groups per warp and VPL batch columns per lane: a group of LG = 32/G lanes covers the BT = VPL*LG batch columns, and the
// groups of a warp walk the runs of G different inputs at a time (a bundle), one entry each per step:
//   batch 65..128: G = 4, VPL = 16;  33..64: G = 4, VPL = 8;  17..32: G = 4, VPL = 4;  9..16: G = 8;  up to 8: G = 16 (VPL = 4).
//
// What bounds it is the shared-memory data pipe and the issue slots: the 4 wavefronts of a row of 128 columns cannot be saved, but
// the fetch of an entry, the store of the lanes' partial dots and their summing up cost about one each per STEP, so the more entries
// a step holds the better.  That the groups work on different inputs means that nothing has to be merged, an input's state is held
// once (16 inputs per warp, so three slices read a tile of 768 inputs, not six), and getting it costs a quarter; the price is
// that a bundle lasts as long as its longest run.
//
// The sums of grad_x and x[:, i] of a warp's 16 inputs are too many for its registers.  Both live in tensor memory (TMEM,
// otherwise unused here): TMEM lane = thread lane of the warp's quarter, 2 * VPL columns per bundle (sums | x).  A bundle
// starts with one load of its columns and ends with a store of the sums, so the loop over the bundles needs no unrolling.
//
// There is no barrier between the warps.  A warp of its own fetches the g tiles (TMA, [rows][BT], rows past L arrive as zeros)
// into two buffers as the walking warps hand them back, and each walking warp stages its own entries: flat positions come a chunk
// ahead and are turned into (W, code) pairs, with W by 4-byte cp.async that completes behind the walk.  So a tile's copy is
// hidden, and the unequal numbers of entries that warps have in a chunk even out.  With 65..128 columns a tile is half a chunk's rows
// (HALVES = 2: both buffers together hold what shared memory can), and a run is walked in two parts, whose border is searched
// when the entries are staged.
//
// Backward with grad_bias from the transposed gradient, N=768, L=670,091, K=32, us: two entries of ONE input per step, six slices, one
// tile, barriers at the chunk's edges -> now: B=128 950 -> 828 (bf16 965 -> 843), 64 707 -> 505, 32 559 -> 367, 16 485 -> 271,
// 8 436 -> 222; B=256, N=512, L=65,536, K=64, bf16 357 -> 313; 513 rows, B=127, N=254, K=73 18.3 -> 16.7.
// Without the warp that fetches (the last warp done with a tile asks for the next; 128 instead of 96 registers): 882 to 921 at B=128.
//
// UNEVEN: a bundle lasts as long as its longest run, so a hot input, walked by one lane group, holds up its warp and the warp its CTA.
// Tables with such inputs have theirs dealt to slices and warps by count (plan_build) and a kernel that lets all groups walk what a
// run has more than the others of its bundle, every G-th entry each (x of the input handed round by shuffles, the groups' sums added
// at the end), and that stages a warp's thousands of entries with as many loads in flight as there are registers for.  What bounds
// it is the chain of the warp that has the hottest input: 13.9 ns an entry at 64 columns, 6 at 8.  Backward at N=768, L=670,091, K=32,
// us, before -> now; "two": grad_x and grad_W by a kernel each, because the entries of the warps did not fit:
//   inputs drawn by Zipf's law, exponent 0.4: B=128 1,310 -> 1,029, 64 904 -> 620, 32 615 -> 462, 8 428 -> 280
//   exponent 0.8: 128 1,973 (two) -> 1,373, 64 1,300 (two) -> 811, 32 2,194 -> 632, 8 1,968 -> 384
//   exponent 1:   128 2,350 (two) -> 1,788, 64 1,375 (two) -> 1,110, 32 4,067 -> 889, 8 3,856 -> 548
//   30 % of the links added to the leading quarter of the inputs: 128 1,974 (two) -> 862, 64 1,201 (two) -> 517
// Warps with fewer inputs than lane groups take this variant, too (see shares_runs), and share all runs longer than one and a half times
// the average of a full bundle (longRun = 0): side by side most groups had no input.  L=300,000, us, before -> now: N=10, K=8 B=128
// 263 -> 114, 8 134 -> 45; N=32, K=16 128 246 -> 177, 8 119 -> 65.  (With longRun 4, 8, 12 and 15 over 112 such shapes 1, 2, 3 and 6 % slower.)
// (An even table: 813, 499, 356, 224.)  With a fifth or more of all links to ONE input two kernels are faster again, see fused_pays.
// In one kernel with the even case and a flag looked up per chunk, even tables took 2 to 6 % longer (registers).
//
// ACC: a batch tile after the first (as a run-time flag it cost 5 %), whose grad_W and grad_bias add to what the tiles
// before stored.
// TX is the storage type of x and W.  bf16 x is widened (exactly) on its way into tensor memory.  A bf16
// weight is fetched as the aligned 4-byte word that holds it (cp.async copies at least 4 bytes) and turned
// into its fp32 bit pattern by the lane that fetched it once the copy has landed (the entry's code tells
// which half: the chunk's first position is even, so the parity of the position within the chunk is the
// parity of the flat position).  W has to start on a word; of the last element of an odd number two bytes are copied.
// =====================================================================================
template <int G, int VPL, int HALVES, typename TX, bool ACC, bool UNEVEN>
__global__ void __launch_bounds__(kThreads, 1) ffi_bwd_runs_kernel(const __grid_constant__ BwdFusedParams p, const __grid_constant__ CUtensorMap g_map) {
    constexpr bool kBf16 = !std::is_same<TX, float>::value;
    constexpr int LG = 32 / G, BT = VPL * LG, COLS = 2 * VPL, NB = kFusedNI / G, SLOTS = 32 / G;
    constexpr unsigned kAll = 0xffffffffu, kRowMask = (1u << kKShift) - 1u;
    static_assert(kFusedNI % G == 0 && (kWarps / 4) * NB * COLS <= tc::kCols, "the warps of a lane quarter share the TMEM columns");
    static_assert((kSideBySide + SLOTS) * 8 <= kWarps * (SLOTS * kDRow + 2 * kBounds) * 4, "fetches past the last run stay inside shared memory");
    using LaneT = LaneVec<VPL, LG>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const int T = p.T, K = p.K, N = p.N, ni = p.ni;
    const int rows = T / HALVES;  // of a tile
    const unsigned tileBytes = static_cast<unsigned>(rows) * (BT * 4);
    unsigned char* tiles_s = smem_raw;                                                 // [2][rows][BT] floats
    unsigned char* zero_s = smem_raw + 2 * tileBytes;                                  // a row of zeros
    uint2* ent_s = reinterpret_cast<uint2*>(zero_s + BT * 4);                          // [2][entOff[kWarps]]
    float* dbuf_s = reinterpret_cast<float*>(ent_s + 2 * p.entOff[kWarps]);            // [kWarps][SLOTS][kDRow]
    int* bounds_s = reinterpret_cast<int*>(dbuf_s + kWarps * SLOTS * kDRow);           // [kWarps][2][kBounds]
    unsigned long long* full = reinterpret_cast<unsigned long long*>(bounds_s + kWarps * 2 * kBounds);  // [2] tile has arrived
    unsigned long long* empty = full + 2;                                              // [2] tile is no longer needed
    unsigned* tmem_base_p = reinterpret_cast<unsigned*>(empty + 2);
    volatile int* dead = reinterpret_cast<volatile int*>(tmem_base_p + 1);             // somebody has given up on a wait

    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int grp = lane / LG, q = lane % LG;
    const int r = blockIdx.x;
    const int i_lo = blockIdx.y * (kWarps * ni);
    const long long c_begin = p.nChunks * r / p.R;
    const long long c_end = p.nChunks * (r + 1) / p.R;
    const bool turns = p.gbias != nullptr;  // the fetching warp reads tiles, too

    chain_wait();
    if (warp == 0) tc::alloc(tmem_base_p);
    if (threadIdx.x == 32) {
        for (int b = 0; b < 2; ++b) tc::bar_init(full + b, 1), tc::bar_init(empty + b, kWarps + (turns ? 1 : 0));
        *dead = 0;
    }
    if (threadIdx.x < BT) reinterpret_cast<float*>(zero_s)[threadIdx.x] = 0.f;
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();

    if (warp == kWarps) {
        // ---- the warp that fetches -----------------------------------------------------------
        const int passes = static_cast<int>(c_end - c_begin) * HALVES;
        auto fetch = [&](int t) {
            if (lane == 0) {
                const long long y = c_begin * T + static_cast<long long>(t) * rows;
                unsigned long long* bar = full + (t & 1);
                tc::fence_smem();
                mbar_expect_tx(bar, tileBytes);
                const int box = rows / p.boxes;
                for (int h = 0; h < p.boxes; ++h)
                    tma_load_2d(tiles_s + (t & 1) * tileBytes + h * box * (BT * 4), &g_map, 0, static_cast<int>(y) + h * box, bar);
            }
        };
        int issued = 0;
        for (; issued < 2 && issued < passes; ++issued) fetch(issued);
        for (int t = 0; t < passes; ++t) {
            if (turns) {
                if (__any_sync(kAll, !mbar_wait_or_dead(full + (t & 1), (t >> 1) & 1, dead))) break;
                // grad_bias of the tile's rows: the slices of a range take turns, each row is one group's sum
                if (static_cast<int>((c_begin * HALVES + t) % gridDim.y) == static_cast<int>(blockIdx.y)) {
                    const long long o0 = c_begin * T + static_cast<long long>(t) * rows;
                    const unsigned char* gs = tiles_s + (t & 1) * tileBytes + q * 16;
                    for (int r0 = 0; r0 < rows; r0 += 2 * G) {  // two rows of a group in flight
                        float sum[2] = {0.f, 0.f};
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int rr = r0 + u * G + grp;
                            LaneT v;
                            v.zero();
                            if (rr < rows) v.load_shared(gs + rr * (BT * 4));
                            sum[u] = v.sum();
                        }
#pragma unroll
                        for (int off = LG / 2; off >= 1; off /= 2)
#pragma unroll
                            for (int u = 0; u < 2; ++u) sum[u] += __shfl_xor_sync(kAll, sum[u], off);
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int rr = r0 + u * G + grp;
                            if (q == 0 && rr < rows && o0 + rr < p.L) p.gbias[o0 + rr] = ACC ? p.gbias[o0 + rr] + sum[u] : sum[u];
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(empty + (t & 1));
            }
            if (t + 2 < passes) {
                if (__any_sync(kAll, !mbar_wait_or_dead(empty + (t & 1), (t >> 1) & 1, dead))) break;
                fetch(t + 2);
                issued = t + 3;
            }
        }
        // No copy may be under way when the CTA releases its shared memory: where the others have given up, wait for the last
        // ones here (bounded, but not by a limit that a caller has lowered).
        for (int t = issued > 2 ? issued - 2 : 0; t < issued; ++t) tc::bar_wait(full + (t & 1), (t >> 1) & 1, kDrainLimit);
    } else {
        // ---- the warps that walk -------------------------------------------------------------
        const TX* xT = static_cast<const TX*>(p.xT);
        const int iw = i_lo + warp * ni;                 // this warp's first input, or its place
        auto input_at = [&](int i) { return UNEVEN && p.order ? __ldg(p.order + i) : i; };
        const int nb = (ni + G - 1) / G;                 // its bundles
        // lanes 32*(warp % 4) .. +31 are the ones this warp may touch; its bundles take NB*COLS columns
        const unsigned taddr0 = *tmem_base_p + ((static_cast<unsigned>(warp & 3) * 32u) << 16) + static_cast<unsigned>(warp >> 2) * (NB * COLS);
        // x of the warp's inputs: all loads are under way before the first is stored (one bundle at a time, this prologue took a third
        // of a small launch)
        {
            LaneT x[NB], zero;
            zero.zero();
#pragma unroll
            for (int j = 0; j < NB; ++j) {
                const int k = j * G + grp;
                int i = iw + k;
                if (UNEVEN && k < ni && i < N) i = input_at(i);
#pragma unroll
                for (int m = 0; m < VPL; m += 2) {
                    const int b = (m / 4) * (4 * LG) + 4 * q + (m & 3);
                    float f[2];
                    if (VPL == 16 && !kBf16 && p.xVec) {  // two neighbours at a time
                        const float2 w = k < ni && i < N && b < p.B
                                             ? *reinterpret_cast<const float2*>(static_cast<const float*>(p.xT) + static_cast<size_t>(i) * p.ldx + b)
                                             : make_float2(0.f, 0.f);
                        f[0] = w.x, f[1] = w.y;
                    } else {
#pragma unroll
                        for (int u = 0; u < 2; ++u)
                            f[u] = (k < ni && i < N && b + u < p.B) ? widen(xT[static_cast<size_t>(i) * p.ldx + b + u]) : 0.f;
                    }
                    x[j].v[m / 2] = pack2(f[0], f[1]);
                }
            }
#pragma unroll
            for (int j = 0; j < NB; ++j) {
                tmem_store(taddr0 + j * COLS, zero);
                tmem_store(taddr0 + j * COLS + VPL, x[j]);
            }
        }
        tc::wait_store();

        const int entOff = p.entOff[warp], entBuf = p.entOff[kWarps];
        float* dbuf = dbuf_s + warp * (SLOTS * kDRow);
        int* bnd_s = bounds_s + warp * (2 * kBounds);

        // Staging runs ahead of the walk.  bnd (lanes 0..ni): where the runs of the chunk to be staged next start; bnd_next: of the chunk
        // after it.  With one tile per chunk its positions wait in registers from one chunk to the next; with two tiles, where registers
        // are short, they are copied to where the codes will be, and turned into these between the halves.
        constexpr int kRegs = HALVES == 1 ? kPosRegs : 1;
        int pos[kRegs];
        int bnd = 0, bnd_next = 0;
        auto load_bounds = [&](long long c) { return c < c_end && lane <= ni ? __ldg(p.cptr + c * (N + 1) + min(iw + lane, N)) : 0; };
        auto load_pos = [&](long long c) {
            const int e_lo = __shfl_sync(kAll, bnd, 0), cnt = __shfl_sync(kAll, bnd, ni) - e_lo;
            const int* src = p.cperm + c * static_cast<long long>(T) * K + e_lo;
            if constexpr (HALVES == 1) {
#pragma unroll
                for (int u = 0; u < kRegs; ++u) {
                    const int e = lane + u * 32;
                    pos[u] = e < cnt ? __ldg(src + e) : -1;
                }
            } else {
                uint2* dst = ent_s + (static_cast<int>(c - c_begin) & 1) * entBuf + entOff;
                for (int e = lane; e < cnt; e += 32) __pipeline_memcpy_async(&dst[e].y, src + e, 4);
                __pipeline_commit();
            }
        };
        auto stage_one = [&](uint2* d, int ps, int pos0) {
            if constexpr (kBf16) __pipeline_memcpy_async(&d->x, static_cast<const unsigned*>(p.W) + (ps >> 1), 4, ps == p.lastHalf ? 2 : 0);
            else __pipeline_memcpy_async(&d->x, static_cast<const float*>(p.W) + ps, 4);
            const int rel = ps - pos0;
            int ol = p.kShift >= 0 ? (rel >> p.kShift) : rel / K;
            if (HALVES == 2 && ol >= rows) ol -= rows;
            d->y = static_cast<unsigned>(ol * (BT * 4)) | (static_cast<unsigned>(rel) << kKShift);
        };
        auto stage = [&](long long c) {
            const int buf = static_cast<int>(c - c_begin) & 1;
            const int pos0 = static_cast<int>(c * T) * K;
            uint2* dst = ent_s + buf * entBuf + entOff;
            const int e_lo = __shfl_sync(kAll, bnd, 0), cnt = __shfl_sync(kAll, bnd, ni) - e_lo;
            if constexpr (HALVES == 1) {
#pragma unroll
                for (int u = 0; u < kRegs; ++u)
                    if (pos[u] >= 0) stage_one(dst + lane + u * 32, pos[u], pos0);
                // more entries than the registers cover: the rest is fetched here
                const int* src = p.cperm + c * static_cast<long long>(T) * K + e_lo;
                if constexpr (UNEVEN) {  // thousands of them, maybe
                    for (int e0 = kRegs * 32; e0 < cnt; e0 += kRegs * 32) {
#pragma unroll
                        for (int u = 0; u < kRegs; ++u) pos[u] = e0 + lane + u * 32 < cnt ? __ldg(src + e0 + lane + u * 32) : -1;
#pragma unroll
                        for (int u = 0; u < kRegs; ++u)
                            if (pos[u] >= 0) stage_one(dst + e0 + lane + u * 32, pos[u], pos0);
                    }
                } else {
                    for (int e = lane + kRegs * 32; e < cnt; e += 32) stage_one(dst + e, __ldg(src + e), pos0);
                }
            } else {
                __pipeline_wait_prior(0);  // (each lane reads what it copied)
                for (int e = lane; e < cnt; e += 32) stage_one(dst + e, static_cast<int>(dst[e].y), pos0);
            }
            int* b = bnd_s + buf * kBounds;
            if (lane <= ni) b[lane * HALVES] = bnd - e_lo;
            const int next = __shfl_down_sync(kAll, bnd, 1);
            if constexpr (UNEVEN) {
                // does the longest run of a bundle (lanes G*j ..) have far more entries than their average?
                int most = lane < ni ? next - bnd : 0, sum = most;
#pragma unroll
                for (int off = 1; off < G; off *= 2) {
                    most = max(most, __shfl_xor_sync(kAll, most, off));
                    sum += __shfl_xor_sync(kAll, sum, off);
                }
                const bool far = p.longRun == 0 || __any_sync(kAll, most > kSideBySide || most > sum / G * 2 + p.longRun);
                if (lane == 0) b[kBounds - 1] = far;
            }
            if constexpr (HALVES == 2) {
                // where the rows of the second half start in each run
                __syncwarp();
                if (lane < ni) {
                    int lo = bnd - e_lo, hi = next - e_lo;
                    const unsigned border = static_cast<unsigned>(rows * K);
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if ((dst[mid].y >> kKShift) < border) lo = mid + 1;
                        else hi = mid;
                    }
                    b[2 * lane + 1] = lo;
                }
            }
            __pipeline_commit();
        };
        bnd = load_bounds(c_begin), bnd_next = load_bounds(c_begin + 1);
        if (c_begin < c_end) {
            load_pos(c_begin);
            stage(c_begin);
            bnd = bnd_next, bnd_next = load_bounds(c_begin + 2);
            if (HALVES == 1 && c_begin + 1 < c_end) load_pos(c_begin + 1);
        }
        const int myrow = lane / G, myent = lane % G;  // the (buffered step, group) this lane reduces
        const float4* drow = reinterpret_cast<const float4*>(dbuf + myrow * kDRow + myent * LG);  // (8-byte aligned where LG = 2)
        float* dlane = dbuf + lane;

        bool gave_up = false;
        for (long long c = c_begin; c < c_end && !gave_up; ++c) {
            const int buf = static_cast<int>(c - c_begin) & 1;
            const uint2* ent = ent_s + buf * entBuf + entOff;
            const int* bounds = bnd_s + buf * kBounds;
            __pipeline_wait_prior(0);  // this lane's staged weights are in place
            __syncwarp();
            if constexpr (kBf16) {
                // the words become fp32 bit patterns
                uint2* dst = ent_s + buf * entBuf + entOff;
                for (int e = lane; e < bounds[ni * HALVES]; e += 32) {
                    const uint2 en = dst[e];
                    dst[e].x = ((en.y >> kKShift) & 1u) ? (en.x & 0xffff0000u) : (en.x << 16);
                }
                __syncwarp();
            }
            auto stage_next = [&]() {
                if (c + 1 < c_end) {
                    stage(c + 1);
                    bnd = bnd_next, bnd_next = load_bounds(c + 3);
                }
            };
            if constexpr (HALVES == 1) {
                stage_next();
                if (c + 2 < c_end) load_pos(c + 2);
            } else if (c + 1 < c_end) {
                load_pos(c + 1);
            }
            float* gWc = p.gW ? p.gW + static_cast<size_t>(c * T) * K : nullptr;
#pragma unroll 1
            for (int half = 0; half < HALVES; ++half) {
                const int t = static_cast<int>(c - c_begin) * HALVES + half;
                if (__any_sync(kAll, !mbar_wait_or_dead(full + (t & 1), (t >> 1) & 1, dead))) {
                    gave_up = true;
                    break;
                }
                const unsigned char* gs_lane = tiles_s + (t & 1) * tileBytes + q * 16;
                const unsigned char* zero_lane = zero_s + q * 16;
                // Lane row*G + h adds the LG dots of group h's entry of buffered step `row` (fixed order) ...
                auto dots_sum = [&]() -> float {
                    if constexpr (LG == 2) {
                        const float2 q0 = *reinterpret_cast<const float2*>(drow);
                        return q0.x + q0.y;
                    } else if constexpr (LG == 4) {
                        return (drow[0].x + drow[0].y) + (drow[0].z + drow[0].w);
                    } else {
                        const float4 q0 = drow[0], q1 = drow[1];
                        return ((q0.x + q0.y) + (q0.z + q0.w)) + ((q1.x + q1.y) + (q1.z + q1.w));
                    }
                };
                // ... and stores grad_W of that entry.
                auto store_grad_w = [&](int at, float sum) {
                    if (!gWc) return;
                    float* dst = gWc + (ent[at].y >> kKShift);
                    // batch tiles after the first add to what the tile before stored: one addition per element and launch
                    if (ACC) atomicAdd(dst, sum);
                    else *dst = sum;
                };
                // The lane groups walk a run each: `n` entries from `e` on, at most `most`, at least `least`.
                auto side_by_side = [&](LaneT& acc, const LaneT& xr, int e, int n, int most, int least) {
                    // the run this lane reduces dots of
                    const int re = __shfl_sync(kAll, e, myent * LG), rn = __shfl_sync(kAll, n, myent * LG);
                    for (int s0 = 0; s0 < most; s0 += SLOTS) {
                        const uint2* en = ent + e + s0;
                        const int steps = min(SLOTS, most - s0);
                        float* d = dlane;
                        // Two steps per iteration: all loads are issued before the stores.  A group whose run has no entry left reads a
                        // row of zeros (weight 0), where that costs the pipe less than branches cost the rest: with 4 columns per lane
                        // throughout (374 against 388 us at B=32, N=768, L=670,091, K=32 with zeroed registers and a branch), with 16 in the
                        // steps that some groups do not have, one at a time (820 against 836 at B=128); with 8 the branch (501, 518).
                        auto row = [&](uint2 en_s, bool there) { return there ? gs_lane + (en_s.y & kRowMask) : zero_lane; };
                        int s = 0;
                        if constexpr (VPL == 4) {
                            for (; s < steps; s += 2) {  // (SLOTS is even: the row after an odd last step is the buffer's)
                                const uint2 en0 = en[s], en1 = en[s + 1];
                                const bool p0 = s0 + s < n, p1 = s0 + s + 1 < n;
                                LaneT g0, g1;
                                g0.load_shared(row(en0, p0));
                                g1.load_shared(row(en1, p1));
                                acc.axpy(p0 ? __uint_as_float(en0.x) : 0.f, g0);
                                d[0] = xr.dot(g0);
                                acc.axpy(p1 ? __uint_as_float(en1.x) : 0.f, g1);
                                d[kDRow] = xr.dot(g1);
                                d += 2 * kDRow;
                            }
                        } else {
                            const int both = min(SLOTS, least - s0);  // steps that every group has
                            for (; s + 2 <= both; s += 2) {
                                const uint2 en0 = en[s], en1 = en[s + 1];
                                LaneT g0, g1;
                                g0.load_shared(gs_lane + (en0.y & kRowMask));
                                g1.load_shared(gs_lane + (en1.y & kRowMask));
                                acc.axpy(__uint_as_float(en0.x), g0);
                                d[0] = xr.dot(g0);
                                acc.axpy(__uint_as_float(en1.x), g1);
                                d[kDRow] = xr.dot(g1);
                                d += 2 * kDRow;
                            }
                            for (; s < steps; ++s) {
                                const bool there = s0 + s < n;
                                LaneT g0;
                                float w = 0.f;
                                if constexpr (VPL == 16) {
                                    const uint2 en0 = en[s];
                                    g0.load_shared(row(en0, there));
                                    if (there) w = __uint_as_float(en0.x);
                                } else {
                                    g0.zero();
                                    if (there) {
                                        const uint2 en0 = en[s];
                                        w = __uint_as_float(en0.x);
                                        g0.load_shared(gs_lane + (en0.y & kRowMask));
                                    }
                                }
                                acc.axpy(w, g0);
                                d[0] = xr.dot(g0);
                                d += kDRow;
                            }
                        }
                        __syncwarp();
                        const float sum = dots_sum();
                        if (s0 + myrow < rn) store_grad_w(re + s0 + myrow, sum);
                        __syncwarp();
                    }
                };
                if (!UNEVEN || bounds[kBounds - 1] == 0) {
#pragma unroll 1
                    for (int j = 0; j < nb; ++j) {
                        const int k = j * G + grp;
                        int e = 0, n = 0;  // first entry of this group's run, its length
                        if (k < ni) e = bounds[k * HALVES + half], n = bounds[k * HALVES + half + 1] - e;
                        const int most = __reduce_max_sync(kAll, n);
                        const int least = VPL == 4 ? 0 : __reduce_min_sync(kAll, n);  // (here: behind the load of the state it costs 10 %)
                        if (most == 0) continue;
                        LaneT acc, xr;
                        tmem_load_input(taddr0 + j * COLS, acc, xr);
                        side_by_side(acc, xr, e, n, most, least);
                        tmem_store(taddr0 + j * COLS, acc);
                    }
                } else {
#pragma unroll 1
                    for (int j = 0; j < nb; ++j) {
                        const int k = j * G + grp;
                        int e = 0, n = 0;  // first entry of this group's run, its length
                        if (k < ni) e = bounds[k * HALVES + half], n = bounds[k * HALVES + half + 1] - e;
                        const int most = __reduce_max_sync(kAll, n);
                        const int least = VPL == 4 ? 0 : __reduce_min_sync(kAll, n);  // (here: behind the load of the state it costs 10 %)
                        if (most == 0) continue;
                        // what a run has more than the longest that is not much above the average is left for all groups together
                        const int mean = __reduce_add_sync(kAll, q == 0 ? n : 0) / G;
                        const int lim = min(kSideBySide, __reduce_max_sync(kAll, n <= mean + mean / 2 + p.longRun ? n : 0));
                        LaneT acc, xr;
                        tmem_load_input(taddr0 + j * COLS, acc, xr);
                        if (lim > 0) side_by_side(acc, xr, e, min(n, lim), lim, min(least, lim));
                        tmem_store(taddr0 + j * COLS, acc);
                        // ... every G-th entry each; the run's sums come from tensor memory and go back there
#pragma unroll 1
                        for (int h = 0; h < G && lim < most; ++h) {
                            constexpr int AT = VPL <= 8 && SLOTS >= 4 ? 4 : 2;
                            constexpr bool kRowsAhead = VPL == 4;
                            const int first = __shfl_sync(kAll, e, h * LG) + lim, cnt = __shfl_sync(kAll, n, h * LG) - lim;
                            if (cnt <= 0) continue;
                            tc::wait_store();
                            LaneT sums, xh;
                            tmem_load_input(taddr0 + j * COLS, sums, xh);
                            xh.from_lane(h * LG + q);
                            if (grp != h) sums.zero();
                            // AT steps at a time.  A hot run is one warp's chain, so the next steps' entries, and where registers allow
                            // their rows, are asked for before these are worked on; a group without an entry has a row of zeros.
                            float w_n[AT];
                            int row_n[AT];
                            LaneT g_n[AT];
                            auto fetch_entries = [&](int s) {
#pragma unroll
                                for (int u = 0; u < AT; ++u) {
                                    const int at = (s + u) * G + grp;
                                    const uint2 en = at < cnt ? ent[first + at] : make_uint2(0u, 0u);
                                    w_n[u] = __uint_as_float(en.x);
                                    row_n[u] = at < cnt ? static_cast<int>(en.y & kRowMask) : static_cast<int>(zero_lane - gs_lane);
                                }
                            };
                            auto fetch_rows = [&]() {
#pragma unroll
                                for (int u = 0; u < AT; ++u) g_n[u].load_shared(gs_lane + row_n[u]);
                            };
                            fetch_entries(0);
                            if constexpr (kRowsAhead) fetch_rows();
                            float* d = dlane;
                            const int total = (cnt + G - 1) / G;
#pragma unroll 1
                            for (int s = 0; s < total; s += AT) {
                                if constexpr (!kRowsAhead) fetch_rows();
                                float w[AT];
                                LaneT g_s[AT];
#pragma unroll
                                for (int u = 0; u < AT; ++u) w[u] = w_n[u], g_s[u] = g_n[u];
                                fetch_entries(s + AT);
                                if constexpr (kRowsAhead) fetch_rows();
#pragma unroll
                                for (int u = 0; u < AT; ++u) {
                                    sums.axpy(w[u], g_s[u]);
                                    d[u * kDRow] = xh.dot(g_s[u]);
                                }
                                d += AT * kDRow;
                                if ((s + AT) % SLOTS == 0 || s + AT >= total) {
                                    const int e0 = s / SLOTS * 32 + lane;
                                    __syncwarp();
                                    const float sum = dots_sum();
                                    if (e0 < cnt) store_grad_w(first + e0, sum);
                                    __syncwarp();
                                    d = dlane;
                                }
                            }
                            sums.add_groups();
                            LaneT own;
                            tmem_load_input(taddr0 + j * COLS, own, xh);
                            if (grp == h) own = sums;
                            tmem_store(taddr0 + j * COLS, own);
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(empty + (t & 1));
                if (HALVES == 2 && half == 0) stage_next();
                tc::wait_store();
            }

            // Every segChunks chunks the running grad_x sums go out as one partial and restart from zero.
            const long long done = c - c_begin + 1;
            if (done % p.segChunks == 0 || c + 1 == c_end) {
                const int seg = static_cast<int>((done - 1) / p.segChunks);
                for (int j = 0; j < nb; ++j) {
                    const int k = j * G + grp, i = iw + k;
                    LaneT a, x;
                    tmem_load_input(taddr0 + j * COLS, a, x);
                    if (k < ni && i < N) {
                        // One partial per range: the first segment stores, the later ones add to what this lane stored before
                        // (a handful of fp32 additions of segment sums; the long sums stay inside the segments, and the
                        // ranges are added in fp64 afterwards).
                        float* dst = p.partial + (static_cast<size_t>(r) * N + input_at(i)) * p.Bpad + 4 * q;
#pragma unroll
                        for (int m = 0; m < VPL / 4; ++m) {
                            float4 out;
                            unpack2(a.v[2 * m], out.x, out.y), unpack2(a.v[2 * m + 1], out.z, out.w);
                            float4* at = reinterpret_cast<float4*>(dst + m * (4 * LG));
                            if (seg > 0) {
                                const float4 b = *at;
                                out.x += b.x, out.y += b.y, out.z += b.z, out.w += b.w;
                            }
                            *at = out;
                        }
                    }
                    a.zero();
                    tmem_store(taddr0 + j * COLS, a);
                }
                tc::wait_store();
            }
        }
        __pipeline_wait_prior(0);

        // A range without chunks still owns a partial: zeros.
        if (c_begin >= c_end) {
            for (int j = 0; j < nb; ++j) {
                const int k = j * G + grp, i = iw + k;
                if (k < ni && i < N)
#pragma unroll
                    for (int m = 0; m < VPL / 4; ++m)
                        *reinterpret_cast<float4*>(p.partial + (static_cast<size_t>(r) * N + i) * p.Bpad + 4 * q + m * (4 * LG)) =
                            make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    }
    chain_release();
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::dealloc(*tmem_base_p);
}

struct FusedConfig {
    int ni, iparts, Bpad, R, segChunks;
    int groups;  // lane groups per warp
    int halves;  // tiles per chunk
    size_t smem;
};

// For one tile of at most 128 batch columns.  `table`: whether the plan's table has to fit, too (the scratch is that of a table that does).
bool fused_config(const ffi_plan* plan, int64_t B, const DeviceInfo& dev, FusedConfig* c, bool table = true) {
    if (!plan || !plan->has_chunks || B > 128) return false;
    // the entry code holds the position within the chunk in 14 bits
    if (static_cast<long long>(plan->chunk_rows) * plan->K > (1 << (32 - kKShift))) return false;
    c->groups = B > 16 ? 4 : (B > 8 ? 8 : 16);
    c->halves = B > 64 ? 2 : 1;
    c->Bpad = B > 64 ? 128 : (B > 32 ? 64 : (B > 16 ? 32 : (B > 8 ? 16 : 8)));
    c->ni = plan->fused_ni;
    c->iparts = static_cast<int>(ceil_div(plan->N, kWarps * c->ni));
    int R = dev.sm_count / c->iparts;
    if (R < 1) R = 1;
    if (R > plan->range_chunks) R = static_cast<int>(plan->range_chunks);
    c->R = R;
    // flush after about 128 summands per (input, batch) pair, and at least once on the way
    const double per_chunk = static_cast<double>(plan->chunk_rows) * plan->K / static_cast<double>(plan->N);
    int seg = static_cast<int>(128.0 / (per_chunk > 1.0 ? per_chunk : 1.0));
    const int halfway = static_cast<int>(ceil_div(plan->n_chunks, R) / 2);
    if (seg > halfway) seg = halfway;
    if (seg < 1) seg = 1;
    c->segChunks = seg;
    const size_t T = static_cast<size_t>(plan->chunk_rows);
    if (T * c->Bpad * 4 > (size_t{1} << kKShift)) return false;
    const size_t total = fused_smem_bytes(static_cast<int64_t>(T) * (c->halves == 2 ? 1 : 2) * c->Bpad * 4, plan->fused_entries[kFusedWarps], c->groups);
    if (table && total > static_cast<size_t>(dev.max_smem_optin)) return false;  // a very uneven table: separate kernels
    c->smem = total;
    return true;
}

// Whether a tile of `cols` columns has the ranges and row width of configuration c.
bool fused_same_layout(const ffi_plan* plan, int64_t cols, const DeviceInfo& dev, const FusedConfig& c) {
    FusedConfig o;
    return fused_config(plan, cols, dev, &o) && o.R == c.R && o.Bpad == c.Bpad;
}

// Columns of the batch tile that starts at b0.
int64_t tile_columns(int64_t B, int64_t b0) { return B - b0 < 128 ? B - b0 : 128; }

// cuTensorMapEncodeTiled through the runtime's driver entry point (the library does not link libcuda).
int encode_g_map(CUtensorMap* map, const float* gT, int64_t L, int64_t ldg, int64_t cols, int chunk_rows, int BT) {
    using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static EncodeFn encode = nullptr;
    if (!encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        FFI_CUDA_CHECK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q));
        if (q != cudaDriverEntryPointSuccess || !fn) return fail(FFI_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
        encode = reinterpret_cast<EncodeFn>(fn);
    }
    if (reinterpret_cast<uintptr_t>(gT) % 16 != 0 || chunk_rows > 256 || (BT != 8 && BT != 16 && BT != 32 && BT != 64 && BT != 128))
        return fail(FFI_ERR_INVALID_ARGUMENT, "transposed gradient must be 16-byte aligned, chunks at most 256 rows");
    // the stored rows may be narrower than the tile (batch <= 32 keeps 32 columns): the box's columns past them
    // are filled with zeros, like its rows past L
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols < BT ? cols : BT), static_cast<cuuint64_t>(L)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ldg) * 4};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(BT), static_cast<cuuint32_t>(chunk_rows)};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(gT), dims, strides, box, elem,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(FFI_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", static_cast<int>(r));
    return FFI_OK;
}

}  // namespace

// Whether the lane groups share the runs of any table because a warp has too few inputs for them.  It pays where the runs are long: graph
// of backwards, side by side against shared, us, by entries in a chunk's average run: one input per warp 8 7.4, 8.3; 20 8.7, 8.3; 32 9.4,
// 8.4; 208 42, 14; two 18 8.1, 8.6; 40 10.5, 9.2; 104 29, 18 (all 8 columns); three, up to 16 columns 27 9.4, 9.5; 69 24, 19; more columns
// of three inputs lose throughout (32 columns 27 9.8, 10.8; 69 24, 26).
static bool shares_runs(const ffi_plan* plan, const FusedConfig& c, int64_t columns) {
    const double run = static_cast<double>(plan->chunk_rows) * plan->K / static_cast<double>(plan->N);
    return c.ni == 1 ? run >= 20.0 : c.ni == 2 ? run >= 32.0 : c.ni == 3 && columns <= 16 && run >= 32.0;
}

// An input belongs to one warp of a range, so what bounds a table with a very hot input is that warp's chain, kChain ns an entry: the
// more slices, the fewer ranges the input's entries are spread over.  The kernels for grad_x and grad_W alone take, with such tables,
// about kTwo ns for every link, and 30 us for the second launch, its partials and short tables in general.  One pass against two, us, with a
// share of 0.2 and 0.8 of the links on ONE input: N=2,048, L=150,000, K=32 B=64 869, 2,956 against 610, 1,295; 128 1,293, 3,990 against
// 1,187, 3,401; 32 709, 2,437 against 570, 825; 8 (0.4 and 0.8) 744, 1,399 against 620, 823; N=768, L=200,000 B=64 494, 1,489 against 519,
// 943; 32 (0.4 and 0.8) 683, 1,236 against 527, 646; N=300, L=100,000 B=64 192, 490 against 192, 325.  With one slice the one-pass kernel is
// the faster one throughout (N=128 at 0.8: 0.3 to 0.94 of the two).
static bool fused_pays(const ffi_plan* plan, const FusedConfig& c, int64_t columns) {
    const double kChain = columns > 64 ? 20.0 : columns > 32 ? 14.5 : columns > 16 ? 11.5 : columns > 8 ? 7.9 : 6.7;
    const double kTwo = columns > 64 ? 0.176 : columns > 32 ? 0.065 : columns > 16 ? 0.08 : columns > 8 ? 0.091 : 0.1;
    const double links = static_cast<double>(plan->L) * plan->K;
    return c.iparts == 1 || plan->longest_input * kChain / c.R <= links * kTwo + 30e3;
}

bool backward_fused_applicable(const ffi_plan* plan, int64_t B) {
    DeviceInfo dev;
    if (get_device_info(&dev) != FFI_OK) return false;
    FusedConfig c;
    const int64_t first = tile_columns(B, 0), last = B - (B - 1) / 128 * 128;
    return fused_config(plan, first, dev, &c) && fused_config(plan, last, dev, &c) && fused_pays(plan, c, first);
}

size_t backward_fused_workspace_bytes(const ffi_plan* plan, int64_t B) {
    DeviceInfo dev;
    if (get_device_info(&dev) != FFI_OK) return 0;
    size_t total = 0;  // the partials of every batch tile, summed by one launch at the end
    for (int64_t b0 = 0; b0 < B; b0 += 128) {
        FusedConfig c;
        if (!fused_config(plan, tile_columns(B, b0), dev, &c, false)) return 0;
        total += static_cast<size_t>(c.R) * plan->N * c.Bpad * 4;
    }
    return total;
}

int reduce_range_partials(const float* partial, float* gx, int R, int N, int cols, int Bpad, int tiles, int B,
                          int x_transposed, cudaStream_t stream);

// grad_x (always), grad_W (when gW != nullptr) and grad_bias (when gbias != nullptr, from gT).  xT is x as [N][ldx].
int launch_backward_fused(const GradXArgs& a, const void* xT, int64_t ldx, float* gW, float* gbias,
                          cudaStream_t stream) {
    DeviceInfo dev;
    int rc = get_device_info(&dev);
    if (rc != FFI_OK) return rc;
    const size_t need = backward_fused_workspace_bytes(a.plan, a.B);
    if (!a.workspace || a.workspace_bytes < need || reinterpret_cast<uintptr_t>(a.workspace) % 16 != 0)
        return fail(FFI_ERR_WORKSPACE, "fused backward needs %zu bytes of 16-byte aligned workspace", need);
    // the tile copy fills the columns past a narrower stored row with zeros
    if (!a.gT || a.ldg < round_up(a.B, 32) || a.ldg % 32 != 0 || !xT)
        return fail(FFI_ERR_INVALID_ARGUMENT, "fused backward needs gT and xT");
    BwdFusedParams p;
    p.W = a.W;
    p.ldg = a.ldg;
    p.ldx = ldx;
    p.cperm = a.plan->cperm;
    p.cptr = a.plan->cptr;
    p.order = a.plan->order;
    p.partial = static_cast<float*>(a.workspace);
    p.gW = gW;
    p.gbias = gbias;
    p.N = a.N;
    p.L = a.L;
    p.K = a.K;
    p.kShift = -1;
    for (int sh = 0; sh < 31; ++sh)
        if ((1 << sh) == a.K) p.kShift = sh;
    p.T = a.plan->chunk_rows;
    p.nChunks = a.plan->n_chunks;
    for (int w = 0; w <= kWarps; ++w) p.entOff[w] = a.plan->fused_entries[w];
    p.lastHalf = a.w_bf16 && (a.plan->L * a.plan->K) % 2 != 0 ? static_cast<int>(a.plan->L * a.plan->K - 1) : -1;
    if (a.w_bf16 && reinterpret_cast<uintptr_t>(a.W) % 4 != 0)
        return fail(FFI_ERR_INVALID_ARGUMENT, "fused backward copies bf16 weights word by word: W must be 4-byte aligned");
    const float* partials = p.partial;  // of the tiles not summed yet
    int tiles = 1;
    for (int64_t b0 = 0; b0 < a.B; b0 += 128) {
        const int cols = static_cast<int>(tile_columns(a.B, b0));
        FusedConfig c;
        if (!fused_config(a.plan, cols, dev, &c)) return fail(FFI_ERR_UNSUPPORTED, "fused backward does not cover this shape");
        p.gT = a.gT + b0;
        p.xT = static_cast<const unsigned char*>(xT) + b0 * (a.w_bf16 ? 2 : 4);
        p.B = cols;
        p.xVec = ldx % 2 == 0 && reinterpret_cast<uintptr_t>(p.xT) % 8 == 0;
        p.R = c.R;
        p.Bpad = c.Bpad;
        p.segChunks = c.segChunks;
        p.ni = c.ni;
        p.longRun = shares_runs(a.plan, c, cols) ? 0 : kLongRun;
        // gT as a 2-D tensor [L rows][BT columns] with row pitch ldg; one or two boxes = a g tile
        CUtensorMap g_map;
        const int rows = p.T / c.halves;  // (T is a multiple of 8)
        p.boxes = rows > 256 ? 2 : 1;
        rc = encode_g_map(&g_map, p.gT, a.L, a.ldg, a.ldg - b0, rows / p.boxes, c.Bpad);
        if (rc != FFI_OK) return rc;
        dim3 grid(static_cast<unsigned>(c.R), static_cast<unsigned>(c.iparts), 1);
        auto launch_kernel = [&](auto kern) -> int {
            FFI_CUDA_CHECK(prepare_kernel(reinterpret_cast<const void*>(kern), 0, c.smem, nullptr));
            FFI_CUDA_CHECK(launch_chained(kern, grid, dim3(kThreads), c.smem, stream, p, g_map));
            return FFI_OK;
        };
        auto launch_typed = [&](auto tx, auto acc, auto uneven) -> int {
            using TX = decltype(tx);
            constexpr bool ACC = decltype(acc)::value, UNEVEN = decltype(uneven)::value;
            if (c.Bpad == 128) return launch_kernel(ffi_bwd_runs_kernel<4, 16, 2, TX, ACC, UNEVEN>);
            if (c.Bpad == 64) return launch_kernel(ffi_bwd_runs_kernel<4, 8, 1, TX, ACC, UNEVEN>);
            if (c.Bpad == 32) return launch_kernel(ffi_bwd_runs_kernel<4, 4, 1, TX, ACC, UNEVEN>);
            if (c.Bpad == 16) return launch_kernel(ffi_bwd_runs_kernel<8, 4, 1, TX, ACC, UNEVEN>);
            return launch_kernel(ffi_bwd_runs_kernel<16, 4, 1, TX, ACC, UNEVEN>);
        };
        auto launch_table = [&](auto tx, auto acc) {
            return p.order || p.longRun == 0 ? launch_typed(tx, acc, std::true_type{}) : launch_typed(tx, acc, std::false_type{});
        };
        auto launch_tile = [&](auto acc) { return a.w_bf16 ? launch_table(__nv_bfloat16{}, acc) : launch_table(float{}, acc); };
        rc = b0 > 0 ? launch_tile(std::true_type{}) : launch_tile(std::false_type{});
        if (rc != FFI_OK) return rc;
        FFI_LAUNCH_CHECK("ffi_bwd_runs_kernel");
        // tiles of the same layout (all of 65..128 columns) are summed together, a narrower last one by itself
        const bool last = b0 + 128 >= a.B;
        if (!last && fused_same_layout(a.plan, tile_columns(a.B, b0 + 128), dev, c)) {
            ++tiles;
        } else {
            const int64_t first = b0 - 128 * (tiles - 1);
            rc = reduce_range_partials(partials, a.gx + (a.x_transposed ? first : first * a.N), c.R, a.N,
                                       static_cast<int>(b0 + cols - first), c.Bpad, tiles, a.B, a.x_transposed, stream);
            if (rc != FFI_OK) return rc;
            partials = p.partial + static_cast<size_t>(c.R) * a.N * c.Bpad;
            tiles = 1;
        }
        p.partial += static_cast<size_t>(c.R) * a.N * c.Bpad;
    }
    return FFI_OK;
}

}  // namespace ffi

// Test hook: how long (clock64 ticks of the current device, about 0.5 ns each) the bounded device-side waits
// may last before they give up.  The default is about two seconds; a test of the give-up path lowers it.
extern "C" int ffi_set_wait_limit_ticks(int64_t ticks) {
    if (ticks < 1000) return ffi::fail(FFI_ERR_INVALID_ARGUMENT, "the wait limit must be at least 1000 ticks");
    const long long t = ticks;
    FFI_CUDA_CHECK(cudaMemcpyToSymbol(ffi::g_wait_limit, &t, sizeof(t)));
    const int rc = ffi::set_dense_forward_wait_limit(t);
    return rc != FFI_OK ? rc : ffi::set_peer_wait_limit(t);
}

// Number of bounded device-side waits that gave up since the library was loaded (0 in a healthy
// run; any other value means the results of the affected call are void).  Synchronises the device.
extern "C" int ffi_wait_timeouts(int* out) {
    if (!out) return ffi::fail(FFI_ERR_INVALID_ARGUMENT, "NULL output passed to ffi_wait_timeouts");
    FFI_CUDA_CHECK(cudaMemcpyFromSymbol(out, ffi::g_wait_timeouts, sizeof(int)));
    int peers = 0;
    const int rc = ffi::peer_wait_timeouts(&peers);
    if (rc != FFI_OK) return rc;
    *out += peers;
    int dense = 0;
    const int rd = ffi::dense_forward_timeouts(&dense);
    if (rd != FFI_OK) return rd;
    *out += dense;
    return FFI_OK;
}
