// Transposed (CSR-by-input) index of an FFI index table, built on the device.
//
// The reference has no such structure: its grad_x scatters with atomicAdd
// (tfsparse/cc/kernels/backward.cu.h:119-182).  Definition (bit-exact contract):
// flat position p = o*K + k; `perm` lists all positions ordered by key idx[p]
// ascending, ties by p ascending; rowptr[i] = number of positions with key < i.
//
// Build: a stable least-significant-digit radix sort of (key, position) pairs, 8 bits
// per pass, one warp per 1024-element tile (per-tile digit histogram, global exclusive
// scan, stable in-tile ranking with warp match).  From the canonical form a chunked
// form is derived for the narrow-input grad_x kernel: the outputs are cut into chunks
// of T rows, and chunk c stores its T*K positions ordered by (key, position) in
// cperm[c*T*K ...], with cptr[c][i] the offset of input i's run inside the chunk.
// Concatenating, for each input i, its runs over the chunks in chunk order gives back
// exactly row i of the canonical form (chunks are ascending ranges of p).  A chunk of an uneven table holds the runs in another
// order of the inputs (`order`).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>

#include "ffi_common.cuh"

namespace ffi {
namespace {

constexpr int kTile = 1024;      // elements per warp tile
constexpr int kSortWarps = 4;    // warps per block in the sort kernels

__global__ void validate_idx_kernel(const int* __restrict__ idx, long long n, int N, int* bad) {
    long long e = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    bool any = false;
    for (; e < n; e += stride) {
        unsigned v = static_cast<unsigned>(idx[e]);
        any |= v >= static_cast<unsigned>(N);
    }
    if (any) *bad = 1;
}

// counts[d * nTiles + tile] = number of elements of `tile` whose digit is d.
__global__ void radix_hist_kernel(const int* __restrict__ keys, long long n, int shift,
                                  int* __restrict__ counts, long long nTiles) {
    __shared__ int h[kSortWarps][256];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long tile = static_cast<long long>(blockIdx.x) * kSortWarps + warp;
    for (int d = lane; d < 256; d += 32) h[warp][d] = 0;
    __syncwarp();
    if (tile < nTiles) {
        const long long base = tile * kTile;
        for (int r = 0; r < kTile / 32; ++r) {
            long long e = base + r * 32 + lane;
            if (e < n) atomicAdd(&h[warp][(keys[e] >> shift) & 255], 1);
        }
        __syncwarp();
        for (int d = lane; d < 256; d += 32) counts[static_cast<long long>(d) * nTiles + tile] = h[warp][d];
    }
}

// In-place exclusive scan of `data[0..n)`: int64 running totals, int32 output (totals are bounded by
// L*K < 2^31).  Three phases: every block adds up its segment of kScanSeg consecutive elements, one block
// scans the segment totals, every block rescans its segment from its offset.
constexpr int kScanThreads = 256;
constexpr int kScanPer = 16;                          // consecutive elements per thread
constexpr int kScanSeg = kScanThreads * kScanPer;     // elements per block

__device__ __forceinline__ long long block_exclusive_scan(long long v, long long* sh, long long* total) {
    // exclusive scan of one value per thread over the block (kScanThreads threads); *total = block sum
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long incl = v;
#pragma unroll
    for (int off = 1; off < 32; off *= 2) {
        const long long up = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += up;
    }
    if (lane == 31) sh[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        long long w = lane < kScanThreads / 32 ? sh[lane] : 0;
        long long wi = w;
#pragma unroll
        for (int off = 1; off < 32; off *= 2) {
            const long long up = __shfl_up_sync(0xffffffffu, wi, off);
            if (lane >= off) wi += up;
        }
        if (lane < kScanThreads / 32) sh[lane] = wi - w;
        if (lane == kScanThreads / 32 - 1) sh[kScanThreads / 32] = wi;
    }
    __syncthreads();
    *total = sh[kScanThreads / 32];
    const long long res = sh[warp] + incl - v;
    __syncthreads();
    return res;
}

__global__ void __launch_bounds__(kScanThreads) scan_segment_sums_kernel(const int* __restrict__ data, long long n,
                                                                        long long* __restrict__ seg_sums) {
    __shared__ long long sh[kScanThreads / 32 + 1];
    const long long base = static_cast<long long>(blockIdx.x) * kScanSeg + static_cast<long long>(threadIdx.x) * kScanPer;
    long long s = 0;
#pragma unroll
    for (int u = 0; u < kScanPer; ++u)
        if (base + u < n) s += data[base + u];
    long long total;
    block_exclusive_scan(s, sh, &total);
    if (threadIdx.x == 0) seg_sums[blockIdx.x] = total;
}

// exclusive scan of the segment totals by one block (a few thousand values)
__global__ void __launch_bounds__(kScanThreads) scan_totals_kernel(long long* __restrict__ seg_sums, long long nseg) {
    __shared__ long long sh[kScanThreads / 32 + 1];
    long long carry = 0;
    for (long long b0 = 0; b0 < nseg; b0 += kScanThreads) {
        const long long i = b0 + threadIdx.x;
        const long long v = i < nseg ? seg_sums[i] : 0;
        long long total;
        const long long ex = block_exclusive_scan(v, sh, &total);
        if (i < nseg) seg_sums[i] = carry + ex;
        carry += total;
    }
}

__global__ void __launch_bounds__(kScanThreads) scan_apply_kernel(int* __restrict__ data, long long n,
                                                                 const long long* __restrict__ seg_offsets) {
    __shared__ long long sh[kScanThreads / 32 + 1];
    const long long base = static_cast<long long>(blockIdx.x) * kScanSeg + static_cast<long long>(threadIdx.x) * kScanPer;
    int v[kScanPer];
    long long s = 0;
#pragma unroll
    for (int u = 0; u < kScanPer; ++u) {
        v[u] = base + u < n ? data[base + u] : 0;
        s += v[u];
    }
    long long total;
    long long run = seg_offsets[blockIdx.x] + block_exclusive_scan(s, sh, &total);
#pragma unroll
    for (int u = 0; u < kScanPer; ++u) {
        if (base + u < n) data[base + u] = static_cast<int>(run);
        run += v[u];
    }
}

// The same scan by one block, for short arrays (the self-check export's N + 1 row totals).
__global__ void small_exclusive_scan_kernel(int* __restrict__ data, long long n) {
    __shared__ long long sums[1024];
    const int t = threadIdx.x;
    const long long chunk = (n + blockDim.x - 1) / blockDim.x;
    const long long lo = min(n, t * chunk), hi = min(n, lo + chunk);
    long long s = 0;
    for (long long e = lo; e < hi; ++e) s += data[e];
    sums[t] = s;
    __syncthreads();
    if (t == 0) {
        long long run = 0;
        for (int j = 0; j < blockDim.x; ++j) {
            long long v = sums[j];
            sums[j] = run;
            run += v;
        }
    }
    __syncthreads();
    long long run = sums[t];
    for (long long e = lo; e < hi; ++e) {
        int v = data[e];
        data[e] = static_cast<int>(run);
        run += v;
    }
}

// `seg_scratch` holds ceil(n / kScanSeg) int64 values.
int launch_exclusive_scan(int* data, long long n, long long* seg_scratch, cudaStream_t stream) {
    const long long nseg = ceil_div(n, kScanSeg);
    scan_segment_sums_kernel<<<static_cast<unsigned>(nseg), kScanThreads, 0, stream>>>(data, n, seg_scratch);
    scan_totals_kernel<<<1, kScanThreads, 0, stream>>>(seg_scratch, nseg);
    scan_apply_kernel<<<static_cast<unsigned>(nseg), kScanThreads, 0, stream>>>(data, n, seg_scratch);
    FFI_LAUNCH_CHECK("exclusive scan");
    return FFI_OK;
}

// Stable scatter of one digit pass. vals_in == nullptr means "value = element index".
__global__ void radix_scatter_kernel(const int* __restrict__ keys_in, const int* __restrict__ vals_in,
                                     int* __restrict__ keys_out, int* __restrict__ vals_out,
                                     long long n, int shift, const int* __restrict__ offsets,
                                     long long nTiles) {
    __shared__ int base[kSortWarps][256];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long tile = static_cast<long long>(blockIdx.x) * kSortWarps + warp;
    if (tile >= nTiles) return;
    for (int d = lane; d < 256; d += 32) base[warp][d] = offsets[static_cast<long long>(d) * nTiles + tile];
    __syncwarp();
    const long long first = tile * kTile;
    const unsigned lt = (1u << lane) - 1u;
    for (int r = 0; r < kTile / 32; ++r) {
        const long long e = first + r * 32 + lane;
        const bool valid = e < n;
        const unsigned active = __ballot_sync(0xffffffffu, valid);
        if (valid) {
            const int key = keys_in[e];
            const int val = vals_in ? vals_in[e] : static_cast<int>(e);
            const int d = (key >> shift) & 255;
            const unsigned same = __match_any_sync(active, d);
            const int rank = __popc(same & lt);
            const int dst = base[warp][d] + rank;
            __syncwarp(active);
            if (rank == 0) base[warp][d] += __popc(same);
            keys_out[dst] = key;
            vals_out[dst] = val;
        }
        __syncwarp();
    }
}

// rowptr[i] = lower_bound(sorted_keys, i), i in [0, N].
__global__ void rowptr_kernel(const int* __restrict__ sorted_keys, long long n, int N,
                              int* __restrict__ rowptr) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > N) return;
    long long lo = 0, hi = n;
    while (lo < hi) {
        long long mid = (lo + hi) >> 1;
        if (sorted_keys[mid] < i) lo = mid + 1;
        else hi = mid;
    }
    rowptr[i] = static_cast<int>(lo);
}

// lb[c][s] = first position e in row i of the canonical form with perm[e] >= c*T*K, where i is the input at place s (order[s], or s).
__global__ void chunk_bounds_kernel(const int* __restrict__ rowptr, const int* __restrict__ perm, const int* __restrict__ order,
                                    int N, long long chunkEntries, long long nChunks,
                                    int* __restrict__ lb) {
    const long long id = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (id >= (nChunks + 1) * N) return;
    const long long c = id / N;
    const int place = static_cast<int>(id - c * N);
    const int i = order ? order[place] : place;
    const long long target = c * chunkEntries;
    int lo = rowptr[i], hi = rowptr[i + 1];
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (perm[mid] < target) lo = mid + 1;
        else hi = mid;
    }
    lb[id] = lo;
}

// One block per chunk: cptr[c][0..N] = exclusive scan over i of the run lengths, and the
// runs themselves are copied into cperm.
__global__ void chunk_fill_kernel(const int* __restrict__ perm, const int* __restrict__ lb, int N,
                                  long long chunkEntries, int* __restrict__ cptr,
                                  int* __restrict__ cperm) {
    extern __shared__ int run_off[];  // N + 1
    const long long c = blockIdx.x;
    const int* lb0 = lb + c * N;
    const int* lb1 = lb + (c + 1) * N;
    if (threadIdx.x == 0) {
        int run = 0;
        for (int i = 0; i < N; ++i) {
            run_off[i] = run;
            run += lb1[i] - lb0[i];
        }
        run_off[N] = run;
    }
    __syncthreads();
    for (int i = threadIdx.x; i <= N; i += blockDim.x) cptr[c * (N + 1) + i] = run_off[i];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    int* dst = cperm + c * chunkEntries;
    for (int i = warp; i < N; i += nwarps) {
        const int s = lb0[i], len = lb1[i] - s, off = run_off[i];
        for (int r = lane; r < len; r += 32) dst[off + r] = perm[s + r];
    }
}

// most[w] = largest number of entries that warp w of a slice has in any chunk and slice, most[kFusedWarps] = largest number that an
// input has in any chunk (zeroed by the caller); a slice is kFusedWarps warps of ni inputs.  One block per warp of all slices.
__global__ void warp_stats_kernel(const int* __restrict__ cptr, int N, long long nChunks, int ni, int* __restrict__ most) {
    const int lo = min(N, static_cast<int>(blockIdx.x) * ni), hi = min(N, lo + ni);
    int best = 0, longest = 0;
    for (long long c = threadIdx.x; c < nChunks; c += blockDim.x) {
        const int* at = cptr + c * (N + 1);
        int before = at[lo];
        best = max(best, at[hi] - before);
        for (int i = lo + 1; i <= hi; ++i) {
            const int here = at[i];
            longest = max(longest, here - before);
            before = here;
        }
    }
    best = __reduce_max_sync(0xffffffffu, best);
    longest = __reduce_max_sync(0xffffffffu, longest);
    if (threadIdx.x % 32 == 0) {
        atomicMax(most + blockIdx.x % kFusedWarps, best);
        atomicMax(most + kFusedWarps, longest);
    }
}

// longest[0] = largest number of entries an input has (zeroed by the caller).
__global__ void longest_row_kernel(const int* __restrict__ rowptr, int N, int* __restrict__ longest) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int most = __reduce_max_sync(0xffffffffu, i < N ? rowptr[i + 1] - rowptr[i] : 0);
    if (threadIdx.x % 32 == 0) atomicMax(longest, most);
}

// Self-check export: rebuild the canonical form from (cptr, cperm).
__global__ void chunked_row_totals_kernel(const int* __restrict__ cptr, const int* __restrict__ order, int N, long long nChunks,
                                          int* __restrict__ totals) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > N) return;
    if (i == N) {
        totals[N] = 0;
        return;
    }
    long long s = 0;
    for (long long c = 0; c < nChunks; ++c) s += cptr[c * (N + 1) + i + 1] - cptr[c * (N + 1) + i];
    totals[order ? order[i] : i] = static_cast<int>(s);
}

__global__ void chunked_gather_kernel(const int* __restrict__ cptr, const int* __restrict__ cperm,
                                      const int* __restrict__ order, const int* __restrict__ rowptr, int N, long long nChunks,
                                      long long chunkEntries, int* __restrict__ perm_out) {
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (i >= N) return;
    long long run = rowptr[order ? order[i] : i];
    for (long long c = 0; c < nChunks; ++c) {
        const int s = cptr[c * (N + 1) + i], len = cptr[c * (N + 1) + i + 1] - s;
        const int* src = cperm + c * chunkEntries + s;
        for (int r = lane; r < len; r += 32) perm_out[run + r] = src[r];
        run += len;
    }
}

int significant_bits(int64_t n) {
    int bits = 0;
    while ((static_cast<int64_t>(1) << bits) < n) ++bits;
    return bits < 1 ? 1 : bits;
}

struct DeviceBuffer {
    void* ptr = nullptr;
    ~DeviceBuffer() {
        if (ptr) cudaFree(ptr);
    }
    cudaError_t alloc(size_t bytes) { return cudaMalloc(&ptr, bytes ? bytes : 4); }
    template <class T>
    T* as() {
        return static_cast<T*>(ptr);
    }
};

}  // namespace

// Rows per chunk of the chunked lists and inputs per warp of the one-pass backward, which keeps, per chunk, g tiles of T x 128 floats
// in all and twice the (weight, code) pairs of a slice of the inputs in shared memory; a chunk's positions fit 14 bits.
//   * T is the largest multiple of 8 for which that fits: long runs per input and chunk are cheap runs, and what they gain
//     is more than the L1 that is left loses in the gathers of W (backward at N=768, L=670,091, K=32, us, by T: 272, 248, 224, 200,
//     176; B=128 828, 833, 839, 874, 909; B=32 368, 373, 386, 402, 424).
//   * it is lowered until the chunks fill the SMs: the kernel runs R = SMs / slices ranges of chunks, so the chunks are cut
//     to a whole number per range; a short L (down to 16 rows per chunk) is cut to one chunk per range, or two where they
//     keep 64 rows.
//   * where even so there are fewer chunks than ranges, the warps take fewer inputs each, so that more slices fill the SMs
//     (backward of 513 rows, B=127, N=254, K=73: 23 -> 16 us).
// That is for tables whose inputs have about equally many entries.  For others see plan_build: their inputs are dealt to the warps
// by count, and T is lowered, to half at the least, until the entries of the largest warps fit.
struct PlanShape {
    int rows, ni;
};
int64_t device_sms() {
    DeviceInfo dev;
    return get_device_info(&dev) == FFI_OK ? dev.sm_count : 148;
}
int64_t device_smem() {
    DeviceInfo dev;
    return get_device_info(&dev) == FFI_OK && dev.max_smem_optin > 0 ? dev.max_smem_optin : 232448;
}
// Whether chunks of T rows fit whose warps' largest numbers of entries add up to `entries`.
bool chunks_fit(int64_t T, int64_t entries) { return fused_smem_bytes(T * 512, entries, 4) <= static_cast<size_t>(device_smem()); }

PlanShape plan_shape(int64_t L, int64_t K, int64_t N) {
    const int64_t sms = device_sms();
    int ni = fused_inputs_per_warp(N);
    const int64_t warps = std::min<int64_t>(kFusedWarps, ceil_div(N, ni));  // that have inputs
    int64_t T = 512;
    for (; T > 8; T -= 8) {
        // a random table's warp with the most entries
        const double entries = static_cast<double>(T) * K * ni / static_cast<double>(N), most = entries + 5.0 * std::sqrt(entries) + 4.0;
        if (T * K <= 16384 && chunks_fit(T, static_cast<int64_t>(warps * most))) break;
    }
    if (T * K > 16384) return {0, ni};  // K in the thousands: no chunked lists
    const int64_t parts = ceil_div(N, kFusedWarps * ni), R = sms / parts > 0 ? sms / parts : 1;
    const int64_t n = ceil_div(L, T);
    const int64_t want = n > R ? round_up(n, R) : (L >= 2 * R * 64 ? 2 * R : R);
    const int64_t even = round_up(ceil_div(L, want), 8);
    if (even < T) T = even < 16 ? (T < 16 ? T : 16) : even;
    const int64_t chunks = ceil_div(L, T);
    while (ni > 4 && chunks * ceil_div(N, kFusedWarps * (ni - 4)) <= sms) ni -= 4;
    return {static_cast<int>(T), ni};
}

// For an uneven table whose chunks of T rows have warps with `entries` entries (see chunks_fit): the most rows that may fit, cut
// to a whole number of chunks per range like plan_shape's; at least `least`.
int lower_rows(int64_t L, int64_t N, int ni, int T, int64_t entries, int least) {
    int64_t t = T - 8;
    while (t > least && !chunks_fit(t, entries * t / T)) t -= 8;
    if (t <= least) return least;
    const int64_t parts = ceil_div(N, kFusedWarps * ni), R = device_sms() / parts > 0 ? device_sms() / parts : 1;
    const int64_t n = ceil_div(L, t), even = n > R ? round_up(ceil_div(L, round_up(n, R)), 8) : t;
    return static_cast<int>(std::max<int64_t>(least, std::min(t, even)));
}

constexpr int64_t kNarrowMaxN = 2048;  // inputs the register-accumulator grad_x kernel covers

}  // namespace ffi

using namespace ffi;

namespace ffi {
namespace {

constexpr size_t kScratchAlign = 256;
size_t scratch_up(size_t v) { return (v + kScratchAlign - 1) / kScratchAlign * kScratchAlign; }

// Geometry of a plan and the carving of its build scratch (one allocation).
struct PlanLayout {
    long long n, nTiles, scan_segs, nChunks, mostChunks, cptrBytes;
    int T, ni;   // rows per chunk of an even table, inputs per warp
    int leastT;  // rows per chunk that an uneven table is cut down to, at most: cptr and lb hold its mostChunks chunks
    bool chunks;
    size_t off_kA, off_vA, off_kB, off_vB, off_counts, off_bad, off_segs, off_lb, off_stats, total;
};

PlanLayout plan_layout(int64_t L, int64_t K, int64_t N) {
    PlanLayout g;
    g.n = L * K;
    g.nTiles = ceil_div(g.n, kTile);
    g.scan_segs = ceil_div(256 * g.nTiles > N + 1 ? 256 * g.nTiles : N + 1, kScanSeg);
    const PlanShape shape = plan_shape(L, K, N);
    g.T = shape.rows, g.ni = shape.ni;
    g.nChunks = ceil_div(L, g.T > 0 ? g.T : 1);
    // (chunks that leave most of shared memory free, those of short tables, need not get shorter, and their arrays stay small: plan creation
    // at 513 x 73 took 0.9 ms instead of 0.17 where they had just outgrown the blocks that cudaMalloc keeps at hand)
    g.leastT = g.T <= 8 || chunks_fit(g.T, 4 * static_cast<int64_t>(g.T) * K) ? std::max(8, g.T) : std::max(8, g.T / 2 / 8 * 8);
    g.mostChunks = ceil_div(L, std::min(g.T, g.leastT) > 0 ? std::min(g.T, g.leastT) : 1);
    g.cptrBytes = g.mostChunks * (N + 1) * 4;
    g.chunks = g.T >= 8 && N <= kNarrowMaxN && g.nChunks * (N + 1) * 4 <= (512LL << 20) && static_cast<long long>(g.T) * K <= 65536;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t at = off;
        off += scratch_up(bytes ? bytes : 4);
        return at;
    };
    g.off_kA = take(g.n * 4);
    g.off_vA = take(g.n * 4);
    g.off_kB = take(g.n * 4);
    g.off_vB = take(g.n * 4);
    g.off_counts = take(256 * g.nTiles * 4);
    g.off_bad = take(4);
    g.off_segs = take(g.scan_segs * 8);
    g.off_lb = take(g.chunks ? (g.mostChunks + 1) * N * 4 : 4);
    g.off_stats = take((kFusedWarps + 2) * sizeof(int));
    g.total = off;
    return g;
}

// Deals the inputs to the places of the chunked lists: place s is input order[s], a warp has ni places, a slice kFusedWarps warps.  By
// descending count, each to the slice and there to the warp with the fewest entries that has a place left, so that slices and warps
// have about the same number of entries and neighbours, which the lane groups of a warp walk side by side, about the same counts.
void deal_inputs(const int* rowptr, int N, int ni, int* order) {
    int by_count[kNarrowMaxN];
    for (int i = 0; i < N; ++i) by_count[i] = i;
    std::sort(by_count, by_count + N, [&](int a, int b) {
        const int na = rowptr[a + 1] - rowptr[a], nb = rowptr[b + 1] - rowptr[b];
        return na != nb ? na > nb : a < b;
    });
    const int warps = static_cast<int>(ceil_div(N, ni)), slices = static_cast<int>(ceil_div(warps, kFusedWarps));
    long long load[kNarrowMaxN] = {}, slice_load[kNarrowMaxN] = {};  // (ni >= 1)
    int used[kNarrowMaxN] = {};
    auto room = [&](int w) { return used[w] < std::min(ni, N - w * ni); };
    for (int r = 0; r < N; ++r) {
        int best = -1;
        for (int s = 0; s < slices; ++s) {
            if (best >= 0 && slice_load[s] >= slice_load[best / kFusedWarps]) continue;
            int w = -1;
            for (int v = s * kFusedWarps; v < std::min(warps, (s + 1) * kFusedWarps); ++v)
                if (room(v) && (w < 0 || load[v] < load[w])) w = v;
            if (w >= 0) best = w;
        }
        const int i = by_count[r], n = rowptr[i + 1] - rowptr[i];
        order[best * ni + used[best]++] = i;
        load[best] += n, slice_load[best / kFusedWarps] += n;
    }
}

// Fills the (already allocated) arrays of `plan` from `idx`; `scratch` holds plan_layout(...).total bytes.
// Synchronises the stream (index validation, slice statistics).
int plan_build(ffi_plan* plan, const int32_t* idx, unsigned char* scratch, cudaStream_t stream) {
    const int64_t L = plan->L, K = plan->K, N = plan->N;
    const PlanLayout g = plan_layout(L, K, N);
    const long long n = g.n, nTiles = g.nTiles;
    int* kA = reinterpret_cast<int*>(scratch + g.off_kA);
    int* vA = reinterpret_cast<int*>(scratch + g.off_vA);
    int* kB = reinterpret_cast<int*>(scratch + g.off_kB);
    int* vB = reinterpret_cast<int*>(scratch + g.off_vB);
    int* counts = reinterpret_cast<int*>(scratch + g.off_counts);
    int* bad = reinterpret_cast<int*>(scratch + g.off_bad);
    long long* segs = reinterpret_cast<long long*>(scratch + g.off_segs);
    int* lb = reinterpret_cast<int*>(scratch + g.off_lb);
    int* stats = reinterpret_cast<int*>(scratch + g.off_stats);
    int most[kFusedWarps + 2] = {};

    FFI_CUDA_CHECK(cudaMemsetAsync(bad, 0, 4, stream));
    validate_idx_kernel<<<1024, 256, 0, stream>>>(idx, n, static_cast<int>(N), bad);
    int h_bad = 0;
    FFI_CUDA_CHECK(cudaMemcpyAsync(&h_bad, bad, 4, cudaMemcpyDeviceToHost, stream));
    FFI_CUDA_CHECK(cudaStreamSynchronize(stream));
    if (h_bad) return fail(FFI_ERR_INDEX_RANGE, "idx holds a value outside [0, %lld)", (long long)N);

    const int passes = (significant_bits(N) + 7) / 8;
    const unsigned sortBlocks = static_cast<unsigned>(ceil_div(nTiles, kSortWarps));
    const int* kin = idx;
    const int* vin = nullptr;
    int* kout = kA;
    int* vout = vA;
    for (int pass = 0; pass < passes; ++pass) {
        const int shift = 8 * pass;
        radix_hist_kernel<<<sortBlocks, 32 * kSortWarps, 0, stream>>>(kin, n, shift, counts, nTiles);
        const int src = launch_exclusive_scan(counts, 256 * nTiles, segs, stream);
        if (src != FFI_OK) return src;
        radix_scatter_kernel<<<sortBlocks, 32 * kSortWarps, 0, stream>>>(kin, vin, kout, vout, n, shift, counts, nTiles);
        kin = kout;
        vin = vout;
        const bool toB = (kout == kA);
        kout = toB ? kB : kA;
        vout = toB ? vB : vA;
    }
    FFI_LAUNCH_CHECK("radix sort");
    rowptr_kernel<<<static_cast<unsigned>(ceil_div(N + 1, 256)), 256, 0, stream>>>(kin, n, static_cast<int>(N),
                                                                                   plan->rowptr);
    FFI_CUDA_CHECK(cudaMemcpyAsync(plan->perm, vin, n * 4, cudaMemcpyDeviceToDevice, stream));
    FFI_LAUNCH_CHECK("rowptr_kernel");

    plan->order = nullptr;
    int* longest_row = stats + kFusedWarps + 1;
    FFI_CUDA_CHECK(cudaMemsetAsync(longest_row, 0, sizeof(int), stream));
    longest_row_kernel<<<static_cast<unsigned>(ceil_div(N, 256)), 256, 0, stream>>>(plan->rowptr, static_cast<int>(N), longest_row);
    FFI_LAUNCH_CHECK("longest_row_kernel");
    if (!g.chunks) {
        FFI_CUDA_CHECK(cudaMemcpyAsync(&plan->longest_input, longest_row, sizeof(int), cudaMemcpyDeviceToHost, stream));
        FFI_CUDA_CHECK(cudaStreamSynchronize(stream));
        return FFI_OK;
    }

    // Chunked lists for the narrow-input kernels, of T rows a chunk, and what the kernel that stages them in shared memory has to
    // know: the entries per warp, the longest run.
    int T = g.T, longest = 0;
    auto chunk_lists = [&]() -> int {
        const long long chunkEntries = static_cast<long long>(T) * K, nChunks = ceil_div(L, T), nb = (nChunks + 1) * N;
        chunk_bounds_kernel<<<static_cast<unsigned>(ceil_div(nb, 256)), 256, 0, stream>>>(
            plan->rowptr, plan->perm, plan->order, static_cast<int>(N), chunkEntries, nChunks, lb);
        chunk_fill_kernel<<<static_cast<unsigned>(nChunks), 256, (N + 1) * sizeof(int), stream>>>(
            plan->perm, lb, static_cast<int>(N), chunkEntries, plan->cptr, plan->cperm);
        FFI_LAUNCH_CHECK("chunk kernels");
        FFI_CUDA_CHECK(cudaMemsetAsync(stats, 0, (kFusedWarps + 1) * sizeof(int), stream));
        warp_stats_kernel<<<static_cast<unsigned>(ceil_div(N, g.ni)), 256, 0, stream>>>(plan->cptr, static_cast<int>(N), nChunks, g.ni, stats);
        FFI_LAUNCH_CHECK("warp_stats_kernel");
        FFI_CUDA_CHECK(cudaMemcpyAsync(most, stats, sizeof(most), cudaMemcpyDeviceToHost, stream));
        FFI_CUDA_CHECK(cudaStreamSynchronize(stream));
        plan->chunk_rows = T;
        plan->n_chunks = nChunks;
        plan->fused_entries[0] = 0;
        for (int w = 0; w < kFusedWarps; ++w) plan->fused_entries[w + 1] = plan->fused_entries[w] + (most[w] + 1) / 2 * 2;
        longest = most[kFusedWarps];
        plan->longest_input = most[kFusedWarps + 1];
        return FFI_OK;
    };
    auto deal = [&]() -> int {
        int rowptr[kNarrowMaxN + 1], order[kNarrowMaxN];
        FFI_CUDA_CHECK(cudaMemcpyAsync(rowptr, plan->rowptr, (N + 1) * sizeof(int), cudaMemcpyDeviceToHost, stream));
        FFI_CUDA_CHECK(cudaStreamSynchronize(stream));
        deal_inputs(rowptr, static_cast<int>(N), g.ni, order);
        plan->order = plan->order_store;
        FFI_CUDA_CHECK(cudaMemcpyAsync(plan->order, order, N * sizeof(int), cudaMemcpyHostToDevice, stream));
        return FFI_OK;
    };
    int rc = chunk_lists();
    if (rc != FFI_OK) return rc;
    const long long average = ceil_div(static_cast<int64_t>(T) * K, N);
    if (longest > 3 * average + kFusedFarRun || longest > kFusedLongestRun || !chunks_fit(T, plan->fused_entries[kFusedWarps])) {
        // An uneven table: the inputs are dealt anew, and the chunks get shorter until the entries of the largest warps fit (each try
        // takes the kernels above and a round trip to the device: a rebuild at N=768, L=670,091, K=32 takes 1.26 ms for an even table,
        // 1.75 with inputs drawn by Zipf's law of exponent 0.6, 2.3 of 1, 2.9 of 1.3).  Dealt, nearly all fit the chunks of an even
        // table: T stays 272 up to exponent 0.8, 264 at 1, 240 at 1.3.
        rc = deal();
        if (rc == FFI_OK) rc = chunk_lists();
        if (rc != FFI_OK) return rc;
    }
    while (plan->order && T > g.leastT && !chunks_fit(T, plan->fused_entries[kFusedWarps])) {
        T = lower_rows(L, N, g.ni, T, plan->fused_entries[kFusedWarps], g.leastT);
        rc = chunk_lists();
        if (rc != FFI_OK) return rc;
    }
    plan->fused_ni = g.ni;
    plan->range_chunks = g.nChunks;
    plan->has_chunks = true;
    return FFI_OK;
}

}  // namespace
}  // namespace ffi

namespace ffi {
namespace {
__device__ int g_bounds_bad = 0;
std::atomic<int> g_debug_bounds{-1};  // -1: not decided yet (environment), 0: off, 1: on
}  // namespace

bool debug_bounds_enabled() {
    int v = g_debug_bounds.load();
    if (v < 0) {
        const char* e = std::getenv("FFI_DEBUG_BOUNDS");
        v = (e && e[0] != '\0' && e[0] != '0') ? 1 : 0;
        g_debug_bounds.store(v);
    }
    return v == 1;
}

int check_index_range(const int32_t* idx, int64_t n, int64_t N, cudaStream_t stream) {
    int zero = 0, h_bad = 0;
    FFI_CUDA_CHECK(cudaMemcpyToSymbolAsync(g_bounds_bad, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, stream));
    int* bad = nullptr;
    FFI_CUDA_CHECK(cudaGetSymbolAddress(reinterpret_cast<void**>(&bad), g_bounds_bad));
    validate_idx_kernel<<<1024, 256, 0, stream>>>(idx, n, static_cast<int>(N), bad);
    FFI_LAUNCH_CHECK("validate_idx_kernel");
    FFI_CUDA_CHECK(cudaMemcpyAsync(&h_bad, bad, sizeof(int), cudaMemcpyDeviceToHost, stream));
    FFI_CUDA_CHECK(cudaStreamSynchronize(stream));
    if (h_bad) return fail(FFI_ERR_INDEX_RANGE, "debug bounds: idx holds a value outside [0, %lld)", (long long)N);
    return FFI_OK;
}
}  // namespace ffi

extern "C" int ffi_set_debug_bounds(int on) {
    ffi::g_debug_bounds.store(on ? 1 : 0);
    return FFI_OK;
}

extern "C" int ffi_plan_create(const int32_t* idx, int64_t L, int64_t K, int64_t N, void* stream_v,
                               ffi_plan** out_plan) {
    FFI_TRACE("ffi_plan_create");
    if (!out_plan) return fail(FFI_ERR_INVALID_ARGUMENT, "out_plan is NULL");
    *out_plan = nullptr;
    if (!idx) return fail(FFI_ERR_INVALID_ARGUMENT, "idx is NULL");
    if (L <= 0 || K <= 0 || N <= 0) return fail(FFI_ERR_INVALID_ARGUMENT, "L, K, N must be positive");
    if (N >= (1LL << 31) || L * K >= (1LL << 31) - kTile)
        return fail(FFI_ERR_UNSUPPORTED, "L*K=%lld (or N) does not fit 32-bit positions", (long long)(L * K));
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);

    // Owns the half-built plan: every early return below (the CUDA check macros included) frees
    // the plan and its device arrays; success hands it to the caller.
    struct PlanOwner {
        ffi_plan* p;
        ~PlanOwner() {
            if (p) ffi_plan_destroy(p);
        }
    } owner{new ffi_plan()};
    ffi_plan* plan = owner.p;
    plan->L = L;
    plan->K = K;
    plan->N = N;
    FFI_CUDA_CHECK(cudaGetDevice(&plan->device));
    const PlanLayout g = plan_layout(L, K, N);

    // the index arrays are one allocation: a cudaMalloc and a cudaFree of this size take about a millisecond each
    const size_t rowptr_at = 0, perm_at = rowptr_at + scratch_up((N + 1) * sizeof(int)), cptr_at = perm_at + scratch_up(g.n * 4);
    const size_t cperm_at = cptr_at + (g.chunks ? scratch_up(g.cptrBytes) : 0), order_at = cperm_at + (g.chunks ? scratch_up(g.n * 4) : 0),
                 total = order_at + (g.chunks ? scratch_up(N * sizeof(int)) : 0);
    if (cudaMalloc(&plan->arrays, total) != cudaSuccess) {
        cudaGetLastError();
        plan->arrays = nullptr;
        return fail(FFI_ERR_ALLOC, "cudaMalloc of the transposed index failed");
    }
    unsigned char* base = static_cast<unsigned char*>(plan->arrays);
    plan->rowptr = reinterpret_cast<int32_t*>(base + rowptr_at);
    plan->perm = reinterpret_cast<int32_t*>(base + perm_at);
    if (g.chunks) {
        plan->cptr = reinterpret_cast<int32_t*>(base + cptr_at);
        plan->cperm = reinterpret_cast<int32_t*>(base + cperm_at);
        plan->order_store = reinterpret_cast<int32_t*>(base + order_at);
    }
    plan->device_bytes = total;
    DeviceBuffer scratch;
    if (scratch.alloc(g.total) != cudaSuccess) {
        cudaGetLastError();
        return fail(FFI_ERR_ALLOC, "cudaMalloc of sort scratch failed");
    }
    const int rc = plan_build(plan, idx, scratch.as<unsigned char>(), stream);
    if (rc != FFI_OK) return rc;
    owner.p = nullptr;
    *out_plan = plan;
    return FFI_OK;
}

extern "C" int ffi_plan_rebuild(ffi_plan* plan, const int32_t* idx, void* stream_v) {
    FFI_TRACE("ffi_plan_rebuild");
    if (!plan || !idx) return fail(FFI_ERR_INVALID_ARGUMENT, "NULL argument to ffi_plan_rebuild");
    int rc = check_plan_device(plan);
    if (rc != FFI_OK) return rc;
    const PlanLayout g = plan_layout(plan->L, plan->K, plan->N);
    if (!plan->build_scratch) {
        if (cudaMalloc(&plan->build_scratch, g.total) != cudaSuccess) {
            cudaGetLastError();
            plan->build_scratch = nullptr;
            return fail(FFI_ERR_ALLOC, "cudaMalloc of the plan's sort scratch failed");
        }
        plan->device_bytes += g.total;
    }
    return plan_build(plan, idx, static_cast<unsigned char*>(plan->build_scratch), static_cast<cudaStream_t>(stream_v));
}

extern "C" int ffi_plan_destroy(ffi_plan* plan) {
    if (!plan) return FFI_OK;
    if (plan->arrays) cudaFree(plan->arrays);
    if (plan->build_scratch) cudaFree(plan->build_scratch);
    delete plan;
    return FFI_OK;
}

extern "C" int ffi_plan_info(const ffi_plan* plan, int64_t* L, int64_t* K, int64_t* N, int64_t* chunk_rows,
                             int64_t* n_chunks, int64_t* device_bytes) {
    if (!plan) return fail(FFI_ERR_INVALID_ARGUMENT, "plan is NULL");
    if (L) *L = plan->L;
    if (K) *K = plan->K;
    if (N) *N = plan->N;
    if (chunk_rows) *chunk_rows = plan->has_chunks ? plan->chunk_rows : 0;
    if (n_chunks) *n_chunks = plan->has_chunks ? plan->n_chunks : 0;
    if (device_bytes) *device_bytes = static_cast<int64_t>(plan->device_bytes);
    return FFI_OK;
}

extern "C" int ffi_plan_export(const ffi_plan* plan, int32_t* rowptr, int32_t* perm, void* stream_v) {
    if (!plan || !rowptr || !perm) return fail(FFI_ERR_INVALID_ARGUMENT, "NULL argument to ffi_plan_export");
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    FFI_CUDA_CHECK(cudaMemcpyAsync(rowptr, plan->rowptr, (plan->N + 1) * 4, cudaMemcpyDeviceToDevice, stream));
    FFI_CUDA_CHECK(cudaMemcpyAsync(perm, plan->perm, plan->L * plan->K * 4, cudaMemcpyDeviceToDevice, stream));
    return FFI_OK;
}

extern "C" int ffi_plan_export_chunked(const ffi_plan* plan, int32_t* rowptr, int32_t* perm, void* stream_v) {
    if (!plan || !rowptr || !perm)
        return fail(FFI_ERR_INVALID_ARGUMENT, "NULL argument to ffi_plan_export_chunked");
    if (!plan->has_chunks) return fail(FFI_ERR_UNSUPPORTED, "plan has no chunked lists (wide N)");
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    const int N = static_cast<int>(plan->N);
    chunked_row_totals_kernel<<<static_cast<unsigned>(ceil_div(N + 1, 256)), 256, 0, stream>>>(
        plan->cptr, plan->order, N, plan->n_chunks, rowptr);
    small_exclusive_scan_kernel<<<1, 1024, 0, stream>>>(rowptr, N + 1);
    chunked_gather_kernel<<<static_cast<unsigned>(ceil_div(N, 4)), 128, 0, stream>>>(
        plan->cptr, plan->cperm, plan->order, rowptr, N, plan->n_chunks,
        static_cast<long long>(plan->chunk_rows) * plan->K, perm);
    FFI_LAUNCH_CHECK("chunked export");
    return FFI_OK;
}
