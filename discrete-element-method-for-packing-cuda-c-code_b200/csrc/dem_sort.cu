// dem_sort.cu -- RadixSort(pData0, pData1, elements, keybits): the stable
// key/value radix sort that dempacking.cu:553-555 takes from the CUDA SDK
// (radixsort.cu, not in the reference).  LSD, 8-bit digits, ping-pong between
// the two buffers, result in pData0.  One histogram launch counts the digits
// of every pass; then one launch per pass (Adinets & Merrill, "Onesweep: a
// faster least significant digit radix sort for GPUs", 2022): tiles of 4,096
// or 8,192 records take tickets, rank their records by digit (eight ballots in each
// warp, in index order: stable; __match_any_sync took 3x as long), publish their digit counts, add up the
// counts of the tiles before them (decoupled look-back, 16 tiles a round; a
// tile that waits too long for a count reads the records before it instead) and
// write the records out from shared memory in digit order, so that the
// writes are runs.  A pass reads and writes each record once.
#include <mutex>
#include <vector>
#include "dem_common.cuh"
#include "dem_compat_state.h"

namespace dem {

namespace {
constexpr int kRsItems = 16;            // records per thread
constexpr int kHistThreads = 256;
// Threads of a pass's block: tiles of 512 x 16 records from 2^18 records on
// (1,000,000 records: 12.7 us a pass, 256 x 16 15.1: half the tiles to look
// back over), of 256 x 16 below (50,000: 7.0 us, 512 x 16 9.3: more blocks).
constexpr uint kRsLarge = 1u << 18;
constexpr int kRsBack = 16;             // look-back words a thread loads side by side
// Polls without a newly published word (~0.1 s) after which a tile no longer
// waits and counts the records before it itself.  The tiles before it have all
// started (tickets) and wait for none behind them, so this is for a block that
// is kept from running: the order must not depend on how long that takes.
constexpr int kRsSpin = 1 << 16;
// scratch: digit counts of 4 passes, 4 tickets, then two regions of tiles x
// 256 look-back words (a pass uses one and clears the other's for the next)
constexpr size_t kRsHead = 4 * 256 + 64;

// Look-back words: the count, and in the top two bits what it is (1: the
// tile's own, 2: the tiles' up to this one).  32 bits to 2^30 - 1 records.
template <typename W> struct LbWord {
    static constexpr W own = (W)1 << (8 * sizeof(W) - 2), incl = (W)2 << (8 * sizeof(W) - 2), mask = own - 1;
};
__device__ __forceinline__ uint rs_load(const uint* p) {
    uint v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long rs_load(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void rs_store(uint* p, uint v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void rs_store(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Digit counts of every pass (grid-stride).
__global__ void __launch_bounds__(kHistThreads) k_radix_hist(const uint2* __restrict__ in, uint n, int passes,
                                                             uint* __restrict__ hist) {
    __shared__ uint cnt[4][256];
    for (int k = threadIdx.x; k < 256 * passes; k += kHistThreads) cnt[k >> 8][k & 255] = 0u;
    __syncthreads();
    const size_t stride = (size_t)gridDim.x * kHistThreads;
    for (size_t i = (size_t)blockIdx.x * kHistThreads + threadIdx.x; i < n; i += 4 * stride) {
        uint k[4];
#pragma unroll
        for (int e = 0; e < 4; e++) k[e] = i + e * stride < n ? in[i + e * stride].x : 0u;   // loads side by side
#pragma unroll
        for (int e = 0; e < 4; e++)
            if (i + e * stride < n)
                for (int p = 0; p < passes; p++) atomicAdd(&cnt[p][(k[e] >> (8 * p)) & 255u], 1u);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < 256 * passes; k += kHistThreads) {
        const uint c = cnt[k >> 8][k & 255];
        if (c) atomicAdd(hist + k, c);
    }
}

// Exclusive scan of one value per thread over the block; tmp: a word per warp.
template <int kRsWarps> __device__ __forceinline__ uint rs_exscan(uint v, uint* tmp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint inc = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint x = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += x;
    }
    if (lane == 31) tmp[warp] = inc;
    __syncthreads();
    uint base = 0;
#pragma unroll
    for (int w = 0; w < kRsWarps; w++) base += w < warp ? tmp[w] : 0u;
    __syncthreads();
    return base + inc - v;
}

template <typename W, int kRsThreads>
__global__ void __launch_bounds__(kRsThreads) k_radix_pass(const uint2* __restrict__ in, uint2* __restrict__ out, uint n,
                                                           int pass, const uint* __restrict__ hist, uint* ticket,
                                                           W* __restrict__ look, W* __restrict__ other) {
    constexpr int kRsTile = kRsThreads * kRsItems, kRsWarps = kRsThreads / 32;
    extern __shared__ __align__(16) unsigned char smem[];
    uint2* s_kv = reinterpret_cast<uint2*>(smem);                              // kRsTile records
    uint(*s_cnt)[256] = reinterpret_cast<uint(*)[256]>(smem + kRsTile * 8);    // per warp and digit
    __shared__ uint s_off[256], s_tmp[kRsWarps], s_tile;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, shift = 8 * pass;
    if (t == 0) s_tile = atomicAdd(ticket, 1u);
    for (int k = t; k < kRsWarps * 256; k += kRsThreads) s_cnt[k >> 8][k & 255] = 0u;
    __syncthreads();
    const uint tile = s_tile;
    if (tile >= gridDim.x) return;
    if (t < 256) other[(size_t)tile * 256 + t] = 0;   // for the next pass
    const uint base = tile * (uint)kRsTile;
    const uint m = min((uint)kRsTile, n - base);   // records of this tile
    const uint lt = (1u << lane) - 1u;
    uint2 kv[kRsItems];
    uint rank[kRsItems];
#pragma unroll
    for (int e = 0; e < kRsItems; e++) {
        const uint j = warp * (kRsItems * 32) + e * 32 + lane;
        kv[e] = j < m ? in[base + j] : make_uint2(0u, 0u);
    }
    uint peers[kRsItems];
#pragma unroll
    for (int e = 0; e < kRsItems; e++) {
        const uint j = warp * (kRsItems * 32) + e * 32 + lane;
        const uint d = kv[e].x >> shift;
        uint same = __ballot_sync(0xffffffffu, j < m);
#pragma unroll
        for (int b = 0; b < 8; b++) {
            const bool bit = (d >> b) & 1u;
            const uint v = __ballot_sync(0xffffffffu, bit);
            same &= bit ? v : ~v;
        }
        peers[e] = same;   // the valid lanes with this digit
    }
#pragma unroll
    for (int e = 0; e < kRsItems; e++) {
        const uint j = warp * (kRsItems * 32) + e * 32 + lane;
        const uint d = (kv[e].x >> shift) & 255u;
        uint before = 0;
        if (j < m) before = s_cnt[warp][d];
        rank[e] = before + __popc(peers[e] & lt);
        __syncwarp();
        if (j < m && lane == __ffs(peers[e]) - 1) s_cnt[warp][d] = before + __popc(peers[e]);
        __syncwarp();
    }
    __syncthreads();
    // digit t: the warps' counts to offsets, the tile's count
    uint cnt = 0;
    W* mine = look + (size_t)tile * 256 + t;
    if (t < 256) {
#pragma unroll
        for (int w = 0; w < kRsWarps; w++) {
            const uint c = s_cnt[w][t];
            s_cnt[w][t] = cnt;
            cnt += c;
        }
        rs_store(mine, (tile == 0 ? LbWord<W>::incl : LbWord<W>::own) | (W)cnt);
    }
    const uint first = rs_exscan<kRsWarps>(cnt, s_tmp);   // digit's first record in the sorted tile
    const uint global = rs_exscan<kRsWarps>(t < 256 ? hist[256 * pass + t] : 0u, s_tmp);   // and in the output
    W pre = 0;
    bool gave_up = false;
    if (tile > 0 && t < 256) {
        long long b = (long long)tile - 1;
        int spin = 0;
        for (bool done = false; !done;) {
            W w[kRsBack];
#pragma unroll
            for (int k = 0; k < kRsBack; k++)
                w[k] = b - k >= 0 ? rs_load(look + (size_t)(b - k) * 256 + t) : LbWord<W>::incl;
            int used = 0;
#pragma unroll
            for (int k = 0; k < kRsBack; k++) {
                if (done || used < k) continue;   // up to the first word not yet published
                if (!(w[k] & ~LbWord<W>::mask)) continue;
                pre += w[k] & LbWord<W>::mask;
                used = k + 1;
                done = (w[k] & LbWord<W>::incl) != 0;
            }
            b -= used;
            spin = used ? 0 : spin + 1;
            gave_up = spin > kRsSpin;
            if (gave_up) break;
        }
        if (!gave_up) rs_store(mine, LbWord<W>::incl | (pre + (W)cnt));
    }
    if (t < 256) {
        s_off[t] = global + (uint)pre - first;
#pragma unroll
        for (int w = 0; w < kRsWarps; w++) s_cnt[w][t] += first;
    }
    if (__syncthreads_or(gave_up)) {   // the records before this tile, counted from the input
        uint* s_before = reinterpret_cast<uint*>(smem);
        if (t < 256) s_before[t] = 0u;
        __syncthreads();
        for (uint j = t; j < base; j += kRsThreads) atomicAdd(&s_before[(in[j].x >> shift) & 255u], 1u);
        __syncthreads();
        if (gave_up) {
            s_off[t] = global + s_before[t] - first;
            rs_store(mine, LbWord<W>::incl | (W)(s_before[t] + cnt));
        }
        __syncthreads();
    }
#pragma unroll
    for (int e = 0; e < kRsItems; e++) {
        const uint j = warp * (kRsItems * 32) + e * 32 + lane;
        if (j < m) s_kv[s_cnt[warp][(kv[e].x >> shift) & 255u] + rank[e]] = kv[e];
    }
    __syncthreads();
    for (uint j = t; j < m; j += kRsThreads) {
        const uint2 v = s_kv[j];
        out[s_off[(v.x >> shift) & 255u] + j] = v;
    }
}

size_t rs_tiles(uint n) {
    const size_t tile = (size_t)kRsItems * (n < kRsLarge ? 256 : 512);
    return n ? ((size_t)n + tile - 1) / tile : 1;
}
size_t rs_word(uint n) { return n < (1u << 30) ? 1 : 2; }

template <typename W, int NT>
int radix_passes(uint2* d0, uint2* d1, uint n, int passes, uint* scratch, cudaStream_t s) {
    constexpr int smem = NT * kRsItems * 8 + (NT / 32) * 256 * 4;
    const unsigned nt = (unsigned)rs_tiles(n);
    uint* hist = scratch;
    uint* ticket = scratch + 4 * 256;
    W* look = reinterpret_cast<W*>(scratch + kRsHead);
    DEM_CUDA_TRY(cudaFuncSetAttribute(k_radix_pass<W, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    // the counts, the tickets and the first pass's look-back words
    DEM_CUDA_TRY(cudaMemsetAsync(scratch, 0, kRsHead * sizeof(uint) + (size_t)nt * 256 * sizeof(W), s));
    const unsigned hb = grid_for(n, 4 * kHistThreads);
    k_radix_hist<<<hb < 296 ? hb : 296, kHistThreads, 0, s>>>(d0, n, passes, hist);
    DEM_LAUNCH_CHECK();
    uint2 *src = d0, *dst = d1;
    for (int p = 0; p < passes; p++) {
        W* mine = look + (size_t)(p & 1) * nt * 256;
        W* other = look + (size_t)(1 - (p & 1)) * nt * 256;
        k_radix_pass<W, NT><<<nt, NT, smem, s>>>(src, dst, n, p, hist, ticket + p, mine, other);
        DEM_LAUNCH_CHECK();
        uint2* t = src; src = dst; dst = t;
    }
    if (src != d0) DEM_CUDA_TRY(cudaMemcpyAsync(d0, src, (size_t)n * sizeof(uint2), cudaMemcpyDeviceToDevice, s));
    return DEM_OK;
}
}  // namespace

size_t radix_scratch_words(uint n) { return kRsHead + 2 * rs_tiles(n) * 256 * rs_word(n); }

// Sort with caller-provided scratch of radix_scratch_words(n) uint32 (8-byte
// aligned).
int radix_sort_pairs(uint2* d0, uint2* d1, uint n, uint keybits, uint* scratch, cudaStream_t s) {
    if (n <= 1) return DEM_OK;
    if (keybits == 0) return DEM_OK;
    if (keybits > 32) keybits = 32;
    const int passes = (int)((keybits + 7) / 8);
    if (n < kRsLarge) return radix_passes<uint, 256>(d0, d1, n, passes, scratch, s);
    return rs_word(n) == 1 ? radix_passes<uint, 512>(d0, d1, n, passes, scratch, s)
                           : radix_passes<unsigned long long, 512>(d0, d1, n, passes, scratch, s);
}

}  // namespace dem

extern "C" int RadixSort(KeyValuePair* pData0, KeyValuePair* pData1, unsigned int elements, unsigned int keybits) {
    if (elements > 1 && (!pData0 || !pData1)) return dem::fail(DEM_ERR_ARG, "RadixSort: null buffer");
    if (elements <= 1) return DEM_OK;
    dem::CompatDevice* cd = nullptr;
    int rc = dem::compat_device(&cd);
    if (rc) return rc;
    uint* scratch = nullptr;
    rc = dem::compat_scratch(cd, dem::radix_scratch_words(elements), &scratch);
    if (rc) return rc;
    return dem::radix_sort_pairs(reinterpret_cast<uint2*>(pData0), reinterpret_cast<uint2*>(pData1), elements, keybits,
                                 scratch, dem::compat_stream());
}

// ---------------------------------------------------------------------------
// RadixSortNoAlloc: the same stable sort for callers that must not allocate
// device memory, e.g. a host loop that owns all of HBM through its own pool
// allocator, or a latency-critical loop in which a first-call cudaMalloc (and
// the device synchronisation it may cause) is not acceptable.  Its scratch
// (digit counts and look-back words) lives in the fixed device array below,
// sized for at most kNoAllocMaxRecords records (about 1 MiB); every GPU that
// loads this library holds that array until the process exits.
//
// The first call on a device resolves the array's device address with
// cudaGetSymbolAddress while that device is current (host code cannot use the
// symbol itself: on the host it names a stand-in, not device memory).  Under
// CUDA's lazy module loading that call may be the one that loads this
// library's device code, which reserves device memory: make the first call
// during set-up, before any stream capture; later calls allocate nothing.  All calls share the one array,
// which keeps the contents of the last call (each call clears what it uses),
// and two calls that overlap on
// the GPU (different streams, or different host threads on the same device)
// race on it and must be serialised by the caller.
namespace dem {
namespace {
constexpr unsigned kNoAllocMaxRecords = 1u << 22;                        // 4,194,304
constexpr size_t kNoAllocWords = kRsHead + (size_t)2 * 256 * (kNoAllocMaxRecords / (kRsItems * 512));
__device__ __align__(256) unsigned int g_noalloc_scratch[kNoAllocWords];

std::mutex g_noalloc_mu;
std::vector<std::pair<int, uint*>> g_noalloc_addr;   // (device, device address of g_noalloc_scratch)

int noalloc_scratch(uint** out) {
    int dev = 0;
    DEM_CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    for (auto& e : g_noalloc_addr)
        if (e.first == dev) { *out = e.second; return DEM_OK; }
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)", __FILE__, __LINE__);
    g_noalloc_addr.emplace_back(dev, (uint*)p);
    *out = (uint*)p;
    return DEM_OK;
}
}  // namespace
}  // namespace dem

extern "C" int RadixSortNoAlloc(KeyValuePair* pData0, KeyValuePair* pData1, unsigned int elements,
                                unsigned int keybits) {
    if (elements > dem::kNoAllocMaxRecords)
        return dem::fail(DEM_ERR_ARG, "RadixSortNoAlloc: %u records exceed the fixed scratch limit of %u records",
                         elements, dem::kNoAllocMaxRecords);
    if (elements > 1 && (!pData0 || !pData1)) return dem::fail(DEM_ERR_ARG, "RadixSortNoAlloc: null buffer");
    if (elements <= 1) return DEM_OK;
    if (dem::radix_scratch_words(elements) > dem::kNoAllocWords)
        return dem::fail(DEM_ERR_ARG, "RadixSortNoAlloc: scratch sizing error");
    uint* scratch = nullptr;
    int rc = dem::noalloc_scratch(&scratch);
    if (rc) return rc;
    return dem::radix_sort_pairs(reinterpret_cast<uint2*>(pData0), reinterpret_cast<uint2*>(pData1), elements, keybits,
                                 scratch, dem::compat_stream());
}
