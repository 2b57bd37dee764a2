// ys_sort.cu -- stable LSD radix sort of (uint32 key, uint32 value) pairs.
//
// Restates the reference RadixSorter (spatial_hash.hpp:48-70,
// radixsort.metal:21-111): 8-bit digits, least significant first, stable, the
// value carried with its key.  Because the sort is stable and the values enter
// in index order, the output is the unique (key, original index) order, so it
// is bit-identical to the CPU twin radixSortCPU (bvh.hpp:723-765).
//
// B200 design: one kernel counts the digits of every pass, then one kernel per
// pass reads each pair once and writes it once.
//   tile     -- a CTA takes the next tile of pairs (a ticket, so a tile's
//               predecessors have started); warp w holds its w-th run of
//               32 x ITEMS pairs, lane l of item k the pair k * 32 + l of it;
//   rank     -- per item, the warp's lanes with the same digit take
//               consecutive ranks after the warp's earlier ones (a private
//               256-entry count per warp: no barrier); then a scan over warps
//               and digits;
//   base     -- the tile publishes its digit counts and adds up its
//               predecessors' (decoupled look-back, Merrill & Garland 2016, in
//               two levels): a word per tile and digit holds the tile's count,
//               a word per 16 tiles and digit their sum or, once known, the
//               sum up to them -- with every tile of a sort resident at once
//               a single level was a walk over all of them;
//   write    -- keys, then values, go to their ranks in shared memory and
//               from there to the output, where a digit's run is contiguous.
// A look-back that meets no count within its poll limit counts that tile's
// keys itself, so no wait is unbounded.  Up to SMALL pairs one CTA runs every
// pass.
//
// Bound by shared-memory accesses and their conflicts (about 30 wavefronts per
// 32 pairs and pass).  A sort of 30-bit keys, us (three launches per pass
// before: histogram, scan, scatter): 5120 pairs 107 -> 32, 300,000 112 -> 59,
// 3M 221 -> 129, 16M 742 -> 457.  Ranking by match.any instead of the mask
// words 165 us a 16M pass, by a ballot per bit 122, by mask words 99.
#include <algorithm>

#include "ys_common.cuh"
#include "ys_sort.cuh"

namespace ys {

// Tile shapes (threads x items); see sort_large.  Four 256-thread CTAs per SM
// with 20 items: a 16M pass 99 us; 12 items 109, 16 items 101, 24 items 106,
// 512 threads x 16 items 132.
static constexpr int LT = 256, LI = 20;              // 5120 pairs
static constexpr int ST = 256, SI = 8;               // 2048 pairs
static constexpr int MT = 512, MI = 11;              // the one-CTA sort: what 48 KB of shared memory hold
static constexpr u32 SMALL = MT * MI;
#ifndef YS_SORT_LOOK_POLLS  // a test builds this file with 0
#define YS_SORT_LOOK_POLLS (1u << 16)
#endif
static constexpr u32 LOOK_POLLS = YS_SORT_LOOK_POLLS;
static constexpr u32 LOOK = 8;         // words loaded together
static constexpr u32 LOOK_GROUP = 16;  // tiles whose counts are summed into one word

// Look-back words: a tag naming the pass and what the value is, then the
// value.  Tags of earlier passes read as "nothing yet", so the words are
// cleared once per sort.  28-bit values in 32-bit words; 60-bit values in
// 64-bit words for 2^28 pairs and more.
template <class W> struct LookWord;
template <> struct LookWord<u32> { static constexpr int BITS = 28; };
template <> struct LookWord<u64> { static constexpr int BITS = 60; };
template <class W> __device__ __forceinline__ W look_word(u32 tag, u64 v) { return ((W)tag << LookWord<W>::BITS) | (W)v; }
__device__ __forceinline__ u32 look_load(const u32* p) {
    u32 v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ u64 look_load(const u64* p) {
    u64 v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void look_store(u32* p, u32 v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void look_store(u64* p, u64 v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Digit counts of every pass: counts[pass * 256 + digit].
static constexpr int COUNT_THREADS = 256;
__global__ void __launch_bounds__(COUNT_THREADS) k_sort_count(const u32* __restrict__ keys, u32 n, int beginBit,
                                                              int passes, u32* __restrict__ counts) {
    __shared__ u32 h[4 * 256];
    for (int k = threadIdx.x; k < 4 * 256; k += COUNT_THREADS) h[k] = 0;
    __syncthreads();
    auto add = [&](u32 key) {
        for (int p = 0; p < passes; ++p) atomicAdd(&h[p * 256 + ((key >> (beginBit + 8 * p)) & 255u)], 1u);
    };
    const u64 step = (u64)gridDim.x * COUNT_THREADS * 4;
    for (u64 i0 = ((u64)blockIdx.x * COUNT_THREADS + (threadIdx.x & ~31u)) * 4 + (threadIdx.x & 31u); i0 < n; i0 += step) {
        u32 k[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) k[q] = i0 + 32 * q < n ? keys[i0 + 32 * q] : 0u;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (i0 + 32 * q < n) add(k[q]);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < passes * 256; k += COUNT_THREADS)
        if (h[k]) atomicAdd(&counts[k], h[k]);
}

template <int THREADS, int ITEMS>
struct SortShared {
    static_assert(THREADS >= 256, "a thread per digit");
    static constexpr int WARPS = THREADS / 32;
    u32 mask[WARPS][256];             // per warp and digit: the lanes of the current item with that digit
    unsigned short warp[WARPS][256];  // per warp and digit: keys so far, then the warp's first rank
    u32 out[256];     // output position of a digit's first pair of this tile, less that rank
    u64 scan[8];
    u32 ticket;
    u32 buf[THREADS * ITEMS];
};

// Exclusive scan of one value per thread over the first 256 threads (every
// thread calls it).
template <int THREADS, class S>
__device__ __forceinline__ u64 scan256(S& sh, u64 v) {
    const u32 tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    u64 x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= (u32)o) x += y;
    }
    if (w < 8 && lane == 31) sh.scan[w] = x;
    __syncthreads();
    u64 before = 0;
    if (w < 8)
        for (u32 q = 0; q < w; ++q) before += sh.scan[q];
    __syncthreads();
    return before + x - v;
}

// Ranks of the thread's pairs among the warp's (stable), and per warp and
// digit the count; then, per digit (threads 0..255), the count of the tile, the
// warps' counts replaced by the warps' first ranks in the digit.
template <int THREADS, int ITEMS, class S>
__device__ __forceinline__ u32 tile_rank(S& sh, const u32 (&key)[ITEMS], int shift, u32 (&rank)[ITEMS]) {
    const u32 tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    for (u32 d = lane; d < 256u; d += 32u) { sh.warp[w][d] = 0; sh.mask[w][d] = 0; }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const u32 d = (key[k] >> shift) & 255u;
        atomicOr(&sh.mask[w][d], 1u << lane);
        __syncwarp();
        const unsigned peers = sh.mask[w][d];
        const u32 before = sh.warp[w][d];
        const u32 lower = (u32)__popc(peers & ((1u << lane) - 1u));
        __syncwarp();
        if (lower == 0) {
            sh.warp[w][d] = (unsigned short)(before + (u32)__popc(peers));
            sh.mask[w][d] = 0;
        }
        __syncwarp();
        rank[k] = before + lower;
    }
    __syncthreads();
    u32 total = 0;
    if (tid < 256u) {
#pragma unroll
        for (int q = 0; q < THREADS / 32; ++q) {
            const u32 c = sh.warp[q][tid];
            sh.warp[q][tid] = (unsigned short)total;
            total += c;
        }
    }
    return total;
}

// The digits' first ranks in the tile (threads 0..255) added to the warps'.
template <int THREADS, class S>
__device__ __forceinline__ void tile_offsets(S& sh, u32 start) {
    if (threadIdx.x < 256u) {
#pragma unroll
        for (int q = 0; q < THREADS / 32; ++q) sh.warp[q][threadIdx.x] += (unsigned short)start;
    }
    __syncthreads();
}

// Sum of this digit's words 0 .. n - 1 (256 apart), from the last down to the
// first or to one tagged `upto`, which holds the sum up to itself.  LOOK words
// are loaded together; one that is not there yet is polled by loading the
// step again from it, and past the poll limit count(word) takes its place.
template <class W, class Count>
__device__ __forceinline__ u64 look_back(const W* words, u32 n, u32 own, u32 upto, Count&& count) {
    u64 sum = 0;
    for (u32 p = n; p > 0;) {
        W v[LOOK];
#pragma unroll
        for (u32 q = 0; q < LOOK; ++q) v[q] = q < p ? look_load(words + (size_t)(p - 1 - q) * 256) : (W)0;
        bool more = true;
#pragma unroll
        for (u32 q = 0; q < LOOK; ++q) {
            const u32 tag = (u32)(v[q] >> LookWord<W>::BITS);
            more = more && p > 0 && (tag == own || tag == upto);
            if (more) {
                sum += (u64)(v[q] & (((W)1 << LookWord<W>::BITS) - 1));
                p = tag == upto ? 0 : p - 1;
            }
        }
        if (more || p == 0) continue;
        // not there yet: poll this word alone (a step's loads, repeated by
        // every thread of every waiting tile, kept the L2 from the others)
        u32 tag = 0;
        for (u32 polls = 0; polls < LOOK_POLLS && tag != own && tag != upto; ++polls) {
            __nanosleep(32);
            tag = (u32)(look_load(words + (size_t)(p - 1) * 256) >> LookWord<W>::BITS);
        }
        if (tag != own && tag != upto) sum += count(--p);
    }
    return sum;
}

// One pass over one tile per CTA.
template <int THREADS, int ITEMS, class W>
__global__ void __launch_bounds__(THREADS, 4) k_sort_pass(const u32* __restrict__ kin, const u32* __restrict__ vin,
                                                       u32* __restrict__ kout, u32* __restrict__ vout, u32 n,
                                                       int shift, u32 pass, const u32* __restrict__ counts,
                                                       u32* __restrict__ tickets, W* __restrict__ look) {
    __shared__ SortShared<THREADS, ITEMS> sh;
    constexpr u32 TILE = THREADS * ITEMS;
    const u32 tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    if (tid == 0) sh.ticket = atomicAdd(&tickets[pass], 1u);
    __syncthreads();
    const u32 tile = sh.ticket, base = tile * TILE;
    const u32 count = min(TILE, n - base);
    // past the end: the largest key, ranked after every real pair of its digit
    u32 key[ITEMS], val[ITEMS], rank[ITEMS];
    const u32 first = w * (32u * ITEMS) + lane;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const u32 i = first + 32u * (u32)k;
        key[k] = i < count ? __ldcs(kin + base + i) : 0xFFFFFFFFu;
    }
    const u32 TAG_OWN = 2u * pass + 1u, TAG_SUM = 2u * pass + 2u;
    W* group = look + (size_t)gridDim.x * 256;
    const u32 mine = tile_rank<THREADS, ITEMS>(sh, key, shift, rank);
    // publish, then scan the digit counts of the tile and of the whole input
    if (tid < 256u) look_store(look + (size_t)tile * 256 + tid, look_word<W>(TAG_OWN, mine));
    const u32 all = tid < 256u ? counts[pass * 256u + tid] : 0u;
    const u64 both = scan256<THREADS>(sh, ((u64)all << 24) | mine);  // the tile's counts sum to THREADS x ITEMS
    const u32 start = (u32)(both & 0xFFFFFFu);
    tile_offsets<THREADS>(sh, start);
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        rank[k] += sh.warp[w][(key[k] >> shift) & 255u];
        sh.buf[rank[k]] = key[k];
    }
    if (tid < 256u) {
        const u32 g = tile / LOOK_GROUP, r = tile % LOOK_GROUP;
        auto count = [&](u32 t0, u32 t1) {  // keys of this digit in tiles [t0, t1)
            u64 c = 0;
            for (size_t i = (size_t)t0 * TILE; i < (size_t)t1 * TILE; ++i) c += ((kin[i] >> shift) & 255u) == tid ? 1u : 0u;
            return c;
        };
        // the group's earlier tiles, then the earlier groups
        u64 sum = look_back<W>(look + (size_t)(g * LOOK_GROUP) * 256 + tid, r, TAG_OWN, 0xFFu,
                               [&](u32 q) { return count(g * LOOK_GROUP + q, g * LOOK_GROUP + q + 1); });
        const bool last = r == LOOK_GROUP - 1u;
        if (last) look_store(group + (size_t)g * 256 + tid, look_word<W>(g ? TAG_OWN : TAG_SUM, sum + mine));
        sum += look_back<W>(group + tid, g, TAG_OWN, TAG_SUM,
                            [&](u32 q) { return count(q * LOOK_GROUP, (q + 1) * LOOK_GROUP); });
        if (last && g) look_store(group + (size_t)g * 256 + tid, look_word<W>(TAG_SUM, sum + mine));
        sh.out[tid] = (u32)((both >> 24) + sum - start);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const u32 i = first + 32u * (u32)k;
        val[k] = i < count ? __ldcs(vin + base + i) : 0u;
    }
    u32 dst[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const u32 i = (u32)k * THREADS + tid;
        const u32 q = sh.buf[i];
        dst[k] = sh.out[(q >> shift) & 255u] + i;
        if (i < count) kout[dst[k]] = q;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) sh.buf[rank[k]] = val[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const u32 i = (u32)k * THREADS + tid;
        if (i < count) vout[dst[k]] = sh.buf[i];
    }
}

// Every pass of up to SMALL pairs in one CTA, in place.
__global__ void __launch_bounds__(MT) k_sort_small(u32* __restrict__ keys, u32* __restrict__ vals, u32 n, int beginBit,
                                                   int endBit) {
    __shared__ SortShared<MT, MI> sh;
    const u32 tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    u32 key[MI], val[MI], rank[MI];
    const u32 first = w * (32u * MI) + lane;
#pragma unroll
    for (int k = 0; k < MI; ++k) {
        const u32 i = first + 32u * (u32)k;
        key[k] = i < n ? keys[i] : 0xFFFFFFFFu;
        val[k] = i < n ? vals[i] : 0u;
    }
    for (int shift = beginBit; shift < endBit; shift += 8) {
        const u32 mine = tile_rank<MT, MI>(sh, key, shift, rank);
        const u64 start = scan256<MT>(sh, mine);
        tile_offsets<MT>(sh, (u32)start);
#pragma unroll
        for (int k = 0; k < MI; ++k) {
            rank[k] += sh.warp[w][(key[k] >> shift) & 255u];
            sh.buf[rank[k]] = key[k];
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < MI; ++k) key[k] = sh.buf[first + 32u * (u32)k];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < MI; ++k) sh.buf[rank[k]] = val[k];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < MI; ++k) val[k] = sh.buf[first + 32u * (u32)k];
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < MI; ++k) {
        const u32 i = first + 32u * (u32)k;
        if (i < n) { keys[i] = key[k]; vals[i] = val[k]; }
    }
}

// Large tiles once there are enough of them to fill the chip (a pass of
// 700,000 pairs 9.9 us in small tiles, of 1M 15.6 in small and 12.2 in large).
static bool sort_large(u32 n) { return n >= 148u * LT * LI; }
static constexpr u32 sort_tiles(u32 n, bool large) {
    const u32 tile = large ? LT * LI : ST * SI;
    return n / tile + (n % tile ? 1u : 0u);
}
static constexpr u32 look_words(u32 tiles) { return 256u * (tiles + (tiles + LOOK_GROUP - 1u) / LOOK_GROUP); }
static constexpr size_t SORT_HEAD = 4 * 256 + 64;  // words: counts of 4 passes, tickets

// Monotone in n: a scratch for n pairs serves every smaller sort.
size_t sort_scratch_bytes(u32 n) {
    if (n == 0) n = 1;
    const u32 edge = 148u * LT * LI - 1u;
    const size_t words = std::max<size_t>(n > edge ? (size_t)look_words(sort_tiles(n, true)) * (n >= (1u << 28) ? 2 : 1) : 0,
                                          look_words(sort_tiles(std::min(n, edge), false)));
    return 4 * (SORT_HEAD + words + (size_t)2 * n) + 8;
}

template <int THREADS, int ITEMS, class W>
static void sort_passes(u32* keys, u32* vals, u32 n, u32* head, W* look, u32* k2, u32* v2, int beginBit, int passes,
                        cudaStream_t s) {
    const u32 tiles = (u32)ceil_div(n, THREADS * ITEMS);
    k_sort_count<<<std::min<u32>((u32)ceil_div(n, COUNT_THREADS * 16), 148 * 8), COUNT_THREADS, 0, s>>>(keys, n, beginBit,
                                                                                                     passes, head);
    for (int p = 0; p < passes; ++p) {
        k_sort_pass<THREADS, ITEMS, W><<<tiles, THREADS, 0, s>>>(keys, vals, k2, v2, n, beginBit + 8 * p, (u32)p, head,
                                                                 head + 4 * 256, look);
        std::swap(keys, k2);
        std::swap(vals, v2);
    }
}

static int sort_pass_count(int beginBit, int endBit) { return (endBit - beginBit + 7) / 8; }

// Scratch: head (counts, tickets), look-back words (8-byte aligned), the other halves.
struct SortScratch {
    u32 *head, *look, *k2, *v2;
    size_t words;  // of look
};
static SortScratch sort_scratch(void* scratch, u32 n, bool large) {
    SortScratch S;
    S.head = (u32*)(((uintptr_t)scratch + 7) & ~(uintptr_t)7);
    S.look = S.head + SORT_HEAD;
    S.words = (size_t)look_words(sort_tiles(n, large)) * (n >= (1u << 28) ? 2 : 1);
    S.k2 = S.look + S.words;
    S.v2 = S.k2 + n;
    return S;
}

// Sort keys/vals in place.  scratch must hold sort_scratch_bytes(n) bytes
// (large: of sort_large tiles only, see the allocation-free sort).  staged: the
// pairs are where sort_input says.
static cudaError_t sort_in(u32* keys, u32* vals, u32 n, void* scratch, int beginBit, int endBit, bool large,
                           cudaStream_t s, bool staged = false) {
    if (n <= 1 || endBit <= beginBit) return cudaSuccess;
    const int passes = sort_pass_count(beginBit, endBit);
    if (n <= SMALL) {
        k_sort_small<<<1, MT, 0, s>>>(keys, vals, n, beginBit, beginBit + 8 * passes);
        return cudaGetLastError();
    }
    const bool wide = n >= (1u << 28);
    const SortScratch S = sort_scratch(scratch, n, large);
    u32 *head = S.head, *look = S.look, *k2 = S.k2, *v2 = S.v2;
    cudaError_t e = cudaMemsetAsync(head, 0, 4 * (SORT_HEAD + S.words), s);
    if (e != cudaSuccess) return e;
    if (staged && (passes & 1)) {  // the last pass ends in the caller's arrays
        std::swap(keys, k2);
        std::swap(vals, v2);
    }
    if (wide) sort_passes<LT, LI, u64>(keys, vals, n, head, (u64*)look, k2, v2, beginBit, passes, s);
    else if (large) sort_passes<LT, LI, u32>(keys, vals, n, head, look, k2, v2, beginBit, passes, s);
    else sort_passes<ST, SI, u32>(keys, vals, n, head, look, k2, v2, beginBit, passes, s);
    if ((passes & 1) && !staged) {
        cudaMemcpyAsync(keys, k2, (size_t)n * 4, cudaMemcpyDeviceToDevice, s);
        cudaMemcpyAsync(vals, v2, (size_t)n * 4, cudaMemcpyDeviceToDevice, s);
    }
    return cudaGetLastError();
}

cudaError_t radix_sort_pairs(u32* keys, u32* vals, u32 n, void* scratch, int beginBit, int endBit, cudaStream_t s) {
    return sort_in(keys, vals, n, scratch, beginBit, endBit, sort_large(n), s);
}

void sort_input(u32*& keys, u32*& vals, u32 n, void* scratch, int beginBit, int endBit) {
    if (n <= SMALL || !(sort_pass_count(beginBit, endBit) & 1)) return;
    const SortScratch S = sort_scratch(scratch, n, sort_large(n));
    keys = S.k2;
    vals = S.v2;
}

cudaError_t radix_sort_staged(u32* keys, u32* vals, u32 n, void* scratch, int beginBit, int endBit, cudaStream_t s) {
    return sort_in(keys, vals, n, scratch, beginBit, endBit, sort_large(n), s, true);
}

}  // namespace ys

// ---------------------------------------------------------------------------
// Sort with no allocation at all, for callers that cannot call cudaMalloc:
// code that runs inside a CUDA-graph capture or an allocation-free real-time
// loop, hosts whose device memory is owned by another allocator (a game
// engine's or a framework's pool), and plugins that must not grow the
// process's device footprint behind the host's back.  The scratch lives in a
// file-scope __device__ array of fixed size, reserved on every GPU that loads
// this library until the process exits.
#include <mutex>
#include <string>

#include "ysim_b200.h"

namespace ys {
ys_status fail(ys_status code, const std::string& msg);

static constexpr u32 NOALLOC_MAX_PAIRS = 1u << 20;  // 1,048,576 pairs
static constexpr size_t NOALLOC_SCRATCH_BYTES = 8651776;
static_assert(4 * (SORT_HEAD + look_words(sort_tiles(NOALLOC_MAX_PAIRS, true)) + 2 * (size_t)NOALLOC_MAX_PAIRS) + 8 <=
                  NOALLOC_SCRATCH_BYTES,
              "the allocation-free sort's scratch holds the large tiles' words");
static __device__ __align__(256) unsigned char g_noalloc_sort_scratch[NOALLOC_SCRATCH_BYTES];

static std::mutex g_noalloc_mutex;
static void* g_noalloc_addr[64] = {};
static unsigned long long g_noalloc_ctx[64] = {};  // context the address was looked up in

// Unique id of the calling thread's current CUDA context (cuCtxGetId, through
// the runtime's driver entry points, so the library needs no -lcuda).  A
// device reset destroys the device's primary context and the next one gets a
// new id, which is how a cached symbol address is known to be stale.
static bool current_context_id(unsigned long long* id) {
    typedef int (*GetCurrent)(void**);
    typedef int (*GetId)(void*, unsigned long long*);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static bool looked = false;
    if (!looked) {
        looked = true;
        cudaDriverEntryPointQueryResult q1, q2;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", (void**)&get_current, cudaEnableDefault, &q1) != cudaSuccess ||
            q1 != cudaDriverEntryPointSuccess)
            get_current = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", (void**)&get_id, cudaEnableDefault, &q2) != cudaSuccess ||
            q2 != cudaDriverEntryPointSuccess)
            get_id = nullptr;
    }
    void* ctx = nullptr;
    if (!get_current || !get_id || get_current(&ctx) != 0 || !ctx) return false;
    return get_id(ctx, id) == 0;
}
}  // namespace ys

extern "C" ys_status ys_radix_sort_pairs_noalloc(uint32_t* d_keys, uint32_t* d_vals, uint32_t n, void* stream) {
    using namespace ys;
    if (n > NOALLOC_MAX_PAIRS)
        return fail(YS_ERR_CAPACITY, "ys_radix_sort_pairs_noalloc: n = " + std::to_string(n) +
                                         " exceeds the fixed scratch capacity of " +
                                         std::to_string(NOALLOC_MAX_PAIRS) + " pairs");
    if (n > 1 && (!d_keys || !d_vals)) return fail(YS_ERR_BAD_ARG, "ys_radix_sort_pairs_noalloc: null array");
    if (n <= 1) return YS_OK;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(YS_ERR_CUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
    if (dev < 0 || dev >= 64) return fail(YS_ERR_BAD_ARG, "device index out of range");
    void* scratch = nullptr;
    {
        // first call on this device (or in a new context of it, after a
        // device reset): look up the device address of the array (its
        // host-side name is only a stand-in and must never reach a kernel)
        std::lock_guard<std::mutex> lock(g_noalloc_mutex);
        unsigned long long ctx = 0;
        const bool known = current_context_id(&ctx);
        if (!g_noalloc_addr[dev] || (known && ctx != g_noalloc_ctx[dev])) {
            void* p = nullptr;
            e = cudaGetSymbolAddress(&p, g_noalloc_sort_scratch);
            if (e != cudaSuccess)
                return fail(YS_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
            g_noalloc_addr[dev] = p;
            g_noalloc_ctx[dev] = current_context_id(&ctx) ? ctx : 0;
        }
        scratch = g_noalloc_addr[dev];
    }
    // The sort clears the words it reads and writes the ping-pong halves before
    // it reads them, so nothing left by an earlier call matters.  4 passes end
    // in the caller's arrays.  Large tiles at every size: their words fit.
    e = sort_in(d_keys, d_vals, n, scratch, 0, 32, true, (cudaStream_t)stream);
    if (e != cudaSuccess) return fail(YS_ERR_CUDA, std::string("radix sort: ") + cudaGetErrorString(e));
    return YS_OK;
}
