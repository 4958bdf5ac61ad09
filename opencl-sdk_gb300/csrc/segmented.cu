// Batched segmented sort: every segment [offsets[i], offsets[i+1]) of a key
// (+ value) array is sorted independently and stably, for many segments of
// uneven length in one call whose launch sequence is fixed (every decision is
// made on the device, so the call can be captured in a CUDA graph).
//
// No reference counterpart: the reference sorts one array per call
// (detail::radix_sort, lib/src/Compute/Algorithm.cpp:453-527); sorting a batch
// there means one call per array. The semantics per segment are the same as
// that sort's: stable, the order-preserving key bijection of Algorithm.cpp:
// 459-469, optional 32-bit values moved alongside.
//
// Size classes (decided by k_seg_classify):
//   * tiny/small (<= WARP_CAP): one warp per segment, stable LSD radix sort in
//     warp-private shared memory over the digit positions that vary inside the
//     segment only;
//   * medium (<= cta_cap): one CTA per segment, the leading digits sorted and
//     the rest repaired (tile_sort.cuh), in three classes by length;
//   * large: the tiles of all large segments form one sequence, and
//     per-segment digit histograms come from one read of the keys. A segment
//     whose highest varying digit splits it into small enough buckets takes
//     the MSD route: one pass on that digit, then one-CTA sorts of ranges of
//     buckets. The others take a batched onesweep over every digit, whose
//     decoupled look-back stops at the first tile of its segment.
// The small/medium path and the large path are independent; where both have much to
// do they run on two streams that fork from and join back to the context's stream.
#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "device_common.cuh"
#include "runtime.hpp"
#include "segmented.hpp"
#include "sort_internal.hpp"
#include "tile_sort.cuh"

namespace gbc {
namespace seg {

using dev::FULL_MASK;
using onesweep::RADIX;
using onesweep::RING_TILES;

constexpr uint64_t FLAG_AGG = 1, FLAG_PRE = 2;
constexpr uint64_t TAG_MASK = (1ull << 30) - 1;
constexpr int WARP_CAP = 256;  // keys a warp sorts on its own
constexpr int SMALL_THREADS = 256;
constexpr int SMALL_WARPS = SMALL_THREADS / 32;

template <typename K> struct Traits;
template <> struct Traits<uint32_t> {
    static constexpr int PASSES = 4;
};
template <> struct Traits<uint64_t> {
    static constexpr int PASSES = 8;
};

// One-CTA sorts by length: up to 4,096, 8,192 and the type's largest capacity
// (16,384 u32 keys; 10,240 u32 pairs or u64 keys, whose registers hold no
// more; 8,192 u64 pairs, which leaves their last class empty).
constexpr int CTA_CLASSES = 3;
constexpr uint32_t CLASS0_CAP = 4096, CLASS1_CAP = 8192;
template <typename K, bool HAS_V> constexpr uint32_t max_cta_cap()
{
    return sizeof(K) == 4 ? (HAS_V ? 10240u : 16384u) : (HAS_V ? 8192u : 10240u);
}
__device__ __forceinline__ int cta_class(uint32_t len)
{
    return len <= CLASS0_CAP ? 0 : len <= CLASS1_CAP ? 1 : 2;
}

// The MSD route joins neighbouring buckets of a segment whose first keys lie
// in the same window of this many keys (a bucket of a few dozen keys is not
// worth a CTA, and a range of neighbouring buckets is as good to sort).
constexpr uint32_t SUB_WINDOW = 2048;

__device__ __forceinline__ uint64_t pack_status(uint64_t flag, uint64_t seq, uint32_t v)
{
    return (flag << 62) | ((seq & TAG_MASK) << 32) | v;
}

//! Per-call control block (zeroed before each call).
struct SegControl {
    uint32_t n_warp, n_cta[CTA_CLASSES], n_large;  // list lengths
    uint32_t large_tiles;                          // tiles of all large segments
    uint32_t lsd_tiles;                            // tiles of those not on the MSD route
    uint32_t rest_tiles;                           // tiles of those counted a second time
    uint32_t warp_next, cta_next[CTA_CLASSES];     // work queue heads
    uint32_t tile_ctr[8];
    uint32_t msd_tile_ctr;
    uint32_t n_sub_warp, n_sub_cta[CTA_CLASSES];  // sub-bucket list lengths (MSD route)
    uint32_t sub_warp_next, sub_cta_next[CTA_CLASSES];
};

template <typename K> struct SegArgs {
    const K* in_k;
    K* out_k;
    K* alt_k;
    const uint32_t* in_v;
    uint32_t* out_v;
    uint32_t* alt_v;
    const uint32_t* off;
    const uint8_t* skip;  // per segment: nonzero = already in order (in-place calls)
    uint32_t nseg;
    uint32_t cta_cap;
    dev::KeyXform<K> xf;
    SegControl* ctl;
    uint32_t* warp_list;
    uint32_t* cta_list;     // nseg entries per class
    uint32_t* large_list;
    uint32_t* tile_begin;   // per large segment: its first tile
    uint32_t* tile_seg;     // large tile -> index into large_list
    uint32_t* lsd_begin;    // the same for the segments that take the LSD passes
    uint32_t* lsd_seg;      // (tile_begin and tile_seg themselves without the MSD route)
    // Counting in two steps (null: all digits at once): the one digit position
    // counted first (or ALL_DIGITS), the bits that differ inside the segment, and
    // the tile sequence of the segments whose other digits are counted after all
    uint8_t* guess;
    unsigned long long* vary;
    uint32_t* rest_begin;
    uint32_t* rest_seg;
    uint32_t* seg_hist;     // [large][PASSES][256]: bin start (absolute) per pass
    uint32_t max_large;
    uint32_t max_tiles;
    uint64_t* ring;
    uint64_t seq0;
    int* err;
    // MSD route of large segments: route[j] = the digit position of large
    // segment j's single pass, or NO_ROUTE for the full LSD passes; its
    // sub-buckets (begin, end pairs) are finished from alt into out by the
    // warp (<= WARP_CAP) and CTA (<= sub_cap) sorts.
    uint8_t* route;
    uint32_t* sub_lists;  // 2 x max_sub (begin, end) pairs, see sub_entry
    uint32_t max_sub;
    uint32_t sub_cap;
};

// The (begin, end) pair at position i of a sub-bucket list: the warp class
// (cls = -1) and class 0 share one array, classes 1 and 2 another, each pair
// growing from both ends (there are at most max_sub sub-buckets in all).
template <typename K> __device__ __forceinline__ uint2* sub_entry(const SegArgs<K>& a, int cls, uint32_t i)
{
    uint2* base = reinterpret_cast<uint2*>(a.sub_lists) + (cls >= 1 ? a.max_sub : 0u);
    return cls == -1 || cls == 1 ? base + i : base + (a.max_sub - 1 - i);
}

constexpr uint8_t NO_ROUTE = 0xFF, REST = 0xFE;  // REST: known after the second count
constexpr uint8_t ALL_DIGITS = 0xFF;
enum : int { COUNT_ALL, COUNT_FIRST, COUNT_REST };  // steps of counting and routing

// ---------------------------------------------------------------------------
// Classification
// ---------------------------------------------------------------------------
template <typename K, int TILE> __device__ __forceinline__ void seg_classify(const SegArgs<K>& a)
{
    // whole warps take every step, so that a class's members in a warp share
    // one addition to its counter
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < a.nseg; i0 += stride) {
        const uint32_t i = i0 + lane;
        uint32_t len = 0;
        if (i < a.nseg) {
            const uint32_t b = a.off[i], e = a.off[i + 1];
            if (e < b) dev::raise_error(a.err, dev::ERR_BAD_SEGMENT);
            else if (a.skip == nullptr || a.skip[i] == 0) len = e - b;
        }
        // -1: nothing to do; 0: a warp's; 1 ..: the one-CTA classes
        const int cls = len == 0 ? -1 : len <= WARP_CAP ? 0 : len <= a.cta_cap ? 1 + cta_class(len) : 1 + CTA_CLASSES;
#pragma unroll
        for (int c = 0; c <= CTA_CLASSES; ++c) {
            const uint32_t members = __ballot_sync(FULL_MASK, cls == c);
            if (members == 0) continue;
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(c == 0 ? &a.ctl->n_warp : &a.ctl->n_cta[c - 1], (uint32_t)__popc(members));
            at = __shfl_sync(FULL_MASK, at, 0) + __popc(members & dev::lanemask_lt());
            if (cls == c) (c == 0 ? a.warp_list : a.cta_list + (std::size_t)(c - 1) * a.nseg)[at] = i;
        }
        if (cls == 1 + CTA_CLASSES) {
            const uint32_t j = atomicAdd(&a.ctl->n_large, 1u);
            if (j < a.max_large) {
                a.large_list[j] = i;
                // the segment's stretch of the tile sequence; the sequence's
                // order among segments does not matter
                a.tile_begin[j] = atomicAdd(&a.ctl->large_tiles, (len + TILE - 1) / TILE);
            } else {
                dev::raise_error(a.err, dev::ERR_BAD_SEGMENT);
            }
        }
    }
}

template <typename K, int TILE> __global__ void k_seg_classify(SegArgs<K> a)
{
    dev::chain();
    seg_classify<K, TILE>(a);
}

// The tile -> segment map (a warp of the first `ctas` CTAs per large segment),
// and zeros in the histogram rows of the large segments present.
template <typename K, int TILE> __device__ __forceinline__ void seg_large_plan(const SegArgs<K>& a, uint32_t ctas)
{
    constexpr int P = Traits<K>::PASSES;
    const uint32_t nl = min(a.ctl->n_large, a.max_large);
    const int lane = threadIdx.x & 31;
    const uint32_t warps = ctas * (blockDim.x / 32);
    for (uint32_t j = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); j < nl; j += warps) {
        const uint32_t s = a.large_list[j];
        const uint32_t t0 = a.tile_begin[j], t1 = min(t0 + (a.off[s + 1] - a.off[s] + TILE - 1) / TILE, a.max_tiles);
        for (uint32_t t = t0 + lane; t < t1; t += 32) a.tile_seg[t] = j;
    }
    const std::size_t words = (std::size_t)nl * P * RADIX;
    const std::size_t stride = (std::size_t)ctas * blockDim.x;
    for (std::size_t i = (std::size_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += stride) a.seg_hist[i] = 0;
}

// The digit position that a large segment's MSD pass will probably use: the
// highest one that varies among 512 of its keys (16 rows of 32 neighbours),
// unless its largest bin is then surely too large for that route. A wrong
// guess costs a second count, nothing else.
template <typename K> __device__ __forceinline__ void seg_guess(const SegArgs<K>& a)
{
    constexpr int ROWS = 16, WARPS = 8;
    __shared__ uint32_t s_count[WARPS][RADIX];
    const uint32_t nl = min(a.ctl->n_large, a.max_large);
    const int lane = threadIdx.x & 31;
    uint32_t* count = s_count[threadIdx.x >> 5];
    for (uint32_t j = blockIdx.x * WARPS + (threadIdx.x >> 5); j < nl; j += gridDim.x * WARPS) {
        const uint32_t s = a.large_list[j];
        const uint32_t b = a.off[s], len = a.off[s + 1] - b;
        K k[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) k[r] = a.in_k[b + min(len / ROWS * r + lane, len - 1)];
        unsigned long long v = 0;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            k[r] = a.xf(k[r]);
            v |= k[r] ^ k[0];
        }
        v |= k[0] ^ __shfl_sync(FULL_MASK, k[0], 0);
        v = (unsigned long long)__reduce_or_sync(FULL_MASK, (uint32_t)(v >> 32)) << 32 |
            __reduce_or_sync(FULL_MASK, (uint32_t)v);
        int top = v == 0 ? -1 : (63 - __clzll((long long)v)) / 8;
        if (top >= 0) {
            for (int d = lane; d < RADIX; d += 32) count[d] = 0;
            __syncwarp();
#pragma unroll
            for (int r = 0; r < ROWS; ++r) atomicAdd(&count[(uint32_t)(k[r] >> (8 * top)) & 0xFFu], 1u);
            __syncwarp();
            uint32_t m = 0;
            for (int d = lane; d < RADIX; d += 32) m = max(m, count[d]);
            m = __reduce_max_sync(FULL_MASK, m);
            // three deviations below the estimate; and evenly filled bins
            const float least = ((float)m - 3.0f * sqrtf((float)m)) * (1.0f / (32 * ROWS)) * (float)len;
            if (least > (float)min(a.sub_cap, sizeof(K) == 4 ? a.sub_cap : len / 2) || len / RADIX + SUB_WINDOW > a.sub_cap) top = -1;
            __syncwarp();
        }
        if (lane == 0) {
            a.guess[j] = top < 0 ? ALL_DIGITS : (uint8_t)top;
            a.vary[j] = 0;
        }
    }
}

template <typename K, int TILE> __global__ void __launch_bounds__(256) k_seg_large_plan(SegArgs<K> a)
{
    seg_large_plan<K, TILE>(a, gridDim.x);
    if (a.guess != nullptr) seg_guess<K>(a);
}

// ---------------------------------------------------------------------------
// Shared-memory LSD sort of one segment by a warp. Stable: items are ranked in
// index order (row, lane) and scattered by digit.
//
// Ranking is by shared-memory peer masks, as in the digit pass: each lane ORs
// its bit into its digit's mask word (256 words in `wm`, all zero between
// rows), reads the word back (its peers) and the count of the digit so far;
// the lowest peer stores the new count and clears the mask.
// (__match_any_sync ranked the same rows about 1.7x slower on this GPU.)
// ---------------------------------------------------------------------------
template <typename K, bool HAS_V>
__device__ void warp_sort(K* k0, K* k1, uint32_t* v0, uint32_t* v1, uint32_t* rd, uint32_t* wh, uint32_t* wm, uint32_t len,
                          dev::KeyXform<K> xf, int lane, bool& in_k1)
{
    constexpr int P = Traits<K>::PASSES;
    // Which digit positions vary inside the segment.
    K diff = 0;
    const K first = xf(k0[0]);
    for (uint32_t i = lane; i < len; i += 32) diff |= xf(k0[i]) ^ first;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) diff |= __shfl_xor_sync(FULL_MASK, diff, o);
    const uint32_t rows = (len + 31) / 32;
    in_k1 = false;
    for (int p = 0; p < P; ++p) {
        if ((((uint64_t)diff >> (8 * p)) & 0xFF) == 0) continue;
        const int shift = 8 * p;
        for (int i = lane; i < RADIX; i += 32) wh[i] = 0;
        __syncwarp();
        const uint32_t lt = dev::lanemask_lt();
        for (uint32_t r = 0; r < rows; ++r) {
            const uint32_t idx = r * 32 + lane;
            const bool valid = idx < len;
            // padding ranks in bin 255 (counted there, never placed)
            const uint32_t d = valid ? (uint32_t)(xf(k0[idx]) >> shift) & 0xFFu : 0xFFu;
            atomicOr(&wm[d], 1u << lane);
            __syncwarp();
            const uint32_t peers = wm[d];
            const uint32_t before = wh[d];
            __syncwarp();
            const uint32_t lower = peers & lt;
            if (lower == 0) {
                wh[d] = before + __popc(peers);
                wm[d] = 0;
            }
            __syncwarp();
            if (valid) rd[idx] = ((before + __popc(lower)) << 8) | d;
        }
        __syncwarp();
        // digit starts
        uint32_t c[8], s = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            c[q] = wh[lane * 8 + q];
            s += c[q];
        }
        uint32_t run = dev::warp_inclusive_scan(s, [](uint32_t x, uint32_t y) { return x + y; }) - s;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            wh[lane * 8 + q] = run;
            run += c[q];
        }
        __syncwarp();
        for (uint32_t r = 0; r < rows; ++r) {
            const uint32_t idx = r * 32 + lane;
            if (idx < len) {
                const uint32_t x = rd[idx];
                const uint32_t pos = wh[x & 0xFF] + (x >> 8);
                k1[pos] = k0[idx];
                if (HAS_V) v1[pos] = v0[idx];
            }
        }
        __syncwarp();
        K* tk = k0;
        k0 = k1;
        k1 = tk;
        uint32_t* tv = v0;
        v0 = v1;
        v1 = tv;
        in_k1 = !in_k1;
    }
}

// SUB: the MSD route's sub-buckets (begin, end pairs, read from alt) instead
// of whole segments (read from the input).
template <typename K, bool HAS_V, bool SUB> __device__ __forceinline__ void seg_small_warp(const SegArgs<K>& a)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr std::size_t per_warp =
        2 * WARP_CAP * sizeof(K) + (HAS_V ? 2 * WARP_CAP * 4 : 0) + WARP_CAP * 4 + 2 * RADIX * 4;
    unsigned char* base = smem + warp * per_warp;
    K* k0 = reinterpret_cast<K*>(base);
    K* k1 = k0 + WARP_CAP;
    uint32_t* v0 = reinterpret_cast<uint32_t*>(k1 + WARP_CAP);
    uint32_t* v1 = v0 + (HAS_V ? WARP_CAP : 0);
    uint32_t* rd = v1 + (HAS_V ? WARP_CAP : 0);
    uint32_t* hist = rd + WARP_CAP;
    uint32_t* masks = hist + RADIX;
    for (int i = lane; i < RADIX; i += 32) masks[i] = 0;
    __syncwarp();
    const uint32_t total = SUB ? min(a.ctl->n_sub_warp, a.max_sub) : a.ctl->n_warp;
    const K* src_k = SUB ? a.alt_k : a.in_k;
    const uint32_t* src_v = SUB ? a.alt_v : a.in_v;
    for (;;) {
        uint32_t w = 0;
        if (lane == 0) w = atomicAdd(SUB ? &a.ctl->sub_warp_next : &a.ctl->warp_next, 1u);
        w = __shfl_sync(FULL_MASK, w, 0);
        if (w >= total) break;
        uint32_t b, len;
        if (SUB) {
            const uint2 r = *sub_entry(a, -1, w);
            b = r.x;
            len = r.y - r.x;
        } else {
            const uint32_t s = a.warp_list[w];
            b = a.off[s];
            len = a.off[s + 1] - b;
        }
        for (uint32_t i = lane; i < len; i += 32) {
            k0[i] = src_k[b + i];
            if (HAS_V) v0[i] = src_v[b + i];
        }
        __syncwarp();
        bool flipped = false;
        if (len > 1) warp_sort<K, HAS_V>(k0, k1, v0, v1, rd, hist, masks, len, a.xf, lane, flipped);
        const K* rk = flipped ? k1 : k0;
        const uint32_t* rv = flipped ? v1 : v0;
        for (uint32_t i = lane; i < len; i += 32) {
            a.out_k[b + i] = rk[i];
            if (HAS_V) a.out_v[b + i] = rv[i];
        }
        __syncwarp();
    }
}

template <typename K, bool HAS_V, bool SUB>
__global__ void __launch_bounds__(SMALL_THREADS) k_seg_small_warp(SegArgs<K> a)
{
    dev::chain();
    seg_small_warp<K, HAS_V, SUB>(a);
}

// The one-CTA sorts of classes cls to last (tile_sort.cuh): persistent CTAs
// take their segments (sub: the MSD route's sub-buckets) one at a time. Bound by
// shared-memory accesses (about 27 wavefronts per 32 pairs and digit pass), so
// what counts is the number of passes and the warps in flight: the sort of
// every digit in two shared-memory copies, one CTA of 256 threads per SM at
// the largest capacity, took 10.3 ms for 200,000 lognormal segments of u64
// pairs (median 256), this one 4.1 ms, each beside its large-segment path.
template <typename K, bool HAS_V, int THREADS, int ITEMS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) k_seg_tile(SegArgs<K> a, int cls, int last, bool sub)
{
    dev::chain();
    using S = tile::Sorter<K, HAS_V, THREADS, ITEMS>;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ tile::Scratch<THREADS> scratch;
    __shared__ uint32_t s_work;
    S st(smem, scratch);
    const K* src_k = sub ? a.alt_k : a.in_k;
    const uint32_t* src_v = sub ? a.alt_v : a.in_v;
    for (;;) {
        if (threadIdx.x == 0) s_work = atomicAdd(sub ? &a.ctl->sub_cta_next[cls] : &a.ctl->cta_next[cls], 1u);
        __syncthreads();
        const uint32_t w = s_work;
        if (w >= (sub ? min(a.ctl->n_sub_cta[cls], a.max_sub) : a.ctl->n_cta[cls])) {
            if (++cls > last) break;
            __syncthreads();  // every thread has read s_work
            continue;
        }
        uint32_t b, len;
        if (sub) {
            const uint2 r = *sub_entry(a, cls, w);
            b = r.x;
            len = r.y - r.x;
        } else {
            const uint32_t s = a.cta_list[(std::size_t)cls * a.nseg + w];
            b = a.off[s];
            len = a.off[s + 1] - b;
        }
        if (len > (uint32_t)S::CAP) {  // the classes end at the capacities
            if (threadIdx.x == 0) dev::raise_error(a.err, dev::ERR_MISPLACED);
            __syncthreads();
            continue;
        }
        st.len = len;
        st.rows = (len + THREADS - 1) / THREADS;
        const uint32_t i0 = st.first_index();
        K key[ITEMS];
        uint32_t val[HAS_V ? ITEMS : 1];
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const uint32_t idx = i0 + i * 16;
            const bool in = i < (int)st.rows && idx < len;
            key[i] = in ? src_k[b + idx] : K(0);
            if (HAS_V) val[i] = in ? src_v[b + idx] : 0u;
        }
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) key[i] = a.xf(key[i]);
        if (!st.sort(key, val) && threadIdx.x == 0) dev::raise_error(a.err, dev::ERR_MISPLACED);
        for (uint32_t i = threadIdx.x; i < len; i += THREADS) {
            a.out_k[b + i] = tile::undo_xform(a.xf, st.keys[i]);
            if (HAS_V) a.out_v[b + i] = st.vals[i];
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Large segments: per-segment digit histograms -> absolute bin starts, over
// the large-segment tile sequence that the passes use (so a long segment is
// spread over many CTAs): count runs of HIST_TILES tiles in shared memory and
// add the counts to the segment's row whenever the segment changes or the run
// ends; turn every row into absolute bin starts.
//
// Shared-memory additions bound the count, one per key and digit. The MSD
// route needs one digit, so batches of more than TWO_STEP_KEYS count in two steps:
// COUNT_FIRST the digit that a sample points to and which bits differ at all
// (which tells whether the guess was right), COUNT_REST every digit of the
// segments that cannot take the route with it.
// ---------------------------------------------------------------------------
constexpr uint32_t HIST_TILES = 8;

template <typename K, int TILE, int STEP>
__device__ __forceinline__ void seg_large_count(const SegArgs<K>& a, uint32_t ctas)
{
    constexpr int P = Traits<K>::PASSES;
    constexpr int BATCH = 8;  // keys in flight per thread
    __shared__ uint32_t sh[2][P * RADIX];  // two copies (warp parity)
    uint32_t* my = sh[(threadIdx.x >> 5) & 1];
    const uint32_t total = min(STEP == COUNT_REST ? a.ctl->rest_tiles : a.ctl->large_tiles, a.max_tiles);
    const uint32_t* tile_seg = STEP == COUNT_REST ? a.rest_seg : a.tile_seg;
    const uint32_t* tile_begin = STEP == COUNT_REST ? a.rest_begin : a.tile_begin;
    const uint32_t runs = (total + HIST_TILES - 1) / HIST_TILES;
    unsigned long long vary = 0;
    auto flush = [&](uint32_t j) {  // adds the counts to row j and clears them
        __syncthreads();
        uint32_t* row = a.seg_hist + (std::size_t)j * P * RADIX;
        const uint32_t g = STEP == COUNT_FIRST ? a.guess[j] : ALL_DIGITS;
        if (g != ALL_DIGITS) {
            const uint32_t hi = sizeof(K) == 8 ? __reduce_or_sync(FULL_MASK, (uint32_t)(vary >> 32)) : 0u;
            const uint32_t lo = __reduce_or_sync(FULL_MASK, (uint32_t)vary);
            if ((threadIdx.x & 31) == 0 && (hi | lo) != 0) atomicOr(&a.vary[j], (unsigned long long)hi << 32 | lo);
            vary = 0;
        }
        const int first = g == ALL_DIGITS ? 0 : (int)g * RADIX, end = g == ALL_DIGITS ? P * RADIX : first + RADIX;
        for (int i = first + threadIdx.x; i < end; i += 256) {
            const uint32_t v = sh[0][i] + sh[1][i];
            if (v != 0) atomicAdd(&row[i], v);
            sh[0][i] = 0;
            sh[1][i] = 0;
        }
        __syncthreads();
    };
    for (int i = threadIdx.x; i < 2 * P * RADIX; i += 256) (&sh[0][0])[i] = 0;
    __syncthreads();
    for (uint32_t r = blockIdx.x; r < runs; r += ctas) {
        const uint32_t t0 = r * HIST_TILES, t1 = min(total, t0 + HIST_TILES);
        uint32_t j = tile_seg[t0];
        for (uint32_t t = t0; t < t1; ++t) {
            const uint32_t jt = tile_seg[t];  // the same for every thread
            if (jt != j) {
                flush(j);
                j = jt;
            }
            const uint32_t s = a.large_list[jt];
            const uint32_t b = a.off[s] + (t - tile_begin[jt]) * TILE;
            const uint32_t e = min(a.off[s + 1], b + TILE);
            const uint32_t g = STEP == COUNT_FIRST ? a.guess[jt] : ALL_DIGITS;
            const K x0 = g != ALL_DIGITS ? a.xf(a.in_k[a.off[s]]) : K(0);
            for (uint32_t i0 = b; i0 < e; i0 += 256 * BATCH) {
                K k[BATCH];
#pragma unroll
                for (int q = 0; q < BATCH; ++q) {
                    const uint32_t i = i0 + q * 256 + threadIdx.x;
                    k[q] = i < e ? a.in_k[i] : K(0);
                }
#pragma unroll
                for (int q = 0; q < BATCH; ++q) {
                    if (i0 + q * 256 + threadIdx.x >= e) break;
                    const K x = a.xf(k[q]);
                    if (STEP == COUNT_FIRST && g != ALL_DIGITS) {
                        atomicAdd(&my[g * RADIX + ((uint32_t)(x >> ((8 * g) & (8 * P - 1))) & 0xFFu)], 1u);
                        vary |= x ^ x0;
                        continue;
                    }
#pragma unroll
                    for (int p = 0; p < P; ++p) atomicAdd(&my[p * RADIX + (uint32_t)((x >> (8 * p)) & 0xFF)], 1u);
                }
            }
        }
        flush(j);
    }
}

template <typename K, int TILE, int STEP> __global__ void __launch_bounds__(256) k_seg_large_count(SegArgs<K> a)
{
    dev::chain();
    seg_large_count<K, TILE, STEP>(a, gridDim.x);
}


// Per large segment (one CTA, thread d = bin d): every digit's counts become
// absolute bin starts. With the MSD route: then the highest digit position
// that varies inside the segment (its bins are not all in one) and, when every
// bin there leaves room for a window in sub_cap, the MSD route: one
// pass on that digit partitions the segment into its bins (stable), and
// ranges of neighbouring bins become sub-buckets for the warp and CTA sorts.
// For 64-bit keys a bin with more than half of the segment is as long a sort as
// all of it (segments of 12,000 u64 keys that are the AND of four words: 894 us by
// that route, 819 by the passes; 100 of 10,000: 395 and 261). 32-bit keys take the
// route all the same (the learned sort's oversized buckets, 2^28 floats: 6.23 ms for
// 6.37);
// else the full LSD passes, over tiles appended to their own sequence.
// COUNT_FIRST: a segment of which one digit was counted takes the MSD route
// with it or is put off to COUNT_REST, with its counts cleared.
template <typename K, int TILE, int STEP>
__device__ __forceinline__ void seg_route(const SegArgs<K>& a, bool with_msd, uint32_t ctas)
{
    constexpr int P = Traits<K>::PASSES;
    __shared__ uint32_t s_max[8];
    __shared__ uint32_t s_scratch[8];
    __shared__ int s_top;
    __shared__ uint32_t s_first;
    const uint32_t nl = min(a.ctl->n_large, a.max_large);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t j = blockIdx.x; j < nl; j += ctas) {
        const uint32_t s = a.large_list[j];
        const uint32_t segb = a.off[s], sege = a.off[s + 1], len = sege - segb;
        if (STEP == COUNT_REST && a.route[j] != REST) continue;
        const int one = STEP == COUNT_FIRST && a.guess[j] != ALL_DIGITS ? a.guess[j] : -1;  // the only row that is counted
        for (int p = one < 0 ? 0 : one; p < (one < 0 ? P : one + 1); ++p) {
            uint32_t* row = a.seg_hist + ((std::size_t)j * P + p) * RADIX;
            const uint32_t ex = dev::bins_exclusive_sum(row[threadIdx.x], s_scratch);
            row[threadIdx.x] = segb + ex;
        }
        if (!with_msd) continue;
        __syncthreads();
        auto bin_size = [&](int p, uint32_t d) {
            const uint32_t* row = a.seg_hist + ((size_t)j * P + p) * RADIX;
            return (d == RADIX - 1 ? sege : row[d + 1]) - row[d];
        };
        if (threadIdx.x == 0) s_top = -1;
        __syncthreads();
        if (one >= 0) {
            const unsigned long long v = a.vary[j];
            if (threadIdx.x == 0) s_top = v == 0 ? -1 : (63 - __clzll((long long)v)) / 8;
        }
        for (int p = one < 0 ? P - 1 : -1; p >= 0; --p) {
            // a position varies when no bin holds the whole segment
            const bool whole = bin_size(p, threadIdx.x) == len;
            if (__syncthreads_or(whole) == 0) {
                if (threadIdx.x == 0) s_top = p;
                break;
            }
        }
        __syncthreads();
        const int top = s_top;
        uint32_t size = top >= 0 && (one < 0 || top == one) ? bin_size(top, threadIdx.x) : len;
        uint32_t m = size;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(FULL_MASK, m, o));
        if (lane == 0) s_max[warp] = m;
        __syncthreads();
        uint32_t biggest = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) biggest = max(biggest, s_max[w]);
        // room for a window's keys and its last bucket
        const bool msd =
            top >= 0 && (one < 0 || top == one) && biggest + SUB_WINDOW <= a.sub_cap && (sizeof(K) == 4 || biggest <= len / 2);
        if (threadIdx.x == 0) a.route[j] = msd ? (uint8_t)top : (uint8_t)(one < 0 ? NO_ROUTE : REST);
        if (msd) {
            const uint32_t* row = a.seg_hist + ((size_t)j * P + top) * RADIX;
            const uint32_t d = threadIdx.x;
            auto window = [&](uint32_t q) { return (row[q] - segb) / SUB_WINDOW; };
            if (d == 0 || window(d) != window(d - 1)) {  // first bucket of its window: the range up to the next one's
                uint32_t q = d + 1;
                while (q < RADIX && window(q) == window(d)) ++q;
                const uint32_t b = row[d], e = q < RADIX ? row[q] : sege;
                if (e > b) {  // a range of one key goes to the warp sort, which copies it
                    const int cls = e - b <= (uint32_t)WARP_CAP ? -1 : cta_class(e - b);
                    const uint32_t at = atomicAdd(cls < 0 ? &a.ctl->n_sub_warp : &a.ctl->n_sub_cta[cls], 1u);
                    if (at < a.max_sub) *sub_entry(a, cls, at) = make_uint2(b, e);
                    else dev::raise_error(a.err, dev::ERR_BAD_SEGMENT);
                }
            }
        } else {
            const uint32_t tiles = (len + TILE - 1) / TILE;
            const bool rest = one >= 0;
            if (threadIdx.x == 0)
                (rest ? a.rest_begin : a.lsd_begin)[j] = s_first =
                    atomicAdd(rest ? &a.ctl->rest_tiles : &a.ctl->lsd_tiles, tiles);
            __syncthreads();
            for (uint32_t t = threadIdx.x; t < tiles; t += blockDim.x)
                if (s_first + t < a.max_tiles) (rest ? a.rest_seg : a.lsd_seg)[s_first + t] = j;
            if (rest) a.seg_hist[((std::size_t)j * P + max(one, 0)) * RADIX + threadIdx.x] = 0;
        }
        __syncthreads();
    }
}

template <typename K, int TILE, int STEP> __global__ void __launch_bounds__(256) k_seg_route(SegArgs<K> a, bool with_msd)
{
    dev::chain();
    seg_route<K, TILE, STEP>(a, with_msd, gridDim.x);
}


// One digit pass over every large segment's tiles (cf. onesweep::k_pass2:
// shared-memory peer-mask ranking, place offsets folded into the per-warp
// counts, a look-back reading LBW predecessors per round trip, which stops at
// the segment's first tile (it publishes an inclusive count), an L2 prefetch
// of the tile a grid ahead and an unrolled write-out of full tiles).
constexpr int LARGE_PAD = 1;  // words between the half-warp count arrays of the large pass

//
// MSD: the one pass of the segments on the MSD route, each on its own digit
// position, over the sequence of all large segments' tiles; else LSD pass
// `slot` over the tiles of the segments that take those. Returns at once when
// its kind has no segment.
template <typename K, bool HAS_V, int THREADS, int ITEMS, int LBW, bool MSD>
__device__ __forceinline__ void seg_large_pass(const SegArgs<K>& a, int slot, bool with_msd, uint32_t ctas)
{
    constexpr int P = Traits<K>::PASSES;
    constexpr int WARPS = THREADS / 32;
    constexpr int TILE = THREADS * ITEMS;
    const uint32_t num_tiles = min(MSD || !with_msd ? a.ctl->large_tiles : a.ctl->lsd_tiles, a.max_tiles);
    if (num_tiles == 0 || (MSD && a.ctl->lsd_tiles == a.ctl->large_tiles)) return;  // no segment of this kind
    const uint32_t* tile_seg = MSD ? a.tile_seg : a.lsd_seg;
    const uint32_t* tile_begin = MSD ? a.tile_begin : a.lsd_begin;
    uint32_t* tile_ctr = MSD ? &a.ctl->msd_tile_ctr : &a.ctl->tile_ctr[slot];
    // pass s writes out when (P - 1 - s) is even; P is even, so pass 0 reads
    // the input and writes the scratch buffer.
    // The MSD pass reads the input and writes the scratch buffer, from which
    // its sub-buckets are finished.
    const bool dst_out = !MSD && ((P - 1 - slot) & 1) == 0;
    K* dst_k = dst_out ? a.out_k : a.alt_k;
    uint32_t* dst_v = dst_out ? a.out_v : a.alt_v;
    const K* src_k = MSD || slot == 0 ? a.in_k : (dst_out ? a.alt_k : a.out_k);
    const uint32_t* src_v = MSD || slot == 0 ? a.in_v : (dst_out ? a.alt_v : a.out_v);
    const bool aligned_src =
        ((reinterpret_cast<uintptr_t>(src_k) | (HAS_V ? reinterpret_cast<uintptr_t>(src_v) : 0)) & 15) == 0;

    extern __shared__ __align__(16) unsigned char smem[];
    // Keys are ranked by half-warps (rows of 16, each half-warp a contiguous
    // run of the tile): one word per half-warp and digit holds the count
    // (high 16 bits) and the current row's peer mask (low 16 bits).
    // A half-warp's words sit LARGE_PAD banks from its partner's, so equal
    // digits in the two halves of a row do not meet in one bank.
    constexpr int GROUPS = 2 * WARPS, GSTRIDE = RADIX + LARGE_PAD;
    static_assert(16 * ITEMS < (1 << 16), "half-warp counts are 16-bit");
    uint32_t* warp_hist = reinterpret_cast<uint32_t*>(smem);  // GROUPS x GSTRIDE: counts, then place offsets
    K* s_keys = reinterpret_cast<K*>(warp_hist + GROUPS * GSTRIDE);
    uint32_t* s_vals = reinterpret_cast<uint32_t*>(s_keys + TILE);
    __shared__ uint32_t s_bin_off[RADIX], s_local[RADIX];
    __shared__ uint32_t s_scratch[8];
    __shared__ uint32_t s_tile;
    __shared__ int s_abort;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int grp = 2 * warp + (lane >> 4), gl = lane & 15;
    if (tid == 0) s_abort = 0;
    // MSD: after the P LSD passes' sequence numbers
    const uint64_t seq0 = a.seq0 + (uint64_t)(MSD ? P : slot) * a.max_tiles;
    int shift = 8 * slot;
    auto digit = [&](K k) -> uint32_t { return (uint32_t)(a.xf(k) >> shift) & 0xFFu; };

    for (;;) {
        if (tid == 0) {
            s_tile = atomicAdd(tile_ctr, 1u);
            // L2 prefetch of the tile a grid further on in the tile sequence
            // (if it takes part)
            const uint32_t ahead = s_tile + ctas;
            if (aligned_src && ahead < num_tiles) {
                const uint32_t ja = tile_seg[ahead];
                const uint32_t sa = a.large_list[ja];
                const uint32_t ba = a.off[sa] + (ahead - tile_begin[ja]) * TILE;
                if ((!MSD || a.route[ja] != NO_ROUTE) && ba + TILE <= a.off[sa + 1] && (ba % (16 / sizeof(K))) == 0) {
                    dev::prefetch_l2(src_k + ba, TILE * sizeof(K));
                    if (HAS_V && (ba & 3) == 0) dev::prefetch_l2(src_v + ba, TILE * 4);
                }
            }
        }
        for (int i = tid; i < GROUPS * GSTRIDE; i += THREADS) warp_hist[i] = 0;
        __syncthreads();
        const uint32_t t = s_tile;
        if (t >= num_tiles) break;
        const uint32_t j = tile_seg[t];
        // a segment takes the MSD pass or the LSD passes; its tiles publish
        // nothing in the others, and no tile of another segment looks back
        // into it
        if (MSD) {
            const uint8_t rt = a.route[j];
            if (rt == NO_ROUTE) {
                __syncthreads();  // every thread has read s_tile before thread 0 takes the next tile
                continue;
            }
            shift = 8 * rt;
        }
        const uint32_t s = a.large_list[j];
        const uint32_t segb = a.off[s], sege = a.off[s + 1];
        const uint32_t lt = t - tile_begin[j];
        if ((uint64_t)lt * TILE >= sege - segb) {  // a tile outside its segment: never read or written
            if (tid == 0) dev::raise_error(a.err, dev::ERR_MISPLACED);
            __syncthreads();
            continue;
        }
        const uint32_t tile_base = segb + lt * TILE;
        const uint32_t valid = min((uint32_t)TILE, sege - tile_base);
        const bool first = lt == 0;

        const uint32_t wbase = tile_base + grp * 16 * ITEMS + gl;
        K key[ITEMS];
        uint32_t rd[ITEMS];
        uint32_t val[HAS_V ? ITEMS : 1];
        if (valid == (uint32_t)TILE) {
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) key[i] = src_k[wbase + i * 16];
            if (HAS_V) {
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) val[i] = src_v[wbase + i * 16];
            }
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) rd[i] = digit(key[i]);
        } else {
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                const uint32_t idx = wbase + i * 16;
                const bool in = idx < sege;
                key[i] = in ? src_k[idx] : K(0);
                if (HAS_V) val[i] = in ? src_v[idx] : 0u;
                rd[i] = in ? digit(key[i]) : 0xFFu;  // padding ranks last
            }
        }

        uint32_t* wh = warp_hist + grp * GSTRIDE;
        const uint32_t hbit = 1u << gl, hlt = hbit - 1u;
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const uint32_t d = rd[i];
            atomicOr(&wh[d], hbit);
            __syncwarp();
            const uint32_t x = wh[d];
            __syncwarp();
            const uint32_t peers = x & 0xFFFFu, before = x >> 16;
            if ((peers & hlt) == 0) wh[d] = (before + __popc(peers)) << 16;  // the new count; the mask cleared
            __syncwarp();
            rd[i] = ((before + __popc(peers & hlt)) << 8) | d;
        }
        __syncthreads();

        uint32_t count = 0;
        if (tid < RADIX) {
#pragma unroll
            for (int w = 0; w < GROUPS; ++w) {
                const uint32_t c = warp_hist[w * GSTRIDE + tid] >> 16;
                warp_hist[w * GSTRIDE + tid] = count;
                count += c;
            }
        }
        uint32_t agg = count;
        if (tid == RADIX - 1) agg -= (uint32_t)TILE - valid;
        uint64_t* my_status = a.ring + ((seq0 + t) & (RING_TILES - 1)) * RADIX;
        if (tid < RADIX) dev::st_relaxed(&my_status[tid], pack_status(first ? FLAG_PRE : FLAG_AGG, seq0 + t, agg));
        const uint32_t local = dev::bins_exclusive_sum(count, s_scratch);
        if (tid < RADIX) {
            s_local[tid] = local;
#pragma unroll
            for (int w = 0; w < GROUPS; ++w) warp_hist[w * GSTRIDE + tid] += local;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const uint32_t pos = warp_hist[grp * GSTRIDE + (rd[i] & 0xFFu)] + (rd[i] >> 8);
            s_keys[pos] = key[i];
            if (HAS_V) s_vals[pos] = val[i];
        }
        if (tid < RADIX) {
            uint32_t excl = 0;
            if (!first) {
                int64_t k = (int64_t)t - 1;
                bool done = false;
                while (!done) {
                    uint64_t w[LBW];
#pragma unroll
                    for (int q = 0; q < LBW; ++q)
                        if (k - q >= 0)
                            w[q] = dev::ld_relaxed(a.ring + ((seq0 + (uint64_t)(k - q)) & (RING_TILES - 1)) * RADIX +
                                                   tid);
#pragma unroll
                    for (int q = 0; q < LBW; ++q) {
                        if (done || k - q < 0) break;
                        const uint64_t seq = seq0 + (uint64_t)(k - q);
                        const uint64_t want = seq & TAG_MASK;
                        uint64_t x = w[q];
                        if ((x >> 62) == 0 || ((x >> 32) & TAG_MASK) != want) {
                            const uint64_t* pw = a.ring + (seq & (RING_TILES - 1)) * RADIX + tid;
                            const unsigned long long start = dev::globaltimer();
                            for (uint32_t spin = 1;; ++spin) {
                                x = dev::ld_relaxed(pw);
                                if ((x >> 62) != 0 && ((x >> 32) & TAG_MASK) == want) break;
                                if ((spin & 63) == 0 && dev::globaltimer() - start > dev::SPIN_LIMIT_NS) {
                                    dev::raise_error(a.err, dev::ERR_LOOKBACK_TIMEOUT);
                                    s_abort = 1;
                                    x = FLAG_PRE << 62;  // stop walking
                                    break;
                                }
                                __nanosleep(spin < 16 ? 32 : 128);
                            }
                        }
                        excl += (uint32_t)x;
                        if ((x >> 62) == FLAG_PRE) done = true;
                    }
                    k -= LBW;
                    if (k < 0) done = true;
                }
                dev::st_relaxed(&my_status[tid], pack_status(FLAG_PRE, seq0 + t, excl + agg));
            }
            s_bin_off[tid] = a.seg_hist[((size_t)j * P + (shift >> 3)) * RADIX + tid] + excl - s_local[tid];
        }
        __syncthreads();
        const uint32_t limit = s_abort ? 0u : valid;
        bool outside = false;  // a place outside the segment: nothing is written there, and the call fails
        if (limit == (uint32_t)TILE) {
            uint32_t o[ITEMS];
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) key[i] = s_keys[tid + i * THREADS];
            if (HAS_V) {
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) val[i] = s_vals[tid + i * THREADS];
            }
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) o[i] = s_bin_off[digit(key[i])] + tid + i * THREADS;
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                if (o[i] >= segb && o[i] < sege) {
                    dst_k[o[i]] = key[i];
                    if (HAS_V) dst_v[o[i]] = val[i];
                } else {
                    outside = true;
                }
            }
        } else {
            for (uint32_t q = tid; q < limit; q += THREADS) {
                const K kk = s_keys[q];
                const uint32_t o = s_bin_off[digit(kk)] + q;
                if (o >= segb && o < sege) {
                    dst_k[o] = kk;
                    if (HAS_V) dst_v[o] = s_vals[q];
                } else {
                    outside = true;
                }
            }
        }
        if (outside) dev::raise_error(a.err, dev::ERR_MISPLACED);
        __syncthreads();
    }
}

template <typename K, bool HAS_V, int THREADS, int ITEMS, int MINB, int LBW, bool MSD>
__global__ void __launch_bounds__(THREADS, MINB) k_seg_large_pass(SegArgs<K> a, int slot, bool with_msd)
{
    dev::chain();
    seg_large_pass<K, HAS_V, THREADS, ITEMS, LBW, MSD>(a, slot, with_msd, gridDim.x);
}

// ---------------------------------------------------------------------------
// Host
// ---------------------------------------------------------------------------
// Batches of few keys are bound by the launches and the longest CTA of each,
// not by the work: up to FEW_KEYS the longer one-CTA classes share a launch,
// up to VERY_FEW_KEYS all of them.
//
// 32-bit keys keep to the LSD passes (four) up to ROUTE_32BIT_KEYS: the MSD
// route's launches cost a batch that cannot use it about 30 us, and such keys
// are common (floats of a normal distribution). Segments of 500,000 keys, LSD
// alone / with the route: 3.4e7 normal floats 793 / 829 us, 6.7e7 1470 / 1496;
// uniform keys 771 / 708, 1426 / 1263. 64-bit keys, with eight passes to save,
// take the route at any size (1,800 segments 181 / 151 us; 5e6 keys 477 / 281).
//
// The count takes one digit first (see seg_large_count) above TWO_STEP_KEYS:
// 200,000 lognormal segments of u64 pairs take 11.67 ms for 12.11; 6.7e7 u64
// keys in segments of 40,000 1741 us for 1854, 1.9e7 592 for 622; at 5e6 the
// two extra launches cost what it saves. Segments whose highest digit the
// sample misses are counted twice: 3405 us for 3353.
constexpr std::size_t FEW_KEYS = std::size_t(1) << 22;
constexpr std::size_t VERY_FEW_KEYS = std::size_t(1) << 18;
constexpr std::size_t ROUTE_32BIT_KEYS = std::size_t(1) << 26;
constexpr std::size_t TWO_STEP_KEYS = std::size_t(1) << 24;
// The large path runs beside the small one, on the second stream, where both have
// much to do. Where most keys are in large segments (a mean of twice the one-CTA
// capacity, or of ONE_STREAM_SHARE of it in small batches), the small path's CTAs
// only keep the large path's from their SMs, and the other way round (us beside /
// after each other: 100 segments of 10,000 u64 keys 198 / 130, u32 pairs 127 / 106;
// of 100,000 u64 pairs 448 / 405, u32 keys 282 / 255). Others gain from running beside
// (1,000 of 200 u64 keys 78 / 104, of 12,000 floats with values 381 / 421).
constexpr float ONE_STREAM_SHARE = 0.7f;

template <typename K, bool HAS_V> struct LargeShape;
template <bool HV> struct LargeShape<uint32_t, HV> {
    static constexpr int THREADS = 256, ITEMS = 24, MINB = 2, LBW = HV ? 1 : 4;
};
template <bool HV> struct LargeShape<uint64_t, HV> {
    static constexpr int THREADS = 256, ITEMS = HV ? 20 : 24, MINB = 2, LBW = 4;
};

// CTAs of the kernel that fit an SM with that much dynamic shared memory,
// after the opt-in to it; asked once per device, kernel and amount (the two
// queries take longer than a launch).
template <typename F> static int occupancy(F* kernel, int threads, std::size_t smem)
{
    static std::mutex m;
    static std::map<std::tuple<int, const void*, std::size_t>, int> known;
    int dev = 0;
    check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
    const std::tuple<int, const void*, std::size_t> key(dev, (const void*)kernel, smem);
    std::lock_guard<std::mutex> lock(m);
    auto it = known.find(key);
    if (it != known.end()) return it->second;
    // static shared memory adds to the dynamic amount against the 48 KiB
    // default, so the opt-in is always made; it only ever grows
    static std::map<std::pair<int, const void*>, std::size_t> opted;
    std::size_t& most = opted[{dev, (const void*)kernel}];
    if (smem > most) {
        check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                   "cudaFuncSetAttribute");
        most = smem;
    }
    int b = 0;
    check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, threads, smem),
               "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
    return known[key] = b;
}

// The one-CTA sorts of the segments (sub: sub-buckets) of at most cap keys
// among n, a launch per class (small batches: the larger CTA's launch takes
// the lower classes too); `threads`: the first class's CTAs, 256 (16 keys per
// thread) or 512 (8).
template <typename K, bool HAS_V>
static void launch_cta_sorts(device_context& ctx, const SegArgs<K>& a, bool sub, uint32_t cap, std::size_t n, int threads,
                             cudaStream_t st)
{
    auto launch = [&](auto kern, int cta, std::size_t smem, uint32_t above, int cls, int last) {
        const std::size_t most = n / (above + 1) + 1;  // segments of the class
        const int grid = (int)std::min<std::size_t>(most, (std::size_t)ctx.sm_count * std::max(1, occupancy(kern, cta, smem)));
        launch_chained(kern, grid, cta, smem, st, a, cls, last, sub);
    };
    constexpr bool SMALL = sizeof(K) == 4;
    const int lowest = n <= VERY_FEW_KEYS ? 0 : n <= FEW_KEYS ? 1 : 2;  // class that the largest CTA's launch starts at
    const uint32_t above[CTA_CLASSES] = {(uint32_t)WARP_CAP, CLASS0_CAP, CLASS1_CAP};
    int done = CTA_CLASSES;  // classes from this one up are launched
    if (cap > CLASS1_CAP && n > CLASS1_CAP && max_cta_cap<K, HAS_V>() > CLASS1_CAP) {
        done = lowest;
        if constexpr (SMALL && !HAS_V)
            launch(&k_seg_tile<K, HAS_V, 1024, 16, 1>, 1024, tile::Sorter<K, HAS_V, 1024, 16>::SMEM, above[done], done, 2);
        else if constexpr (max_cta_cap<K, HAS_V>() > CLASS1_CAP)
            launch(&k_seg_tile<K, HAS_V, 512, 20, 1>, 512, tile::Sorter<K, HAS_V, 512, 20>::SMEM, above[done], done, 2);
    }
    if (done > 1 && cap > CLASS0_CAP && n > CLASS0_CAP) {
        done = std::min(lowest, 1);
        launch(&k_seg_tile<K, HAS_V, 512, 16, SMALL ? 2 : 1>, 512, tile::Sorter<K, HAS_V, 512, 16>::SMEM, above[done], done, 1);
    }
    if (done > 0 && threads == 512)
        launch(&k_seg_tile<K, HAS_V, 512, 8, 2>, 512, tile::Sorter<K, HAS_V, 512, 8>::SMEM, WARP_CAP, 0, 0);
    else if (done > 0)
        launch(&k_seg_tile<K, HAS_V, 256, 16, SMALL ? 3 : 2>, 256, tile::Sorter<K, HAS_V, 256, 16>::SMEM, WARP_CAP, 0, 0);
    check_cuda(cudaGetLastError(), "segmented sort cta launch");
}

template <typename K, bool HAS_V>
void run(device_context& ctx, const K* in_k, K* out_k, const uint32_t* in_v, uint32_t* out_v, std::size_t n,
         const uint32_t* off, std::size_t nseg, dev::KeyXform<K> xf, const seg_options& opt)
{
    constexpr int P = Traits<K>::PASSES;
    using LS = LargeShape<K, HAS_V>;
    constexpr int TILE = LS::THREADS * LS::ITEMS;
    constexpr int MAX_CAP = (int)max_cta_cap<K, HAS_V>();
    const uint32_t cta_cap =
        (uint32_t)std::max<int>(WARP_CAP + 1, std::min<int>(opt.cta_cap > 0 ? opt.cta_cap : MAX_CAP, MAX_CAP));
    const uint32_t max_large = (uint32_t)std::min<std::size_t>(nseg, n / (cta_cap + 1) + 1);
    const uint32_t max_tiles = (uint32_t)(n / TILE + max_large + 1);

    temp_buffer ctl(ctx.resource, sizeof(SegControl));
    temp_buffer lists(ctx.resource, ((1 + CTA_CLASSES) * nseg + 3 * (std::size_t)max_large) * sizeof(uint32_t));
    temp_buffer tile_seg(ctx.resource, 2 * (std::size_t)max_tiles * sizeof(uint32_t));
    temp_buffer seg_hist(ctx.resource, (std::size_t)max_large * P * RADIX * sizeof(uint32_t));
    const bool maybe_large = n > cta_cap;
    temp_buffer alt_k(ctx.resource, maybe_large && opt.alt_keys == nullptr ? n * sizeof(K) : 0);
    temp_buffer alt_v(ctx.resource, maybe_large && HAS_V && opt.alt_vals == nullptr ? n * sizeof(uint32_t) : 0);
    // MSD route: per large segment its pass (or none), and at most one
    // sub-bucket per window of a segment's keys
    const uint32_t msd_cap = opt.msd_cap <= 0 ? 0u : (uint32_t)std::max<int>(WARP_CAP + 1, std::min(opt.msd_cap, MAX_CAP));
    const bool msd = maybe_large && msd_cap > 0;
    const uint32_t max_sub = msd ? (uint32_t)(n / SUB_WINDOW) + max_large : 0;
    temp_buffer route(ctx.resource, maybe_large ? max_large : 0);
    temp_buffer sub_lists(ctx.resource, (std::size_t)max_sub * 4 * sizeof(uint32_t));
    const bool two_steps = msd && n > TWO_STEP_KEYS;
    temp_buffer rest(ctx.resource, two_steps ? (std::size_t)max_large * 16 + (std::size_t)max_tiles * 4 : 0);
    check_cuda(cudaMemsetAsync(ctl.get(), 0, sizeof(SegControl), ctx.stream), "cudaMemsetAsync");
    if (maybe_large && !msd)
        check_cuda(cudaMemsetAsync(route.get(), NO_ROUTE, max_large, ctx.stream), "cudaMemsetAsync");

    SegArgs<K> a;
    a.in_k = in_k;
    a.out_k = out_k;
    a.alt_k = opt.alt_keys != nullptr ? static_cast<K*>(opt.alt_keys) : alt_k.as<K>();
    a.in_v = in_v;
    a.out_v = out_v;
    a.alt_v = opt.alt_vals != nullptr ? opt.alt_vals : alt_v.as<uint32_t>();
    a.off = off;
    a.skip = opt.skip;
    a.nseg = (uint32_t)nseg;
    a.cta_cap = cta_cap;
    a.xf = xf;
    a.ctl = ctl.as<SegControl>();
    uint32_t* l = lists.as<uint32_t>();
    a.warp_list = l;
    a.cta_list = l + nseg;
    a.large_list = l + (1 + CTA_CLASSES) * nseg;
    a.tile_begin = a.large_list + max_large;
    a.tile_seg = tile_seg.as<uint32_t>();
    a.lsd_begin = msd ? a.tile_begin + max_large : a.tile_begin;
    a.lsd_seg = msd ? a.tile_seg + max_tiles : a.tile_seg;
    a.vary = two_steps ? rest.as<unsigned long long>() : nullptr;
    a.rest_begin = two_steps ? reinterpret_cast<uint32_t*>(a.vary + max_large) : nullptr;
    a.rest_seg = two_steps ? a.rest_begin + max_large : nullptr;
    a.guess = two_steps ? reinterpret_cast<uint8_t*>(a.rest_seg + max_tiles) : nullptr;
    a.seg_hist = seg_hist.as<uint32_t>();
    a.max_large = max_large;
    a.max_tiles = max_tiles;
    a.ring = ctx.lookback_ring;
    a.seq0 = maybe_large ? ctx.reserve_seq((uint64_t)(P + 1) * max_tiles) : 0;
    a.err = ctx.d_error;
    a.route = route.as<uint8_t>();
    a.sub_lists = sub_lists.as<uint32_t>();
    a.max_sub = max_sub;
    a.sub_cap = msd_cap;

    constexpr std::size_t per_warp_smem =
        2 * WARP_CAP * sizeof(K) + (HAS_V ? 2 * WARP_CAP * 4 : 0) + WARP_CAP * 4 + 2 * RADIX * 4;
    // the large pass: two half-warp count arrays of RADIX + LARGE_PAD words per warp, and a tile
    constexpr std::size_t large_pass_smem = (std::size_t)(LS::THREADS / 32) * (RADIX + LARGE_PAD) * 8 +
                                            (std::size_t)TILE * sizeof(K) + (HAS_V ? (std::size_t)TILE * 4 : 0);
    {
        kernel_timer kt(ctx, "segsort.classify");
        const int grid = (int)std::max<std::size_t>(1, std::min<std::size_t>((nseg + 255) / 256, (std::size_t)ctx.sm_count * 4));
        k_seg_classify<K, TILE><<<grid, 256, 0, ctx.stream>>>(a);
        check_cuda(cudaGetLastError(), "segmented sort classify launch");
    }
    // Fork: the large-segment path runs on the auxiliary stream (ONE_STREAM_SHARE).
    const float mean = (float)n / (float)nseg / (float)cta_cap;  // segment, in capacities
    const bool fork = !opt.sparse && maybe_large && mean < (n <= FEW_KEYS ? ONE_STREAM_SHARE : 2.0f);
    cudaStream_t aux = fork ? ctx.aux_stream() : ctx.stream;
    if (fork) {
        check_cuda(cudaEventRecord(ctx.fork_event, ctx.stream), "cudaEventRecord");
        check_cuda(cudaStreamWaitEvent(aux, ctx.fork_event, 0), "cudaStreamWaitEvent");
    }

    {
        kernel_timer kt(ctx, "segsort.small_warp");
        const std::size_t smem = per_warp_smem * SMALL_WARPS;
        auto kern = &k_seg_small_warp<K, HAS_V, false>;
        const int grid = (int)std::min<std::size_t>((nseg + SMALL_WARPS - 1) / SMALL_WARPS,
                                                    (std::size_t)ctx.sm_count * std::max(1, occupancy(kern, SMALL_THREADS, smem)));
        kern<<<grid, SMALL_THREADS, smem, ctx.stream>>>(a);
        check_cuda(cudaGetLastError(), "segmented sort warp launch");
    }
    {
        kernel_timer kt(ctx, "segsort.small_cta");
        launch_cta_sorts<K, HAS_V>(ctx, a, false, cta_cap, opt.sparse ? VERY_FEW_KEYS : n, opt.cta_threads, ctx.stream);
    }
    if (maybe_large) {
        {
            kernel_timer kt(ctx, "segsort.large_histogram", aux);
            const int tgrid = (int)std::min<std::size_t>(max_tiles, (std::size_t)ctx.sm_count * 4);
            k_seg_large_plan<K, TILE><<<tgrid, 256, 0, aux>>>(a);
            auto count = [&](auto hk) {
                launch_chained(hk, (int)std::min<std::size_t>(max_tiles, (std::size_t)ctx.sm_count * std::max(1, occupancy(hk, 256, 0))),
                               256, 0, aux, a);
            };
            const int rgrid = (int)std::min<std::size_t>(max_large, (std::size_t)ctx.sm_count * 8);
            if (two_steps) {
                count(&k_seg_large_count<K, TILE, COUNT_FIRST>);
                launch_chained(&k_seg_route<K, TILE, COUNT_FIRST>, rgrid, 256, 0, aux, a, true);
                count(&k_seg_large_count<K, TILE, COUNT_REST>);
                launch_chained(&k_seg_route<K, TILE, COUNT_REST>, rgrid, 256, 0, aux, a, true);
            } else {
                count(&k_seg_large_count<K, TILE, COUNT_ALL>);
                launch_chained(&k_seg_route<K, TILE, COUNT_ALL>, rgrid, 256, 0, aux, a, msd);
            }
            check_cuda(cudaGetLastError(), "segmented sort histogram launch");
        }
        const std::size_t psmem = large_pass_smem;
        auto pass_grid = [&](auto kern) {
            return (int)std::min<std::size_t>(max_tiles, (std::size_t)ctx.sm_count * std::max(1, occupancy(kern, LS::THREADS, psmem)));
        };
        if (msd) {
            auto mk = &k_seg_large_pass<K, HAS_V, LS::THREADS, LS::ITEMS, LS::MINB, LS::LBW, true>;
            const int mgrid = pass_grid(mk);
            kernel_timer kt(ctx, "segsort.msd_pass", aux);
            launch_chained(mk, mgrid, LS::THREADS, psmem, aux, a, 0, true);
            check_cuda(cudaGetLastError(), "segmented sort MSD pass launch");
        }
        auto pk = &k_seg_large_pass<K, HAS_V, LS::THREADS, LS::ITEMS, LS::MINB, LS::LBW, false>;
        const int pgrid = pass_grid(pk);
        // an even number of passes left out, so that the last one writes the output
        const int passes = opt.low_digits > 0 ? std::min(P, (opt.low_digits + 1) / 2 * 2) : P;
        for (int s = 0; s < passes; ++s) {
            kernel_timer kt(ctx, "segsort.large_pass", aux);
            launch_chained(pk, pgrid, LS::THREADS, psmem, aux, a, s, msd);
            check_cuda(cudaGetLastError(), "segmented sort pass launch");
        }
        if (msd) {
            // the MSD route's sub-buckets: from the scratch buffer into the output
            kernel_timer kt(ctx, "segsort.sub_buckets", aux);
            const std::size_t smem = per_warp_smem * SMALL_WARPS;
            auto wk = &k_seg_small_warp<K, HAS_V, true>;
            const int grid = (int)std::min<std::size_t>((max_sub + SMALL_WARPS - 1) / SMALL_WARPS,
                                                        (std::size_t)ctx.sm_count * std::max(1, occupancy(wk, SMALL_THREADS, smem)));
            launch_chained(wk, grid, SMALL_THREADS, smem, aux, a);
            launch_cta_sorts<K, HAS_V>(ctx, a, true, msd_cap, n, opt.cta_threads, aux);
        }
    }
    if (fork) {  // join
        check_cuda(cudaEventRecord(ctx.join_event, aux), "cudaEventRecord");
        check_cuda(cudaStreamWaitEvent(ctx.stream, ctx.join_event, 0), "cudaStreamWaitEvent");
    }
}

}  // namespace seg

void selftest_misplaced(device_context& ctx)
{
    // One segment of equal keys, whose bin starts lie just past its end: the
    // large pass must write none of them and record the error.
    using namespace seg;
    using LS = LargeShape<uint32_t, false>;
    constexpr uint32_t N = 1000, P = Traits<uint32_t>::PASSES;
    constexpr std::size_t smem =
        (std::size_t)(LS::THREADS / 32) * (RADIX + LARGE_PAD) * 8 + (std::size_t)LS::THREADS * LS::ITEMS * sizeof(uint32_t);
    ctx.activate();
    // the keys and the two other arrays; the segment's offsets; its index, first tile and tile; the bin starts
    std::vector<uint32_t> host(3 * N, 0u);
    host.insert(host.end(), {0u, N, 0u, 0u, 0u});
    host.resize(host.size() + P * RADIX, N);
    SegControl control{};
    control.n_large = control.large_tiles = 1;
    temp_buffer words(ctx.resource, host.size() * 4), ctl(ctx.resource, sizeof(SegControl));
    check_cuda(cudaMemcpyAsync(words.get(), host.data(), host.size() * 4, cudaMemcpyHostToDevice, ctx.stream), "cudaMemcpyAsync");
    check_cuda(cudaMemcpyAsync(ctl.get(), &control, sizeof(control), cudaMemcpyHostToDevice, ctx.stream), "cudaMemcpyAsync");
    SegArgs<uint32_t> a{};
    uint32_t* w = words.as<uint32_t>();
    a.in_k = w;
    a.out_k = w + N;
    a.alt_k = w + 2 * N;
    a.off = w + 3 * N;
    a.large_list = w + 3 * N + 2;
    a.tile_begin = a.lsd_begin = w + 3 * N + 3;
    a.tile_seg = a.lsd_seg = w + 3 * N + 4;
    a.seg_hist = w + 3 * N + 5;
    a.nseg = a.max_large = a.max_tiles = 1;
    a.ctl = ctl.as<SegControl>();
    a.ring = ctx.lookback_ring;
    a.seq0 = ctx.reserve_seq(P + 1);
    a.err = ctx.d_error;
    auto kernel = &k_seg_large_pass<uint32_t, false, LS::THREADS, LS::ITEMS, LS::MINB, LS::LBW, false>;
    occupancy(kernel, LS::THREADS, smem);  // opts in to the shared memory
    kernel<<<1, LS::THREADS, smem, ctx.stream>>>(a, 0, false);
    check_cuda(cudaGetLastError(), "segmented sort pass launch");
    check_cuda(cudaStreamSynchronize(ctx.stream), "cudaStreamSynchronize");  // the host's copies are read
}

uint32_t segsort_cta_cap(int key_bytes, bool has_values)
{
    return key_bytes == 4 ? (has_values ? seg::max_cta_cap<uint32_t, true>() : seg::max_cta_cap<uint32_t, false>())
                          : (has_values ? seg::max_cta_cap<uint64_t, true>() : seg::max_cta_cap<uint64_t, false>());
}

std::string segsort_batch_tuning_key(int key_bytes, bool has_values, std::size_t n, std::size_t num_segments)
{
    return segsort_tuning_key(key_bytes, has_values, n, num_segments) + ":batch";
}

std::string segsort_cta_threads_tuning_key() { return "segsort:cta_threads"; }

std::string segsort_threads_tuning_key(int key_bytes, bool has_values, std::size_t n, std::size_t num_segments)
{
    return segsort_tuning_key(key_bytes, has_values, n, num_segments) + ":threads";
}

std::string segsort_msd_tuning_key(int key_bytes, bool has_values, std::size_t n, std::size_t num_segments)
{
    return segsort_tuning_key(key_bytes, has_values, n, num_segments) + ":msd";
}

std::string segsort_tuning_key(int key_bytes, bool has_values, std::size_t n, std::size_t num_segments)
{
    // distribution class: average segment length, as a power of two
    const std::size_t avg = num_segments ? n / num_segments : n;
    return std::string("segsort:") + (key_bytes == 4 ? "u32" : "u64") + (has_values ? "kv" : "k") + ":" +
           tuning_table::size_class(n) + ":avg" + tuning_table::size_class(avg);
}

void segmented_sort(device_context& ctx, const void* keys_in, void* keys_out, int key_bytes, int key_kind,
                    const uint32_t* vals_in, uint32_t* vals_out, std::size_t n, const uint32_t* offsets,
                    std::size_t num_segments, bool descending, const seg_options& opt)
{
    if (key_bytes != 4 && key_bytes != 8) throw std::invalid_argument("segmented_sort: keys must be 32 or 64 bits");
    if (key_kind < 0 || key_kind > 2) throw std::invalid_argument("segmented_sort: unknown key kind");
    if ((vals_in == nullptr) != (vals_out == nullptr))
        throw std::invalid_argument("segmented_sort: values need both an input and an output");
    check_size(n);
    if (num_segments == 0 || n == 0) return;
    if (offsets == nullptr || keys_in == nullptr || keys_out == nullptr)
        throw std::invalid_argument("segmented_sort: null argument");
    if (num_segments > 0x7FFFFFFFu) throw std::length_error("segmented_sort: too many segments");
    if (opt.skip != nullptr && (keys_in != keys_out || vals_in != vals_out))
        throw std::invalid_argument("segmented_sort: skipped segments need an in-place call");
    ctx.activate();
    seg_options o = opt;
    if (o.msd_cap < 0) {
        launch_shape shape;
        o.msd_cap = ctx.tuning.lookup(segsort_msd_tuning_key(key_bytes, vals_in != nullptr, n, num_segments), shape)
                        ? shape.variant
                    : key_bytes == 4 && n <= seg::ROUTE_32BIT_KEYS ? 0
                                                           : (int)segsort_cta_cap(key_bytes, vals_in != nullptr);
    }
    if (o.cta_threads == 0) {
        launch_shape shape;
        if (ctx.tuning.lookup(segsort_threads_tuning_key(key_bytes, vals_in != nullptr, n, num_segments), shape) ||
            ctx.tuning.lookup(segsort_cta_threads_tuning_key(), shape))
            o.cta_threads = shape.variant;
    }
    if (key_bytes == 4) {
        const auto xf = dev::make_xform<uint32_t>(key_kind, descending);
        if (vals_in)
            seg::run<uint32_t, true>(ctx, static_cast<const uint32_t*>(keys_in), static_cast<uint32_t*>(keys_out),
                                     vals_in, vals_out, n, offsets, num_segments, xf, o);
        else
            seg::run<uint32_t, false>(ctx, static_cast<const uint32_t*>(keys_in), static_cast<uint32_t*>(keys_out),
                                      nullptr, nullptr, n, offsets, num_segments, xf, o);
    } else {
        const auto xf = dev::make_xform<uint64_t>(key_kind, descending);
        if (vals_in)
            seg::run<uint64_t, true>(ctx, static_cast<const uint64_t*>(keys_in), static_cast<uint64_t*>(keys_out),
                                     vals_in, vals_out, n, offsets, num_segments, xf, o);
        else
            seg::run<uint64_t, false>(ctx, static_cast<const uint64_t*>(keys_in), static_cast<uint64_t*>(keys_out),
                                      nullptr, nullptr, n, offsets, num_segments, xf, o);
    }
}

void segmented_sort_xf(device_context& ctx, uint64_t* keys, uint32_t* vals, uint64_t xf_a, uint64_t xf_b, std::size_t n,
                       const uint32_t* offsets, std::size_t num_segments, const seg_options& opt)
{
    const dev::KeyXform<uint64_t> xf{xf_a, xf_b};
    if (vals != nullptr) seg::run<uint64_t, true>(ctx, keys, keys, vals, vals, n, offsets, num_segments, xf, opt);
    else seg::run<uint64_t, false>(ctx, keys, keys, nullptr, nullptr, n, offsets, num_segments, xf, opt);
}

}  // namespace gbc
