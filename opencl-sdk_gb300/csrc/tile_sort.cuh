// Stable sort of up to THREADS x ITEMS keys (and 32-bit values) by one CTA:
// the keys stay in registers, each digit pass ranks them by half-warps and
// exchanges them through one shared-memory copy of the tile.
//
// No reference counterpart (the reference sorts every array with the same
// eight device-wide passes, lib/src/Compute/Algorithm.cpp:453-527); used for
// segments and buckets that fit one CTA and for small whole arrays.
//
// Only the highest digits are sorted. With `diff` the bits on which the keys
// differ and 2^b >= len, the passes cover at least the b + SLACK_BITS bits
// from the highest differing one down (whole 8-bit digits); a sample of the
// keys decides whether few enough neighbours will agree in those bits, or
// another digit is needed. The tile is then checked: wherever a key is
// larger than its successor, the run of equal leading bits around it is put
// in order by insertion (stable). A run too long for that sends the tile
// through all its digits after all; it starts from the order reached, in
// which equal keys still stand in input order, so the result is the same.
// For 64-bit keys this is two or three passes instead of eight; uniform keys
// take two up to 8,192 of them (SLACK_BITS = 3: one key in eight has an equal
// neighbour in 16 bits), normally distributed floats three instead of four.
#pragma once

#include <cstdint>

#include "device_common.cuh"
#include "sort_internal.hpp"

namespace gbc {
namespace tile {

using onesweep::RADIX;

constexpr int SLACK_BITS = 3;     // bits sorted beyond log2 of the tile's length
constexpr int SAMPLE_ROWS = 4;    // rows of every group that the sample takes
constexpr float MAX_SHARE = 0.35f;  // keys with an equal neighbour in the sorted bits, per key, that repair is worth
constexpr uint32_t MAX_RUN = 24;  // longest run put in order by insertion, to either side of its first fault

template <int THREADS> struct Scratch {
    uint32_t part[THREADS / RADIX][RADIX];  // per 256 threads: counts of each digit
    uint32_t start[RADIX];
    uint32_t warp[8];
    uint64_t diff[THREADS / 32];
    uint64_t first;
    uint32_t tally[3];
};

// The inverse of KeyXform (whose `a` never has the top bit set).
template <typename K> __device__ __forceinline__ K undo_xform(const dev::KeyXform<K>& xf, K t)
{
    return dev::KeyXform<K>{xf.a, 0}(t ^ xf.b);
}

template <typename K, bool HAS_V, int THREADS, int ITEMS> struct Sorter {
    static constexpr int CAP = THREADS * ITEMS;
    static constexpr int GROUPS = THREADS / 16;  // ranking groups: half-warps
    // One word of padding: equal digits in the two halves of a warp fall into
    // different banks.
    static constexpr int GSTRIDE = RADIX + 1;
    static constexpr int SETS = THREADS / RADIX;  // each 256 threads scan the counts of 16 groups
    static constexpr std::size_t SMEM =
        (std::size_t)GROUPS * GSTRIDE * 4 + (std::size_t)CAP * sizeof(K) + (HAS_V ? (std::size_t)CAP * 4 : 0);
    static_assert(THREADS % RADIX == 0 && 16 * ITEMS < (1 << 16) && ITEMS <= 32, "16-bit counts; one bit per item");

    uint32_t* counts;
    K* keys;         // the tile, exchanged and finally sorted (transformed keys)
    uint32_t* vals;
    Scratch<THREADS>& sc;
    uint32_t len, rows;  // rows of 16 keys per group in use
    int misplaced;       // the last digit's thread: the counts do not add up to the tile

    __device__ __forceinline__ Sorter(unsigned char* smem, Scratch<THREADS>& s) : sc(s), len(0), rows(0), misplaced(0)
    {
        counts = reinterpret_cast<uint32_t*>(smem);
        keys = reinterpret_cast<K*>(smem + (std::size_t)GROUPS * GSTRIDE * 4);
        vals = reinterpret_cast<uint32_t*>(keys + CAP);
    }

    //! Index within the tile of this thread's first key; key i is 16 i further on.
    __device__ __forceinline__ uint32_t first_index() const
    {
        return (threadIdx.x >> 4) * 16 * rows + (threadIdx.x & 15);
    }

    // One digit pass: the keys in registers go to their places in shared memory.
    __device__ __forceinline__ void pass(const K (&key)[ITEMS], const uint32_t (&val)[HAS_V ? ITEMS : 1], int shift)
    {
        const int tid = threadIdx.x, gl = tid & 15, grp = tid >> 4;
        uint4* c4 = reinterpret_cast<uint4*>(counts);
        for (int i = tid; i < GROUPS * GSTRIDE / 4; i += THREADS) c4[i] = make_uint4(0, 0, 0, 0);
        __syncthreads();
        const uint32_t base = first_index();
        uint32_t* wh = counts + grp * GSTRIDE;
        const uint32_t hbit = 1u << gl, hlt = hbit - 1u;
        uint32_t rd[ITEMS];  // (rank << 8) | digit
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if (i < (int)rows) {
                // past the end the digit is 255, so padding ranks last
                const uint32_t d = base + i * 16 < len ? (uint32_t)(key[i] >> shift) & 0xFFu : 0xFFu;
                atomicOr(&wh[d], hbit);
                __syncwarp();
                const uint32_t x = wh[d];
                __syncwarp();
                const uint32_t peers = x & 0xFFFFu, before = x >> 16;
                if ((peers & hlt) == 0) wh[d] = (before + __popc(peers)) << 16;
                __syncwarp();
                rd[i] = ((before + __popc(peers & hlt)) << 8) | d;
            }
        }
        __syncthreads();
        // Counts become places: exclusive over digits, then over groups.
        const int d = tid & (RADIX - 1), set = tid / RADIX;
        uint32_t* col = counts + set * 16 * GSTRIDE + d;
        uint32_t c[16], sum = 0;
#pragma unroll
        for (int w = 0; w < 16; ++w) {
            c[w] = col[w * GSTRIDE] >> 16;
            sum += c[w];
        }
        uint32_t total = sum, before = 0;
        if (SETS > 1) {
            sc.part[set][d] = sum;
            __syncthreads();
            total = 0;
#pragma unroll
            for (int s = 0; s < SETS; ++s) {
                const uint32_t p = sc.part[s][d];
                if (s < set) before += p;
                total += p;
            }
        }
        uint32_t incl = 0;
        if (tid < RADIX) {
            incl = dev::warp_inclusive_scan(total, [](uint32_t x, uint32_t y) { return x + y; });
            if ((tid & 31) == 31) sc.warp[tid >> 5] = incl;
        }
        __syncthreads();
        if (tid < RADIX) {
            uint32_t lower = 0;
#pragma unroll
            for (int w = 0; w < 8; ++w)
                if (w < (tid >> 5)) lower += sc.warp[w];
            sc.start[d] = lower + incl - total;
            if (d == RADIX - 1 && lower + incl != rows * THREADS) misplaced = 1;
        }
        __syncthreads();
        uint32_t run = sc.start[d] + before;
#pragma unroll
        for (int w = 0; w < 16; ++w) {
            col[w * GSTRIDE] = run;
            run += c[w];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if (i < (int)rows) {
                // always below CAP unless the counts are wrong (see `total`)
                const uint32_t pos = min(wh[rd[i] & 0xFFu] + (rd[i] >> 8), (uint32_t)CAP - 1);
                keys[pos] = key[i];
                if (HAS_V) vals[pos] = val[i];
            }
        }
        __syncthreads();
    }

    __device__ __forceinline__ void read_back(K (&key)[ITEMS], uint32_t (&val)[HAS_V ? ITEMS : 1])
    {
        const uint32_t base = first_index();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
            if (i < (int)rows) {
                key[i] = keys[base + i * 16];
                if (HAS_V) val[i] = vals[base + i * 16];
            }
    }

    // Puts every run of keys that agree from bit `lo` up in order; false when
    // a run is too long. A fault (a key larger than its successor) is taken
    // by the thread that finds it unless its run has an earlier one.
    __device__ __forceinline__ bool repair(int lo)
    {
        const int tid = threadIdx.x;
        int long_run = 0;   // this thread met a run that is too long
        uint32_t mine = 0;  // bit i: the fault at i * THREADS + tid is this thread's
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const uint32_t idx = i * THREADS + tid;
            if (i < (int)rows && idx > 0 && idx < len && keys[idx - 1] > keys[idx]) {
                bool take = true;
                uint32_t h = idx - 1;  // towards the run's first key
                for (; h > 0 && (keys[h - 1] >> lo) == (keys[h] >> lo); --h) {
                    if (keys[h - 1] > keys[h]) {
                        take = false;
                        break;
                    }
                    if (idx - h > MAX_RUN) {
                        long_run = 1;
                        take = false;
                        break;
                    }
                }
                if (take) mine |= 1u << i;
            }
        }
        // The barrier's OR is the same for every thread (a shared flag could be
        // set again by a thread already past the barrier before another reads it).
        __syncwarp();
        if (__syncthreads_or(long_run)) return false;
        // Runs change from here on, each by one thread.
        while (mine != 0) {
            const int i = __ffs(mine) - 1;
            mine &= mine - 1;
            const uint32_t idx = i * THREADS + tid;
            const K top = keys[idx] >> lo;
            uint32_t h = idx - 1;
            while (h > 0 && (keys[h - 1] >> lo) == top) --h;
            for (uint32_t j = idx; j < len; ++j) {
                const K x = keys[j];
                if ((x >> lo) != top) break;
                if (j - idx > MAX_RUN) {
                    long_run = 1;
                    break;
                }
                const uint32_t v = HAS_V ? vals[j] : 0u;
                uint32_t m = j;
                for (; m > h && keys[m - 1] > x; --m) {
                    keys[m] = keys[m - 1];
                    if (HAS_V) vals[m] = vals[m - 1];
                }
                keys[m] = x;
                if (HAS_V) vals[m] = v;
            }
        }
        __syncwarp();
        return __syncthreads_or(long_run) == 0;
    }

    // The number of leading digits to sort, from `want` up to all of them: a
    // sample of the keys is marked in a bitmap of 2^16 leading-bit patterns
    // (hashed beyond 16 bits), and the marks found already set estimate the
    // chance that two keys agree in those bits. Costs about a twentieth of a
    // digit pass. Marks that hardly get fewer from digit to digit are those of
    // keys that cluster, whose runs are too long for repair however few they
    // are: a number beyond `want` has to leave few of them, or a third of them per
    // digit (10,000 segments of 1,000 u64 keys that are the AND of four words: six
    // passes, a failed repair and all eight 1377 us, all eight at once 752).
    __device__ __forceinline__ int choose_passes(const K (&key)[ITEMS], int bits, int want, int all_passes)
    {
        static_assert(GROUPS * GSTRIDE >= 2048, "the bitmap lies in the counts");
        const int tid = threadIdx.x;
        const uint32_t base = first_index();
        int slot = 0;  // of this round's tally; the last one's is kept, the next one's is another
        for (int p = want; p < all_passes; slot = slot == 2 ? 0 : slot + 1) {
            uint4* c4 = reinterpret_cast<uint4*>(counts);
            for (int i = tid; i < 2048 / 4; i += THREADS) c4[i] = make_uint4(0, 0, 0, 0);
            uint32_t* tally = &sc.tally[slot];
            if (tid == 0) *tally = 0;
            __syncthreads();
            const int lo = bits - 8 * p;
            const bool hashed = p > 2;
            uint32_t seen = 0;  // (keys << 16) | marks already set
#pragma unroll
            for (int i = 0; i < (SAMPLE_ROWS < ITEMS ? SAMPLE_ROWS : ITEMS); ++i) {
                if (i < (int)rows && base + i * 16 < len) {
                    const uint64_t x = (uint64_t)key[i] >> lo;
                    const uint32_t h = (hashed ? ((uint32_t)x ^ (uint32_t)(x >> 32) * 0x85EBCA6Bu) * 0x9E3779B1u >> 16
                                               : (uint32_t)x) & 0xFFFFu;
                    const uint32_t old = atomicOr(&counts[h >> 5], 1u << (h & 31));
                    seen += (1u << 16) + ((old >> (h & 31)) & 1u);
                }
            }
            seen = __reduce_add_sync(dev::FULL_MASK, seen);
            if ((tid & 31) == 0) atomicAdd(tally, seen);
            __syncthreads();
            const uint32_t all = *tally;
            const float s = (float)(all >> 16);
            // pairs expected at the largest share worth repairing, and by the hash alone
            const float limit = s * s * (MAX_SHARE / 2 / (float)len + (hashed ? 1.0f / 131072 : 0.0f)) + 2.0f;
            const uint32_t marks = all & 0xFFFFu;
            if ((float)marks <= limit) {
                if (p == want || marks <= 2 || 8.0f * (float)marks <= limit) return p;
                const uint32_t last = sc.tally[slot == 0 ? 2 : slot - 1];
                if (marks * (2 * (last & 0xFFFFu) > last >> 16 ? 9 : 3) <= (last & 0xFFFFu)) return p;
            }
            // most keys agree: not the next number either, where there are many
            p += 2 * marks > all >> 16 && all_passes - p > 3 ? 2 : 1;
        }
        return all_passes;
    }

    //! Sorts the `n` <= CAP transformed keys held in registers (key i of the
    //! thread is tile index first_index() + 16 i, so load after setting
    //! `rows`) into keys[0, n) / vals[0, n). Every thread of the CTA calls it;
    //! false (for all) if a pass's counts were wrong, which no input leads to.
    __device__ __forceinline__ bool sort(K (&key)[ITEMS], uint32_t (&val)[HAS_V ? ITEMS : 1])
    {
        const int tid = threadIdx.x;
        const uint32_t base = first_index();
        if (tid == 0) sc.first = (uint64_t)key[0];
        __syncthreads();
        const K first = (K)sc.first;
        K diff = 0;
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
            if (i < (int)rows && base + i * 16 < len) diff |= key[i] ^ first;
        uint32_t lo32 = __reduce_or_sync(dev::FULL_MASK, (uint32_t)diff), hi32 = 0;
        if (sizeof(K) == 8) hi32 = __reduce_or_sync(dev::FULL_MASK, (uint32_t)((uint64_t)diff >> 32));
        if ((tid & 31) == 0) sc.diff[tid >> 5] = ((uint64_t)hi32 << 32) | lo32;
        __syncthreads();
        uint64_t all = 0;
#pragma unroll
        for (int w = 0; w < THREADS / 32; ++w) all |= sc.diff[w];
        if (all == 0) {  // one key value: already in order
#pragma unroll
            for (int i = 0; i < ITEMS; ++i)
                if (i < (int)rows) {
                    keys[base + i * 16] = key[i];
                    if (HAS_V) vals[base + i * 16] = val[i];
                }
            __syncthreads();
            return true;
        }
        const int bits = 64 - __clzll((long long)all);  // the keys agree above these
        const int all_passes = (bits + 7) / 8;
        const int want = (32 - __clz((int)(len - 1)) + SLACK_BITS + 7) / 8;  // len >= 2: some bit differs
        // Digits from the top down; the lowest may overlap the next when
        // `bits` is no multiple of 8, which sorts some bits twice.
        int passes = want < all_passes ? choose_passes(key, bits, want, all_passes) : all_passes;
        for (bool again = false;; again = true) {
            for (int p = 0; p < passes; ++p) {
                if (again || p > 0) read_back(key, val);
                pass(key, val, max(0, bits - 8 * (passes - p)));
            }
            if (passes == all_passes || repair(bits - 8 * passes)) return __syncthreads_or(misplaced) == 0;
            passes = all_passes;
        }
    }
};

}  // namespace tile
}  // namespace gbc
