// 64-bit keys: sorting the leading digits only, and putting right what they
// leave out of order. Included by sort.cu.
//
// No reference counterpart (the reference sorts 32-bit keys in eight 4-bit
// passes, lib/src/Compute/Algorithm.cpp:453-527). Every digit pass of 2^29
// pairs takes 3.8 ms, and 2^29 keys that differ in all eight digits are mostly
// in order after the four highest: n keys have about n / 2^32 neighbours
// each that agree in 32 bits and yet differ. So (2^29 pairs 32.2 -> 19.6 ms,
// 2^28 keys alone 12.1 -> 7.5):
//
//   k_sample    (before the passes) a sample of up to 2^17 keys, entered in hash tables
//               by their leading digits, counts the pairs that agree in those
//               digits but differ (equal keys need no further digit). The
//               fewest digits for which at most LAMBDA such neighbours per key
//               are expected become the pass plan; if none, the plan stays;
//   k_faults    (after the passes) finds every key larger than its successor.
//               Around it lies a run of keys that agree in the sorted digits.
//               A short run inside the CTA's tile is put in order at once, by
//               a thread (insertion) or a warp (ranks); one that crosses the
//               tile's edge goes into a list, a long run's bounds into another;
//   k_repair    puts the listed short runs in order, one warp each;
//   k_long_runs turns the long runs into segments for the segmented sort.
//
// All of it is stable: passes, insertion, ranks and the segmented sort are, and equal
// keys are never apart. When there are too many long runs (keys that the sample
// judged wrongly), the array takes all its digit passes after all, from the
// order reached. Everything is decided on the device.
#pragma once

#include "tile_sort.cuh"

namespace gbc {
namespace onesweep {
namespace partial {

using dev::FULL_MASK;

// MIN_KEYS: the extra steps cost a sort that has no use for them about what the
// overlapped launches save it, and take 40% off one that has (pairs, before both /
// now: 2^23 keys that are the AND of 4 words 702 / 704 us, of 2 687 / 600, uniform
// ones 654 / 406; 2^24 1227 / 1196, 1219 / 1017, 1169 / 694; keys alone, 2^23,
// AND of 4 560 / 565, three digits 230 / 223).
// SEGMENTED_KEYS: long runs of any length go to the segmented sort, about 15
// launches more; below, one kernel sorts those of up to a CTA's capacity (sort and
// reduce_by_key of 1.5 10^8 Zipf keys: 5.91 ms for 6.78). Keys of few digits pay 35
// us for it (2^27.2 keys of two digits 1.92 -> 1.95 ms, 2^28 3.29 -> 3.32).
constexpr std::size_t MIN_KEYS = std::size_t(1) << 23, SEGMENTED_KEYS = std::size_t(1) << 27;
constexpr int CANDIDATES = 3;  // digit counts tried: the least possible, and one or two more
constexpr int FIRST_PASSES = 6;  // digit passes launched before the faults are looked for
constexpr uint32_t MIN_SAMPLE = 1u << 15, MAX_SAMPLE = 1u << 17;
constexpr float LAMBDA = 0.35f;                         // leaves a fault at about one key in twelve
constexpr uint32_t REACH = 24;       // a short run ends within this many keys of its first fault
// A run of more keys than this is a warp's: a thread's insertion takes about a
// microsecond per key of a run of 20 and more, and the tile's CTA waits for it. (Keys
// that are the AND of two uniform words have few runs, but some of up to 50
// keys, many of them in the first tiles. 2^24 of them: k_faults 288 -> 182 us, of
// it the walks to the ends of the first tile's runs 50; k_repair 60 -> 16.)
constexpr uint32_t MANY_KEYS = 6;
constexpr int FT_ROWS = 16;
constexpr uint32_t FT_TILE = 256 * FT_ROWS, FT_HALO = 32;  // k_faults' tile, and the keys read to either side of it
constexpr uint32_t MAX_LONG = 8192;  // long runs
constexpr uint32_t LONG_SET = 4 * MAX_LONG;

//! Device control block of the extra steps (zeroed before each sort).
struct Control {
    uint32_t conflicts[CANDIDATES];
    uint32_t repeats;   // sampled keys met again
    uint32_t done;
    uint32_t lowest;    // the sorted digits start at this bit; 0: all are sorted, nothing to check
    uint32_t faults;    // short runs listed
    uint32_t long_runs;
    uint32_t overflow;  // too many long runs: all digits after all
    uint32_t later;     // passes of the second plan (an even number, so that it ends where it began)
};

template <typename K> struct Args {
    SortArgs<K> a;
    Control* ctl;
    SortControl* all;          // the second plan, from the order reached
    bool segmented;            // long runs go to the segmented sort
    uint32_t sample;             // keys sampled, a power of two
    unsigned long long* tables;  // CANDIDATES x 2 sample keys' complements, zero where empty
    int least;                 // digits of the first candidate
    uint32_t* fault;           // first faults of the short runs that cross a tile's edge (one per tile at most)
    uint32_t* set;             // LONG_SET begins of long runs plus one, zero where empty
    uint32_t* begin;           // MAX_LONG
    uint32_t* end;
    uint32_t* off;             // 2 MAX_LONG segment offsets: even segments are the runs
};

// The sample's size: pairs that agree in the least digits tried grow with its
// square, so that the n / sample^2 keys a pair stands for stay few.
inline uint32_t sample_size(std::size_t n)
{
    uint32_t s = MIN_SAMPLE;
    while (s < MAX_SAMPLE && (uint64_t)s * s < 32 * (uint64_t)n) s *= 2;
    return s;
}

// One sampled key per thread.
template <typename K> __global__ void __launch_bounds__(256) k_sample(Args<K> p)
{
    dev::chain();
    __shared__ uint32_t s_found[CANDIDATES + 1];
    __shared__ int s_last, s_digits;
    const SortArgs<K>& a = p.a;
    const int tid = threadIdx.x;
    PassPlan& plan = a.ctl->plan;
    const int active = (int)plan.num_active;
    uint32_t lo[CANDIDATES];  // first bit of the candidate's digits, or 64
#pragma unroll
    for (int c = 0; c < CANDIDATES; ++c) {
        const int digits = p.least + c;
        lo[c] = digits < active && digits <= FIRST_PASSES ? plan.shift[active - digits] : 64u;
    }
    if (tid <= CANDIDATES) s_found[tid] = 0;
    __syncthreads();
    const uint32_t step = a.n / p.sample;  // >= 256
    const uint32_t mask = 2 * p.sample - 1;
    for (uint32_t i = blockIdx.x * 256 + tid; i < p.sample; i += gridDim.x * 256) {
        // a varying place within each step, so that no period of the input is followed
        const K k = a.in_keys[(uint64_t)i * step + (i * 0x9E3779B1u >> 8) % step];
        const unsigned long long x = a.xf(k), mine = ~x;
        if (mine == 0) continue;
        uint32_t slot[CANDIDATES];
        unsigned long long old[CANDIDATES];  // all candidates' first slots at once
#pragma unroll
        for (int c = 0; c < CANDIDATES; ++c) {
            if (lo[c] == 64) continue;
            slot[c] = (uint32_t)(((x >> lo[c]) * 0x9E3779B97F4A7C15ull) >> 32) & mask;
            old[c] = atomicCAS(p.tables + (size_t)c * (mask + 1) + slot[c], 0ull, mine);
        }
#pragma unroll
        for (int c = 0; c < CANDIDATES; ++c) {
            if (lo[c] == 64) continue;
            unsigned long long* table = p.tables + (size_t)c * (mask + 1);
            unsigned long long seen = old[c];
            for (uint32_t s = slot[c]; seen != 0;) {  // at most half full
                if (seen == mine) {
                    if (c == 0) atomicAdd(&s_found[CANDIDATES], 1u);
                    break;
                }
                if ((~seen >> lo[c]) == (x >> lo[c])) {
                    atomicAdd(&s_found[c], 1u);
                    break;
                }
                s = (s + 1) & mask;
                seen = table[s];
                if (seen == 0) seen = atomicCAS(&table[s], 0ull, mine);
            }
        }
    }
    __syncthreads();
    if (tid < CANDIDATES && s_found[tid] != 0) atomicAdd(&p.ctl->conflicts[tid], s_found[tid]);
    if (tid == CANDIDATES && s_found[tid] != 0) atomicAdd(&p.ctl->repeats, s_found[tid]);
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(&p.ctl->done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // The last CTA chooses. Where values repeat, a long run is as likely as a
    // frequent value's meeting any other: without the segmented sort behind,
    // one digit more.
    if (tid == 0) {
        s_digits = 0;
        const int from = !p.segmented && dev::ld_relaxed(&p.ctl->repeats) > p.sample / 64 ? 1 : 0;
        for (int c = from; c < CANDIDATES && s_digits == 0; ++c) {
            const int digits = p.least + c;
            if (digits >= active || digits > FIRST_PASSES) break;
            const float pairs = (float)dev::ld_relaxed(&p.ctl->conflicts[c]);
            if (pairs * 2.0f * (float)a.n <= LAMBDA * (float)p.sample * (float)p.sample) s_digits = digits;
        }
    }
    __syncthreads();
    // Two plans: the leading digits now and, if the lists overflow, all of them
    // later; or the lowest FIRST_PASSES digits now and the rest later. The later
    // plan sorts its first digit twice where that makes its passes even.
    const int digits = s_digits;
    const int now = digits != 0 ? digits : min(active, FIRST_PASSES);
    const int drop = digits != 0 ? active - digits : 0;          // digits before the first plan's
    const int from = digits != 0 ? 0 : now;                      // digits before the second plan's
    const int later = active - from, pad = later & 1;
    PassPlan& all = p.all->plan;
    uint32_t start[8];  // this thread's column, read before any of it is moved
#pragma unroll
    for (int s = 0; s < 8; ++s) start[s] = s < active ? plan.bin_start[s][tid] : 0u;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        if (s >= from && s < active) all.bin_start[s - from + pad][tid] = start[s];
        if (s == from && s < active) all.bin_start[0][tid] = start[s];
        if (drop > 0 && s >= drop && s < drop + now) plan.bin_start[s - drop][tid] = start[s];
    }
    if (tid == 0) {
        uint32_t shift[8];
#pragma unroll
        for (int s = 0; s < 8; ++s) shift[s] = plan.shift[s];
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            if (s >= from && s < active) all.shift[s - from + pad] = shift[s];
            if (s == from && s < active) all.shift[0] = shift[s];
            if (drop > 0 && s >= drop && s < drop + now) plan.shift[s - drop] = shift[s];
        }
        plan.num_active = now;
        p.ctl->later = later + pad;
        if (digits != 0) p.ctl->lowest = plan.shift[0];
        else all.num_active = later + pad;
    }
}

template <typename K> struct Output {
    const K* keys;
    dev::KeyXform<K> xf;
    uint32_t n, lo;
    // read anew each time: other threads put other runs in order meanwhile,
    // which changes no key's leading digits
    __device__ K at(uint32_t i) const { return xf(*(const volatile K*)&keys[i]); }
    // whether keys i - 1 and i agree in the sorted digits
    __device__ bool joined(uint32_t i) const { return (at(i - 1) >> lo) == (at(i) >> lo); }
};

// A long run around position i: its bounds, once per run, into the list.
template <typename K> __device__ __noinline__ void note_long_run(const Args<K>& p, const Output<K>& out, uint32_t i)
{
    if (dev::ld_relaxed(&p.ctl->overflow) != 0) return;
    const K top = out.at(i) >> out.lo;
    // Steps that double, then a binary search: most long runs are short ones
    // and a bit, and a search of the whole array is 48 dependent loads, 20 us.
    uint32_t lo = 0, hi = i;  // the run's first key is one of lo .. hi
    for (uint32_t d = 32; d <= i; d *= 2) {
        if ((out.at(i - d) >> out.lo) < top) {
            lo = i - d + 1;
            break;
        }
        hi = i - d;
    }
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if ((out.at(mid) >> out.lo) < top) lo = mid + 1;
        else hi = mid;
    }
    const uint32_t b = lo;
    for (uint32_t s = b * 0x9E3779B1u >> 8, tries = 0;; ++s, ++tries) {
        if (tries == 64) {
            p.ctl->overflow = 1;
            return;
        }
        const uint32_t seen = atomicCAS(&p.set[s & (LONG_SET - 1)], 0u, b + 1);
        if (seen == b + 1) return;
        if (seen == 0) break;
    }
    lo = i + 1, hi = out.n;  // the run ends before one of lo .. hi
    for (uint32_t d = 32; d < out.n - i; d *= 2) {
        if ((out.at(i + d) >> out.lo) > top) {
            hi = i + d;
            break;
        }
        lo = i + d + 1;
    }
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if ((out.at(mid) >> out.lo) > top) hi = mid;
        else lo = mid + 1;
    }
    const uint32_t r = atomicAdd(&p.ctl->long_runs, 1u);
    if (r < MAX_LONG) {
        p.begin[r] = b;
        p.end[r] = lo;
    } else {
        p.ctl->overflow = 1;
    }
}

// The rank of x, key `self` of `count` keys, in their stable order; key(j) is
// the same for the whole warp.
template <typename K, typename F> __device__ __forceinline__ uint32_t stable_rank(K x, uint32_t self, uint32_t count, F key)
{
    uint32_t r = 0;
#pragma unroll 4
    for (uint32_t j = 0; j < count; ++j) {
        const K y = key(j);
        r += y < x || (y == x && j < self) ? 1u : 0u;
    }
    return r;
}

// Reads the sorted keys once, a tile and its halo at a time. A short run
// belongs to the thread that finds its first fault, or to the warp that takes it
// from the tile's list, so no two write the same keys; a thread that meets keys of another run only looks at their
// leading digits, which stay. (Walking the runs in global memory took 2.5 ms
// for 2^29 Zipf keys and 6 ms for uniform ones.)
template <typename K, bool HAS_V> __global__ void __launch_bounds__(256) k_faults(Args<K> p)
{
    dev::chain();
    const uint32_t lo = p.ctl->lowest;
    if (lo == 0) return;
    __shared__ K s_keys[FT_TILE + 2 * FT_HALO];
    __shared__ uint32_t s_run[FT_TILE / (MANY_KEYS + 1) + 1];  // (keys << 16) | first key within the tile
    __shared__ uint32_t s_runs;
    static_assert(2 * REACH <= 64, "a short run is at most two keys per lane");
    const Output<K> out{p.a.out_keys, p.a.xf, p.a.n, lo};
    const uint32_t n = p.a.n;
    const uint32_t tiles = (n + FT_TILE - 1) / FT_TILE;
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint32_t b = t * FT_TILE, end = min(b + FT_TILE, n);  // n < 2^31
        volatile K* key = s_keys + FT_HALO;                         // key[(int)(i - b)]: key i
        auto at = [&](uint32_t i) -> K { return key[(int)(i - b)]; };
        auto joined = [&](uint32_t i) { return (at(i - 1) >> lo) == (at(i) >> lo); };
        for (uint32_t j = threadIdx.x; j < FT_TILE + 2 * FT_HALO; j += 256) {
            const uint32_t i = b + j - FT_HALO;  // wraps before the first key
            s_keys[j] = i < n ? p.a.xf(p.a.out_keys[i]) : K(0);
        }
        if (threadIdx.x == 0) s_runs = 0;
        __syncthreads();
        // bit r: key b + 256 r + threadIdx.x is the first fault of a short run inside the tile; a fault of a long run
        uint32_t mine = 0, far = 0;
#pragma unroll 4
        for (int r = 0; r < FT_ROWS; ++r) {
            const uint32_t i = b + r * 256 + threadIdx.x;
            if (i >= end || i == 0 || at(i - 1) <= at(i)) continue;
            uint32_t h = i - 1, e = i + 1;  // towards the run's first key, and past its last
            bool first = true;
            while (first && h > 0 && i - h <= REACH && joined(h)) {
                if (at(h - 1) > at(h)) first = false;
                --h;
            }
            if (!first) continue;  // an earlier fault stands for the run
            while (e < n && e - i <= REACH && joined(e)) ++e;
            if (i - h > REACH || e - i > REACH) far |= 1u << r;
            else if (h >= b && e <= end && e - h > MANY_KEYS) s_run[atomicAdd(&s_runs, 1u)] = ((e - h) << 16) | (h - b);
            else if (h >= b && e <= end) mine |= 1u << r;
            else p.fault[atomicAdd(&p.ctl->faults, 1u)] = i;
        }
        for (; far != 0; far &= far - 1) note_long_run(p, out, b + (__ffs(far) - 1) * 256 + threadIdx.x);
        __syncthreads();  // every run is known before any is changed
        for (uint32_t r = threadIdx.x >> 5; r < s_runs; r += 8) {
            const uint32_t h = b + (s_run[r] & 0xFFFFu), count = s_run[r] >> 16;
            const K* run = s_keys + FT_HALO + (h - b);
            K x[2];
            uint32_t rank[2], v[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const uint32_t self = q * 32 + (threadIdx.x & 31);
                x[q] = self < count ? at(h + self) : K(0);
                v[q] = HAS_V && self < count ? p.a.out_vals[h + self] : 0u;
                // a run's keys stay where they are until its warp writes them out
                if (q * 32 < count) rank[q] = stable_rank(x[q], self, count, [&](uint32_t j) { return run[j]; });
            }
            __syncwarp();  // every value is read before any is written
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (q * 32 + (threadIdx.x & 31) >= count) continue;
                p.a.out_keys[h + rank[q]] = tile::undo_xform(p.a.xf, x[q]);
                if (HAS_V) p.a.out_vals[h + rank[q]] = v[q];
            }
        }
        for (; mine != 0; mine &= mine - 1) {
            const uint32_t i = b + (__ffs(mine) - 1) * 256 + threadIdx.x;
            uint32_t h = i - 1, j = i;
            while (h > b && joined(h)) --h;
            const K top = at(i) >> lo;
            for (; j < end; ++j) {
                const K x = at(j);
                if ((x >> lo) != top) break;
                uint32_t m = j;
                while (m > h && at(m - 1) > x) --m;
                if (m == j) continue;
                const uint32_t v = HAS_V ? p.a.out_vals[j] : 0u;
                for (uint32_t q = j; q > m; --q) {
                    key[(int)(q - b)] = at(q - 1);
                    if (HAS_V) p.a.out_vals[q] = p.a.out_vals[q - 1];
                }
                key[(int)(m - b)] = x;
                if (HAS_V) p.a.out_vals[m] = v;
            }
            for (uint32_t q = h; q < j; ++q) p.a.out_keys[q] = tile::undo_xform(p.a.xf, at(q));
        }
        __syncthreads();
    }
}

// The listed short runs, one warp each, on the output arrays; `warp` of `warps`.
template <typename K, bool HAS_V> __device__ __forceinline__ void repair_listed(const Args<K>& p, uint32_t warp, uint32_t warps)
{
    const uint32_t lo = p.ctl->lowest;
    const Output<K> out{p.a.out_keys, p.a.xf, p.a.n, lo};
    const uint32_t faults = p.ctl->faults, lane = threadIdx.x & 31;
    for (uint32_t f = warp; f < faults; f += warps) {
        const uint32_t i = p.fault[f];
        const K top = out.at(i) >> lo;
        // fewer than 32 keys to either side
        const bool before = lane < i && (out.at(i - 1 - lane) >> lo) == top;
        const bool after = lane < p.a.n - i && (out.at(i + lane) >> lo) == top;
        const uint32_t h = i - __popc(__ballot_sync(FULL_MASK, before));
        const uint32_t count = i + __popc(__ballot_sync(FULL_MASK, after)) - h;
        K x[2];
        uint32_t rank[2], v[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const bool in = q * 32 + lane < count;
            x[q] = in ? out.at(h + q * 32 + lane) : K(0);
            v[q] = HAS_V && in ? p.a.out_vals[h + q * 32 + lane] : 0u;
        }
        __syncwarp();  // every value is read before any is written
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const uint32_t self = q * 32 + lane;
            if (q * 32 >= count) break;
            rank[q] = stable_rank(x[q], self, count, [&](uint32_t j) {
                const K a = __shfl_sync(FULL_MASK, x[0], j & 31), b = __shfl_sync(FULL_MASK, x[1], j & 31);
                return j < 32 ? a : b;
            });
            if (self >= count) continue;
            p.a.out_keys[h + rank[q]] = tile::undo_xform(p.a.xf, x[q]);
            if (HAS_V) p.a.out_vals[h + rank[q]] = v[q];
        }
    }
}

template <typename K, bool HAS_V> __global__ void __launch_bounds__(256) k_repair(Args<K> p)
{
    dev::chain();
    repair_listed<K, HAS_V>(p, (blockIdx.x * 256 + threadIdx.x) / 32, gridDim.x * 8);
}

// One CTA: the long runs in order of position become the even segments of an
// offset array (the odd ones are the keys between them); unused ones are empty.
// After an overflow there are none, and the plan of all digits is put in force.
__global__ void __launch_bounds__(1024) k_long_runs(Control* ctl, SortControl* all, const uint32_t* begin,
                                                    const uint32_t* end, uint32_t* off, uint32_t* skip, uint32_t n, int* err)
{
    dev::chain();
    // a byte per segment: the odd ones are left alone
    for (uint32_t i = threadIdx.x; i < 2 * MAX_LONG / 4; i += 1024) skip[i] = 0x01000100u;
    constexpr int ITEMS = MAX_LONG / 1024;
    using S = tile::Sorter<uint32_t, true, 1024, ITEMS>;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ tile::Scratch<1024> scratch;
    const bool over = ctl->overflow != 0;
    const uint32_t runs = over ? 0u : min(ctl->long_runs, MAX_LONG);
    if (over && threadIdx.x == 0) all->plan.num_active = ctl->later;
    for (uint32_t i = runs + threadIdx.x; i < MAX_LONG; i += 1024) off[2 * i] = off[2 * i + 1] = n;
    if (runs == 0) return;
    S st(smem, scratch);
    st.len = runs;
    st.rows = (runs + 1023) / 1024;
    uint32_t key[ITEMS], val[ITEMS];
    const uint32_t i0 = st.first_index();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const uint32_t at = i0 + i * 16;
        const bool in = i < (int)st.rows && at < runs;
        key[i] = in ? begin[at] : 0u;
        val[i] = in ? end[at] : 0u;
    }
    if (!st.sort(key, val) && threadIdx.x == 0) dev::raise_error(err, dev::ERR_MISPLACED);
    for (uint32_t i = threadIdx.x; i < runs; i += 1024) {
        off[2 * i] = st.keys[i];
        off[2 * i + 1] = st.vals[i];
    }
}

// The listed short runs, and the long ones, where there is no segmented sort
// behind: one CTA each. One that fits no CTA sends the array through all its digits.
template <typename K, bool HAS_V> __global__ void __launch_bounds__(512, 1) k_sort_long_runs(Args<K> p, int* err)
{
    dev::chain();
    using S = tile::Sorter<K, HAS_V, 512, 16>;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ tile::Scratch<512> scratch;
    Control* ctl = p.ctl;
    repair_listed<K, HAS_V>(p, (blockIdx.x * 512 + threadIdx.x) / 32, gridDim.x * 16);
    bool over = ctl->overflow != 0;
    const uint32_t runs = min(ctl->long_runs, MAX_LONG);
    S st(smem, scratch);
    for (uint32_t r = blockIdx.x; r < runs; r += gridDim.x) {
        const uint32_t b = p.begin[r], len = p.end[r] - b;
        if (len > (uint32_t)S::CAP) {
            over = true;
            continue;
        }
        st.len = len;
        st.rows = (len + 511) / 512;
        const uint32_t i0 = st.first_index();
        K key[16];
        uint32_t val[HAS_V ? 16 : 1];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const uint32_t at = i0 + i * 16;
            const bool in = i < (int)st.rows && at < len;
            key[i] = in ? p.a.xf(p.a.out_keys[b + at]) : K(0);
            if (HAS_V) val[i] = in ? p.a.out_vals[b + at] : 0u;
        }
        if (!st.sort(key, val) && threadIdx.x == 0) dev::raise_error(err, dev::ERR_MISPLACED);
        for (uint32_t i = threadIdx.x; i < len; i += 512) {
            p.a.out_keys[b + i] = tile::undo_xform(p.a.xf, st.keys[i]);
            if (HAS_V) p.a.out_vals[b + i] = st.vals[i];
        }
        __syncthreads();
    }
    if (over && threadIdx.x == 0) p.all->plan.num_active = ctl->later;
}

}  // namespace partial
}  // namespace onesweep
}  // namespace gbc
