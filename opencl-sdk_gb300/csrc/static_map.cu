// static_map: a fixed-capacity GPU hash map from 32-bit keys to 32-bit values.
//
// Reference path replaced: cl::compute::static_map (lib/include/CL/Compute/
// HashMap.hpp, lib/src/Compute/HashMap.cpp:16-184) with kernels
// clc_map_insert / clc_map_find / clc_map_contains. Kept, because callers
// observe them: open addressing with linear probing over a power-of-two table
// (capacity rounded up, at least 2, at most 2^31), the MurmurHash3 32-bit
// finalizer as the hash (the reference's clc_hash_u32, DeviceHeaders.cpp:
// 136-145, the published fmix32), empty_key marking free slots and never
// inserted, empty_value returned for missing keys, the first value stored for
// a key kept by later inserts (which count nothing), a probe walk that ends at
// an empty slot, and insert reporting how many keys were new while a full
// table fails the call with the number it could not place.
//
// Here each slot is one 64-bit word, key in the low half and value in the
// high half, claimed with one 64-bit compare-and-swap: a lookup reads one
// word per probe (the reference reads the key array, then the value array),
// and a slot's key and value appear together. Inserted and failed counts are
// aggregated per warp (one atomic per warp instead of one per key). The
// separate key and value arrays of the reference (slot_keys(), slot_values())
// are produced on request by an unzip kernel.
#include <algorithm>
#include <memory>
#include <stdexcept>
#include <string>

#include "device_common.cuh"
#include "runtime.hpp"
#include "sort_internal.hpp"

namespace gbc {
namespace hashmap {

constexpr int THREADS = 256;

__device__ __forceinline__ uint32_t fmix32(uint32_t k)
{
    k ^= k >> 16;
    k *= 0x85ebca6bu;
    k ^= k >> 13;
    k *= 0xc2b2ae35u;
    k ^= k >> 16;
    return k;
}

__device__ __forceinline__ uint64_t pack(uint32_t key, uint32_t value) { return ((uint64_t)value << 32) | key; }

__global__ void __launch_bounds__(THREADS) k_map_fill(unsigned long long* slots, uint64_t count, uint64_t empty)
{
    for (uint64_t i = (uint64_t)blockIdx.x * THREADS + threadIdx.x; i < count; i += (uint64_t)gridDim.x * THREADS)
        slots[i] = empty;
}

// Written by one call, read by the host: zero at its start.
struct Outcome {
    unsigned int added, failed;  // keys newly inserted; keys not placed (table full)
    unsigned int met;            // sampled keys that were there already
};

struct Table {
    unsigned long long* slots;
    uint32_t mask, empty_key, empty_value;
    Outcome* outcome;
};

enum class Found { nothing, added, present, full };

__device__ __forceinline__ Found insert_pair(const Table& t, uint32_t key, uint32_t value)
{
    if (key == t.empty_key) return Found::nothing;
    const unsigned long long empty = pack(t.empty_key, t.empty_value), pair = pack(key, value);
    uint32_t slot = fmix32(key) & t.mask;
    for (uint32_t probe = 0; probe <= t.mask; ++probe) {
        unsigned long long seen = t.slots[slot];
        if ((uint32_t)seen == t.empty_key) seen = atomicCAS(&t.slots[slot], empty, pair);
        if (seen == empty) return Found::added;
        if ((uint32_t)seen == key) return Found::present;  // the first value stays
        slot = (slot + 1) & t.mask;
    }
    return Found::full;
}

// Adds the lanes that found `what` to the counter; every lane of the warp calls it.
__device__ __forceinline__ void count_found(unsigned int* counter, Found f, Found what)
{
    const uint32_t who = __ballot_sync(dev::FULL_MASK, f == what);
    if (who != 0 && (threadIdx.x & 31) == 0) atomicAdd(counter, (unsigned)__popc(who));
}

// Whether the insert by regions (below) is the faster one depends on how many of
// the keys are distinct: the direct insert of a key that is there already is a
// read of a cached line, while the regions' cost is the table's and the keys' size
// (2^24 keys into 2^25 slots, directly and by regions: all distinct 1.00 / 0.54 ms,
// 2^22 values 0.75 / 0.45, 2^20 0.35 / 0.41, 1,000 0.08 / 0.51). So SAMPLE keys are
// inserted first, and those that are there already counted: `least` distinct and
// equally frequent values would give SAMPLE^2 / (2 least) of them. That takes up to
// 15 us where the rest follows directly (2^22 keys into 2^25 slots: 1,000 values 35
// us with and without it, 65,536 69 / 84, 2^20 191 / 203), and without it one value
// repeated 2^24 times took 26 ms for 0.25, Zipf keys 9.2 for 0.17.
constexpr uint32_t SAMPLE = 1u << 15;
constexpr uint32_t DISTINCT_SHARE = 16;  // the lines cross at about capacity / 16 distinct values

__host__ __device__ inline bool mostly_distinct(unsigned int met, uint32_t least)
{
    return (uint64_t)met * 2 * least <= (uint64_t)SAMPLE * SAMPLE;
}

__global__ void __launch_bounds__(THREADS)
    k_map_sample(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ values, uint32_t n, Table t)
{
    const uint32_t i = blockIdx.x * THREADS + threadIdx.x, step = n / SAMPLE;
    const uint32_t at = i * step + fmix32(i) % step;  // a varying place, so that no period of the input is followed
    const Found f = insert_pair(t, keys[at], values[at]);
    count_found(&t.outcome->added, f, Found::added);
    count_found(&t.outcome->met, f, Found::present);
}

// SAMPLED: nothing to do when the sample says that the regions come next.
template <bool SAMPLED>
__global__ void __launch_bounds__(THREADS)
    k_map_insert(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ values, uint32_t n, Table t, uint32_t least)
{
    dev::chain();
    if (SAMPLED && mostly_distinct(*(volatile unsigned int*)&t.outcome->met, least)) return;
    const uint32_t stride = gridDim.x * THREADS;
    const uint32_t rounds = (n + stride - 1) / stride;
    for (uint32_t r = 0; r < rounds; ++r) {
        const uint32_t i = r * stride + blockIdx.x * THREADS + threadIdx.x;
        const Found f = i < n ? insert_pair(t, keys[i], values[i]) : Found::nothing;
        count_found(&t.outcome->added, f, Found::added);
        count_found(&t.outcome->failed, f, Found::full);
    }
}

// ---------------------------------------------------------------------------
// Inserting many keys into a table larger than L2: by regions.
//
// Directly, every key costs one compare-and-swap on a random line of memory
// (2^26 keys into 2^27 slots: 5.3 ms, bound by their rate at L2). Here the pairs
// are first brought into the order of their home slots (two digit passes of the
// library's sort on the hash, whose 32 bits give the key back), and each region
// of 8,192 slots is filled in shared memory: read once, written once. A
// key whose probe leaves the region, or goes on for longer than PROBES slots,
// is inserted directly afterwards; the slots it passed stay full, so the table
// obeys the linear-probing rule as before. (2^26 keys into 2^27 slots: 1.76 ms,
// of which the passes 0.72 and the regions 0.91, whose 2.6 GB would take 0.39;
// more pairs on their way per thread, 4 or 8, took 0.99 and 1.26 ms, regions of
// 4,096 slots 0.85 to 0.87.)
// ---------------------------------------------------------------------------
constexpr uint32_t REGION_BITS = 13, REGION = 1u << REGION_BITS;
constexpr int REGION_THREADS = 512;
constexpr uint32_t PROBES = 64;
// A region given more pairs than this (keys repeated very often) would keep one
// CTA busy long after the others: its pairs are inserted directly, by all of them.
constexpr uint32_t REGION_PAIRS = 4 * REGION;

__device__ __forceinline__ uint32_t undo_fmix32(uint32_t k)
{
    k ^= k >> 16;
    k *= 0x7ed1b41du;  // the inverse of 0xc2b2ae35 modulo 2^32
    k ^= k >> 13 ^ k >> 26;
    k *= 0xa5cb9243u;  // the inverse of 0x85ebca6b
    k ^= k >> 16;
    return k;
}

// The hash rotated so that its home slot's bits lead: hashed[i], and the counts
// of its two highest digits; the last CTA makes them the plan of two passes.
__global__ void __launch_bounds__(THREADS) k_map_hash(const uint32_t* __restrict__ keys, uint32_t n, int rotate,
                                                     uint32_t* __restrict__ hashed, onesweep::SortControl* ctl)
{
    __shared__ uint32_t s_hist[4][2][256];  // per pair of warps
    __shared__ uint32_t s_scratch[8];
    __shared__ int s_last;
    const int tid = threadIdx.x;
    for (int i = tid; i < 4 * 2 * 256; i += THREADS) (&s_hist[0][0][0])[i] = 0;
    __syncthreads();
    uint32_t(*h)[256] = s_hist[tid >> 6];
    const uint32_t stride = gridDim.x * THREADS;
    auto one = [&](uint32_t key) {
        const uint32_t x = fmix32(key), r = __funnelshift_l(x, x, rotate);
        atomicAdd(&h[0][r >> 16 & 0xFF], 1u);
        atomicAdd(&h[1][r >> 24], 1u);
        return r;
    };
    uint32_t i = blockIdx.x * THREADS + tid;
    for (; (uint64_t)i + 3ull * stride < n; i += 4 * stride) {
        uint32_t k[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) k[q] = keys[i + q * stride];
#pragma unroll
        for (int q = 0; q < 4; ++q) hashed[i + q * stride] = one(k[q]);
    }
    for (; i < n; i += stride) hashed[i] = one(keys[i]);
    __syncthreads();
    for (int d = 0; d < 2; ++d) {
        const uint32_t c = s_hist[0][d][tid] + s_hist[1][d][tid] + s_hist[2][d][tid] + s_hist[3][d][tid];
        if (c != 0) atomicAdd(&ctl->hist[d][tid], c);
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(&ctl->done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int d = 0; d < 2; ++d)
        ctl->plan.bin_start[d][tid] = dev::bins_exclusive_sum(dev::ld_relaxed(&ctl->hist[d][tid]), s_scratch);
    if (tid < 2) ctl->plan.shift[tid] = 16 + 8 * tid;
    if (tid == 0) ctl->plan.num_active = 2;
}

// first[r] = the first pair of region r or a later one (regions + 1 entries).
__global__ void __launch_bounds__(THREADS)
    k_map_regions(const uint32_t* __restrict__ hashed, uint32_t n, int shift, uint32_t regions, uint32_t* __restrict__ first)
{
    for (uint32_t i = blockIdx.x * THREADS + threadIdx.x; i <= n; i += gridDim.x * THREADS) {
        const uint32_t after = i < n ? hashed[i] >> shift : regions;
        const uint32_t before = i > 0 ? (hashed[i - 1] >> shift) + 1 : 0;
        for (uint32_t r = before; r <= after; ++r) first[r] = i;
    }
}

// What the region kernel leaves to direct inserts.
struct Rest {
    uint32_t *keys, *values;  // pairs
    uint32_t* count;          // how many, and how many regions
    uint32_t* regions;        // those with more than REGION_PAIRS
};

__global__ void __launch_bounds__(REGION_THREADS, 3)
    k_map_fill_regions(const uint32_t* __restrict__ hashed, const uint32_t* __restrict__ values, int rotate,
                       const uint32_t* __restrict__ first, uint32_t regions, Table t, Rest rest)
{
    extern __shared__ __align__(16) unsigned char smem[];
    volatile unsigned long long* region = reinterpret_cast<volatile unsigned long long*>(smem);
    const unsigned long long empty = pack(t.empty_key, t.empty_value);
    const int tid = threadIdx.x, lane = tid & 31;
    uint32_t added = 0;
    auto leave = [&](bool mine, uint32_t key, uint32_t value) {  // every lane of the warp
        const uint32_t who = __ballot_sync(dev::FULL_MASK, mine);
        if (who == 0) return;
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(&rest.count[0], (uint32_t)__popc(who));
        at = __shfl_sync(dev::FULL_MASK, at, 0) + __popc(who & dev::lanemask_lt());
        if (mine) {
            rest.keys[at] = key;
            rest.values[at] = value;
        }
    };
    for (uint32_t r = blockIdx.x; r < regions; r += gridDim.x) {
        const uint32_t b = first[r], e = first[r + 1];
        if (b == e) continue;
        if (e - b > REGION_PAIRS) {
            if (tid == 0) rest.regions[atomicAdd(&rest.count[1], 1u)] = r;
            continue;
        }
        // the first pairs are on their way while the region is read
        constexpr int AHEAD = 2;
        uint32_t x[AHEAD], v[AHEAD];
        auto fetch = [&](uint32_t i0) {
#pragma unroll
            for (int q = 0; q < AHEAD; ++q) {
                const uint32_t i = i0 + q * REGION_THREADS + tid;
                x[q] = i < e ? hashed[i] : 0u;
                v[q] = i < e ? values[i] : 0u;
            }
        };
        fetch(b);
        uint4* mem = reinterpret_cast<uint4*>(t.slots + (size_t)r * REGION);
        uint4* copy = reinterpret_cast<uint4*>(smem);
#pragma unroll
        for (uint32_t i = 0; i < REGION / 2 / REGION_THREADS; ++i)
            copy[i * REGION_THREADS + tid] = dev::ld_stream(mem + i * REGION_THREADS + tid);
        __syncthreads();
        for (uint32_t i0 = b; i0 < e; i0 += AHEAD * REGION_THREADS) {
            if (i0 != b) fetch(i0);
            uint32_t left = 0;  // bit q: pair q is not placed here
#pragma unroll
            for (int q = 0; q < AHEAD; ++q) {
                const uint32_t h = __funnelshift_r(x[q], x[q], rotate);
                const uint32_t key = undo_fmix32(h);
                if (i0 + q * REGION_THREADS + tid >= e || key == t.empty_key) continue;
                const unsigned long long mine = pack(key, v[q]);
                uint32_t slot = h & (REGION - 1);
                bool placed = false;
                for (uint32_t p = 0; p < PROBES && slot < REGION; ++p, ++slot) {
                    unsigned long long seen = region[slot];
                    if ((uint32_t)seen == t.empty_key)
                        seen = atomicCAS(const_cast<unsigned long long*>(&region[slot]), empty, mine);
                    if (seen == empty) ++added;
                    if (seen == empty || (uint32_t)seen == key) {  // placed, or present: the first value stays
                        placed = true;
                        break;
                    }
                }
                if (!placed) left |= 1u << q;
            }
            if (__any_sync(dev::FULL_MASK, left != 0)) {
#pragma unroll
                for (int q = 0; q < AHEAD; ++q)
                    leave(left >> q & 1u, undo_fmix32(__funnelshift_r(x[q], x[q], rotate)), v[q]);
            }
        }
        __syncthreads();
#pragma unroll
        for (uint32_t i = 0; i < REGION / 2 / REGION_THREADS; ++i)
            mem[i * REGION_THREADS + tid] = copy[i * REGION_THREADS + tid];
        __syncthreads();
    }
    added = __reduce_add_sync(dev::FULL_MASK, added);
    if (lane == 0 && added != 0) atomicAdd(&t.outcome->added, added);
}

// The direct inserts: the pairs that left their region, then the regions left whole.
__global__ void __launch_bounds__(THREADS)
    k_map_insert_rest(const uint32_t* __restrict__ hashed, const uint32_t* __restrict__ values, int rotate,
                      const uint32_t* __restrict__ first, Table t, Rest rest)
{
    const uint32_t stride = gridDim.x * THREADS;
    const uint32_t n = rest.count[0], whole = rest.count[1];
    for (uint32_t i0 = blockIdx.x * THREADS; i0 < n; i0 += stride) {
        const uint32_t i = i0 + threadIdx.x;
        const Found f = i < n ? insert_pair(t, rest.keys[i], rest.values[i]) : Found::nothing;
        count_found(&t.outcome->added, f, Found::added);
        count_found(&t.outcome->failed, f, Found::full);
    }
    for (uint32_t w = 0; w < whole; ++w) {
        const uint32_t r = rest.regions[w], e = first[r + 1];
        for (uint32_t i0 = first[r] + (blockIdx.x + w) % gridDim.x * THREADS; i0 < e; i0 += stride) {
            const uint32_t i = i0 + threadIdx.x, x = i < e ? hashed[i] : 0u;
            const Found f = i < e ? insert_pair(t, undo_fmix32(__funnelshift_r(x, x, rotate)), values[i]) : Found::nothing;
            count_found(&t.outcome->added, f, Found::added);
            count_found(&t.outcome->failed, f, Found::full);
        }
    }
}

// The slot holding key, or mask + 1 when absent (the walk ends at an empty slot).
__device__ __forceinline__ uint64_t probe(const unsigned long long* __restrict__ slots, uint32_t mask, uint32_t key,
                                          uint32_t empty_key, uint32_t& value)
{
    if (key == empty_key) return (uint64_t)mask + 1;
    uint32_t slot = fmix32(key) & mask;
    for (uint32_t p = 0; p <= mask; ++p) {
        const unsigned long long w = __ldg(slots + slot);
        if ((uint32_t)w == key) {
            value = (uint32_t)(w >> 32);
            return slot;
        }
        if ((uint32_t)w == empty_key) break;
        slot = (slot + 1) & mask;
    }
    return (uint64_t)mask + 1;
}

__global__ void __launch_bounds__(THREADS)
    k_map_find(const uint32_t* __restrict__ keys, uint32_t n, const unsigned long long* __restrict__ slots,
               uint32_t mask, uint32_t empty_key, uint32_t empty_value, uint32_t* __restrict__ out)
{
    for (uint32_t i = blockIdx.x * THREADS + threadIdx.x; i < n; i += gridDim.x * THREADS) {
        uint32_t v = empty_value;
        probe(slots, mask, keys[i], empty_key, v);
        out[i] = v;
    }
}

__global__ void __launch_bounds__(THREADS)
    k_map_contains(const uint32_t* __restrict__ keys, uint32_t n, const unsigned long long* __restrict__ slots,
                   uint32_t mask, uint32_t empty_key, uint8_t* __restrict__ out)
{
    for (uint32_t i = blockIdx.x * THREADS + threadIdx.x; i < n; i += gridDim.x * THREADS) {
        uint32_t v = 0;
        out[i] = probe(slots, mask, keys[i], empty_key, v) <= mask ? 1 : 0;
    }
}

__global__ void __launch_bounds__(THREADS)
    k_map_unzip(const unsigned long long* __restrict__ slots, uint64_t count, uint32_t* __restrict__ keys,
                uint32_t* __restrict__ values)
{
    for (uint64_t i = (uint64_t)blockIdx.x * THREADS + threadIdx.x; i < count; i += (uint64_t)gridDim.x * THREADS) {
        const unsigned long long w = slots[i];
        if (keys != nullptr) keys[i] = (uint32_t)w;
        if (values != nullptr) values[i] = (uint32_t)(w >> 32);
    }
}

int grid(device_context& ctx, uint64_t work)
{
    return (int)std::max<uint64_t>(1, std::min<uint64_t>((work + THREADS - 1) / THREADS, (uint64_t)ctx.sm_count * 8));
}

// 2^24 slots are 128 MB, about L2; two 8-bit digits order at most 2^16 regions.
constexpr std::size_t REGION_MIN_SLOTS = std::size_t(1) << 25, REGION_MAX_SLOTS = std::size_t(REGION) << 16;

// Enqueues the insert by regions; false when there is no memory for its scratch.
bool insert_by_regions(device_context& ctx, const Table& t, std::size_t capacity, const uint32_t* keys, const uint32_t* values,
                       uint32_t n)
{
    int bits = 0;
    while ((std::size_t(1) << bits) < capacity) ++bits;
    const int rotate = 32 - bits, shift = 32 - (bits - (int)REGION_BITS);
    const uint32_t regions = (uint32_t)(capacity / REGION);
    const std::size_t words = ((std::size_t)n + 63) / 64 * 64;
    const std::size_t whole = (n / REGION_PAIRS + 63) / 64 * 64;
    std::unique_ptr<temp_buffer> scratch;
    try {
        scratch = std::make_unique<temp_buffer>(ctx.resource,
                                                (4 * words + regions + 64 + whole) * 4 + sizeof(onesweep::SortControl));
    } catch (const out_of_memory&) {
        return false;
    }
    uint32_t* hashed = scratch->as<uint32_t>();
    uint32_t *alt_hashed = hashed + words, *ordered = hashed + 2 * words, *alt_values = hashed + 3 * words;
    uint32_t* first = hashed + 4 * words;  // regions + 1, then the rest's two counts
    Rest rest{alt_hashed, alt_values, first + regions + 1, first + regions + 64};
    auto* ctl = reinterpret_cast<onesweep::SortControl*>(rest.regions + whole);
    check_cuda(cudaMemsetAsync(rest.count, 0, 8, ctx.stream), "cudaMemsetAsync");
    check_cuda(cudaMemsetAsync(ctl, 0, sizeof(onesweep::SortControl), ctx.stream), "cudaMemsetAsync");
    {
        kernel_timer kt(ctx, "static_map.hash");
        k_map_hash<<<ctx.sm_count * 8, THREADS, 0, ctx.stream>>>(keys, n, rotate, hashed, ctl);
        check_cuda(cudaGetLastError(), "static_map hash launch");
    }
    radix_passes_pairs(ctx, hashed, hashed, alt_hashed, values, ordered, alt_values, n, ctl, 2);
    {
        kernel_timer kt(ctx, "static_map.regions");
        k_map_regions<<<ctx.sm_count * 8, THREADS, 0, ctx.stream>>>(hashed, n, shift, regions, first);
        constexpr std::size_t smem = (std::size_t)REGION * 8;
        if (first_use_on_device((const void*)&k_map_fill_regions))
            check_cuda(cudaFuncSetAttribute(&k_map_fill_regions, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                       "cudaFuncSetAttribute");
        // the ordered pairs are read, so the passes' other buffers take the rest
        k_map_fill_regions<<<ctx.sm_count * 3, REGION_THREADS, smem, ctx.stream>>>(hashed, ordered, rotate, first, regions, t,
                                                                                   rest);
        check_cuda(cudaGetLastError(), "static_map region launch");
    }
    {
        kernel_timer kt(ctx, "static_map.insert");
        k_map_insert_rest<<<grid(ctx, n), THREADS, 0, ctx.stream>>>(hashed, ordered, rotate, first, t, rest);
        check_cuda(cudaGetLastError(), "static_map insert launch");
    }
    return true;
}

}  // namespace hashmap

std::size_t static_map_slots(std::size_t capacity)
{
    if (capacity > (std::size_t(1) << 31)) throw std::length_error("static_map: capacity above 2^31");
    std::size_t c = 2;
    while (c < capacity) c <<= 1;
    return c;
}

void static_map_clear(device_context& ctx, void* slots, std::size_t capacity, uint32_t empty_key,
                      uint32_t empty_value)
{
    using namespace hashmap;
    ctx.activate();
    kernel_timer kt(ctx, "static_map.clear");
    k_map_fill<<<grid(ctx, capacity), THREADS, 0, ctx.stream>>>(static_cast<unsigned long long*>(slots), capacity,
                                                              ((uint64_t)empty_value << 32) | empty_key);
    check_cuda(cudaGetLastError(), "static_map clear launch");
}

std::size_t static_map_insert(device_context& ctx, void* slots, std::size_t capacity, uint32_t empty_key,
                              uint32_t empty_value, const uint32_t* keys, const uint32_t* values, std::size_t n,
                              std::size_t& not_placed)
{
    using namespace hashmap;
    not_placed = 0;
    if (n == 0) return 0;
    check_size(n);
    if (keys == nullptr || values == nullptr) throw std::invalid_argument("static_map::insert: null keys or values");
    ctx.activate();
    auto* o = reinterpret_cast<Outcome*>(ctx.d_small);
    check_cuda(cudaMemsetAsync(o, 0, sizeof(Outcome), ctx.stream), "cudaMemsetAsync");
    const Table t{static_cast<unsigned long long*>(slots), (uint32_t)(capacity - 1), empty_key, empty_value, o};
    // By regions where the table is larger than L2 and the keys are dense in
    // it (a region is read and written whole for its share of the keys):
    // into 2^26 slots, directly and by regions, capacity / 16 keys 0.29 / 0.31
    // ms, / 8 0.57 / 0.36, / 2 2.43 / 0.96; and where enough of them are distinct,
    // which the host learns with the direct insert's counts.
    const bool dense = capacity >= REGION_MIN_SLOTS && capacity <= REGION_MAX_SLOTS && n >= capacity / 8;
    const uint32_t least = (uint32_t)(capacity / DISTINCT_SHARE);
    auto* h = static_cast<Outcome*>(ctx.pinned);
    auto read = [&] {
        check_cuda(cudaMemcpyAsync(h, o, sizeof(Outcome), cudaMemcpyDeviceToHost, ctx.stream), "cudaMemcpyAsync");
        check_cuda(cudaStreamSynchronize(ctx.stream), "cudaStreamSynchronize");
    };
    auto direct = [&](auto kernel) {
        kernel_timer kt(ctx, "static_map.insert");
        launch_chained(kernel, grid(ctx, n), THREADS, 0, ctx.stream, keys, values, (uint32_t)n, t, least);
        check_cuda(cudaGetLastError(), "static_map insert launch");
    };
    if (dense) {
        {
            kernel_timer kt(ctx, "static_map.sample");
            k_map_sample<<<SAMPLE / THREADS, THREADS, 0, ctx.stream>>>(keys, values, (uint32_t)n, t);
            check_cuda(cudaGetLastError(), "static_map sample launch");
        }
        direct(&k_map_insert<true>);
        read();
        if (mostly_distinct(h->met, least)) {
            if (!insert_by_regions(ctx, t, capacity, keys, values, (uint32_t)n)) direct(&k_map_insert<false>);
            read();
        }
    } else {
        direct(&k_map_insert<false>);
        read();
    }
    not_placed = h->failed;
    return h->added;
}

void static_map_find(device_context& ctx, const void* slots, std::size_t capacity, uint32_t empty_key,
                     uint32_t empty_value, const uint32_t* keys, std::size_t n, uint32_t* out)
{
    using namespace hashmap;
    if (n == 0) return;
    check_size(n);
    if (keys == nullptr || out == nullptr) throw std::invalid_argument("static_map::find: null argument");
    ctx.activate();
    kernel_timer kt(ctx, "static_map.find");
    k_map_find<<<grid(ctx, n), THREADS, 0, ctx.stream>>>(keys, (uint32_t)n,
                                                        static_cast<const unsigned long long*>(slots),
                                                        (uint32_t)(capacity - 1), empty_key, empty_value, out);
    check_cuda(cudaGetLastError(), "static_map find launch");
}

void static_map_contains(device_context& ctx, const void* slots, std::size_t capacity, uint32_t empty_key,
                         const uint32_t* keys, std::size_t n, uint8_t* out)
{
    using namespace hashmap;
    if (n == 0) return;
    check_size(n);
    if (keys == nullptr || out == nullptr) throw std::invalid_argument("static_map::contains: null argument");
    ctx.activate();
    kernel_timer kt(ctx, "static_map.contains");
    k_map_contains<<<grid(ctx, n), THREADS, 0, ctx.stream>>>(keys, (uint32_t)n,
                                                            static_cast<const unsigned long long*>(slots),
                                                            (uint32_t)(capacity - 1), empty_key, out);
    check_cuda(cudaGetLastError(), "static_map contains launch");
}

void static_map_unzip(device_context& ctx, const void* slots, std::size_t capacity, uint32_t* keys, uint32_t* values)
{
    using namespace hashmap;
    ctx.activate();
    kernel_timer kt(ctx, "static_map.unzip");
    k_map_unzip<<<grid(ctx, capacity), THREADS, 0, ctx.stream>>>(static_cast<const unsigned long long*>(slots),
                                                               capacity, keys, values);
    check_cuda(cudaGetLastError(), "static_map unzip launch");
}

}  // namespace gbc
