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

// counters[0]: keys newly inserted, counters[1]: keys not placed (table full)
__global__ void __launch_bounds__(THREADS)
    k_map_insert(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ values, uint32_t n,
                 unsigned long long* slots, uint32_t mask, uint32_t empty_key, uint32_t empty_value,
                 unsigned int* counters, const uint32_t* n_device)
{
    if (n_device != nullptr) n = *n_device;  // at most n
    const unsigned long long empty = pack(empty_key, empty_value);
    const uint32_t stride = gridDim.x * THREADS;
    const uint32_t rounds = (n + stride - 1) / stride;
    const int lane = threadIdx.x & 31;
    for (uint32_t r = 0; r < rounds; ++r) {
        const uint32_t i = r * stride + blockIdx.x * THREADS + threadIdx.x;
        bool added = false, failed = false;
        if (i < n) {
            const uint32_t key = keys[i];
            if (key != empty_key) {
                const unsigned long long mine = pack(key, values[i]);
                uint32_t slot = fmix32(key) & mask;
                failed = true;
                for (uint32_t probe = 0; probe <= mask; ++probe) {
                    unsigned long long seen = slots[slot];
                    if ((uint32_t)seen == empty_key) seen = atomicCAS(&slots[slot], empty, mine);
                    if (seen == empty) {
                        added = true, failed = false;
                        break;
                    }
                    if ((uint32_t)seen == key) {  // present: the first value stays
                        failed = false;
                        break;
                    }
                    slot = (slot + 1) & mask;
                }
            }
        }
        const uint32_t a = __ballot_sync(dev::FULL_MASK, added), f = __ballot_sync(dev::FULL_MASK, failed);
        if (lane == 0) {
            if (a) atomicAdd(&counters[0], (unsigned)__popc(a));
            if (f) atomicAdd(&counters[1], (unsigned)__popc(f));
        }
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
// A region given more pairs than this is not worth one CTA's time (a few keys
// repeated very often): they are inserted directly.
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

// counters: as k_map_insert; rest: pairs left over for it, rest_count of them.
__global__ void __launch_bounds__(REGION_THREADS, 3)
    k_map_fill_regions(const uint32_t* __restrict__ hashed, const uint32_t* __restrict__ values, int rotate,
                       const uint32_t* __restrict__ first, uint32_t regions, unsigned long long* slots, uint32_t empty_key,
                       uint32_t empty_value, unsigned int* counters, uint32_t* rest_keys, uint32_t* rest_values,
                       uint32_t* rest_count)
{
    extern __shared__ __align__(16) unsigned char smem[];
    volatile unsigned long long* region = reinterpret_cast<volatile unsigned long long*>(smem);
    const unsigned long long empty = pack(empty_key, empty_value);
    const int tid = threadIdx.x, lane = tid & 31;
    uint32_t added = 0;
    auto leave = [&](bool mine, uint32_t key, uint32_t value) {  // every lane of the warp
        const uint32_t who = __ballot_sync(dev::FULL_MASK, mine);
        if (who == 0) return;
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(rest_count, (uint32_t)__popc(who));
        at = __shfl_sync(dev::FULL_MASK, at, 0) + __popc(who & dev::lanemask_lt());
        if (mine) {
            rest_keys[at] = key;
            rest_values[at] = value;
        }
    };
    for (uint32_t r = blockIdx.x; r < regions; r += gridDim.x) {
        const uint32_t b = first[r], e = first[r + 1];
        if (b == e) continue;
        const bool direct = e - b > REGION_PAIRS;
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
        uint4* mem = reinterpret_cast<uint4*>(slots + (size_t)r * REGION);
        uint4* copy = reinterpret_cast<uint4*>(smem);
        if (!direct) {
#pragma unroll
            for (uint32_t i = 0; i < REGION / 2 / REGION_THREADS; ++i)
                copy[i * REGION_THREADS + tid] = dev::ld_stream(mem + i * REGION_THREADS + tid);
        }
        __syncthreads();
        for (uint32_t i0 = b; i0 < e; i0 += AHEAD * REGION_THREADS) {
            if (i0 != b) fetch(i0);
            uint32_t left = 0;  // bit q: pair q is not placed here
#pragma unroll
            for (int q = 0; q < AHEAD; ++q) {
                const uint32_t h = __funnelshift_r(x[q], x[q], rotate);
                const uint32_t key = undo_fmix32(h);
                if (i0 + q * REGION_THREADS + tid >= e || key == empty_key) continue;
                const unsigned long long mine = pack(key, v[q]);
                uint32_t slot = h & (REGION - 1);
                bool placed = false;
                for (uint32_t p = 0; !direct && p < PROBES && slot < REGION; ++p, ++slot) {
                    unsigned long long seen = region[slot];
                    if ((uint32_t)seen == empty_key)
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
        if (!direct) {
#pragma unroll
            for (uint32_t i = 0; i < REGION / 2 / REGION_THREADS; ++i)
                mem[i * REGION_THREADS + tid] = copy[i * REGION_THREADS + tid];
        }
        __syncthreads();
    }
    added = __reduce_add_sync(dev::FULL_MASK, added);
    if (lane == 0 && added != 0) atomicAdd(&counters[0], added);
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
bool insert_by_regions(device_context& ctx, unsigned long long* slots, std::size_t capacity, uint32_t empty_key,
                       uint32_t empty_value, const uint32_t* keys, const uint32_t* values, uint32_t n,
                       unsigned int* counters)
{
    int bits = 0;
    while ((std::size_t(1) << bits) < capacity) ++bits;
    const int rotate = 32 - bits, shift = 32 - (bits - (int)REGION_BITS);
    const uint32_t regions = (uint32_t)(capacity / REGION);
    const std::size_t words = ((std::size_t)n + 63) / 64 * 64;
    std::unique_ptr<temp_buffer> scratch;
    try {
        scratch = std::make_unique<temp_buffer>(ctx.resource, (4 * words + regions + 64) * 4 + sizeof(onesweep::SortControl));
    } catch (const out_of_memory&) {
        return false;
    }
    uint32_t* hashed = scratch->as<uint32_t>();
    uint32_t *alt_hashed = hashed + words, *ordered = hashed + 2 * words, *alt_values = hashed + 3 * words;
    uint32_t* first = hashed + 4 * words;  // regions + 1, then the rest's count
    uint32_t* rest_count = first + regions + 1;
    auto* ctl = reinterpret_cast<onesweep::SortControl*>(first + regions + 64);
    check_cuda(cudaMemsetAsync(rest_count, 0, 4, ctx.stream), "cudaMemsetAsync");
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
        k_map_fill_regions<<<ctx.sm_count * 3, REGION_THREADS, smem, ctx.stream>>>(
            hashed, ordered, rotate, first, regions, slots, empty_key, empty_value, counters, alt_hashed, alt_values,
            rest_count);
        check_cuda(cudaGetLastError(), "static_map region launch");
    }
    {
        kernel_timer kt(ctx, "static_map.insert");
        k_map_insert<<<grid(ctx, n), THREADS, 0, ctx.stream>>>(alt_hashed, alt_values, n, slots, (uint32_t)(capacity - 1),
                                                             empty_key, empty_value, counters, rest_count);
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
    unsigned int* counters = reinterpret_cast<unsigned int*>(ctx.d_small);
    check_cuda(cudaMemsetAsync(counters, 0, 8, ctx.stream), "cudaMemsetAsync");
    // By regions where the table is larger than L2 and the keys are dense in
    // it (a region is read and written whole for its share of the keys):
    // into 2^26 slots, directly and by regions, capacity / 16 keys 0.29 / 0.31
    // ms, / 8 0.57 / 0.36, / 2 2.43 / 0.96.
    bool done = false;
    if (capacity >= REGION_MIN_SLOTS && capacity <= REGION_MAX_SLOTS && n >= capacity / 8)
        done = insert_by_regions(ctx, static_cast<unsigned long long*>(slots), capacity, empty_key, empty_value, keys, values,
                                 (uint32_t)n, counters);
    if (!done) {
        kernel_timer kt(ctx, "static_map.insert");
        k_map_insert<<<grid(ctx, n), THREADS, 0, ctx.stream>>>(keys, values, (uint32_t)n,
                                                             static_cast<unsigned long long*>(slots),
                                                             (uint32_t)(capacity - 1), empty_key, empty_value,
                                                             counters, nullptr);
        check_cuda(cudaGetLastError(), "static_map insert launch");
    }
    unsigned int* h = static_cast<unsigned int*>(ctx.pinned);
    check_cuda(cudaMemcpyAsync(h, counters, 8, cudaMemcpyDeviceToHost, ctx.stream), "cudaMemcpyAsync");
    check_cuda(cudaStreamSynchronize(ctx.stream), "cudaStreamSynchronize");
    not_placed = h[1];
    return h[0];
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
