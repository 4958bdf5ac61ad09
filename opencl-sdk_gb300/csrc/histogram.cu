// histogram_even: counts in[i] into `bins` equal-width bins over [lower, upper).
//
// Reference path replaced: detail::histogram_even (lib/src/Compute/
// Algorithm.cpp:569-615) with kernel clc_histogram (240-273). The bin rule is
// kept operation for operation, because it decides bit-exact parity at bin
// edges: ACC is float unless the input is double; x = (ACC)in[i]; samples
// with !(x >= lower && x < upper) are ignored; b = (uint)((x - lower) * scale)
// with scale = (ACC)bins / (upper - lower) computed on the device in ACC;
// b >= bins is clamped to bins - 1. The histogram is zeroed first.
//
// The reference privatises the histogram in local memory when it fits and
// otherwise uses global atomics. Here: per-warp shared sub-histograms with
// shared atomics when bins x 8 warps fit in 64 KiB, one shared histogram per
// CTA while it fits in the opt-in shared memory, else global atomics; inputs
// are read with 128-bit loads (16 samples per load for u8). For 8- and 16-bit
// integer inputs whose bin rule reduces exactly to value - offset (checked on
// the host over every value of the type), the float arithmetic is skipped.
// (Lane-private 16-bit counters, bank-conflict free but 64 KiB per 4 warps,
// measured slower: occupancy. Four or eight interleaved copies of each
// warp's histogram, lane l counting into copy l % copies, measured no faster
// for 2^30 bytes (0.41 / 0.37 ms against 0.38) and slower for floats: the
// shared atomic instruction rate, not bank conflicts, is the limit.) Many
// bytes are therefore counted in pairs, one atomic for two of them
// (k_histogram_pairs).
#include <cmath>
#include <cstring>
#include <limits>

#include "device_common.cuh"
#include "runtime.hpp"

namespace gbc {
namespace {

constexpr int THREADS = 256;
constexpr int WARPS = THREADS / 32;

enum class mode : int { per_warp = 0, per_cta = 1, global = 2 };

template <typename T, typename ACC, int MODE, bool OFFSET>
__global__ void __launch_bounds__(THREADS)
    k_histogram(const T* __restrict__ in, uint32_t n, uint32_t* __restrict__ hist, uint32_t bins,
                ACC lower, ACC upper, int offset)
{
    constexpr int VEC = 16 / sizeof(T);
    extern __shared__ __align__(16) uint32_t sh[];
    const uint32_t copies = MODE == 0 ? WARPS : 1;
    if (MODE != 2) {
        for (uint32_t i = threadIdx.x; i < bins * copies; i += THREADS) sh[i] = 0;
        __syncthreads();
    }
    uint32_t* target = MODE == 2 ? hist : sh + (MODE == 0 ? (threadIdx.x >> 5) * bins : 0);
    const ACC scale = (ACC)bins / (upper - lower);
    auto count = [&](T v) {
        if (OFFSET) {
            const uint32_t b = (uint32_t)((int)v - offset);
            if (b < bins) atomicAdd(&target[b], 1u);
            return;
        }
        const ACC x = (ACC)v;
        if (x >= lower && x < upper) {
            uint32_t b = (uint32_t)((x - lower) * scale);
            if (b >= bins) b = bins - 1;
            atomicAdd(&target[b], 1u);
        }
    };
    const uint32_t gtid = blockIdx.x * THREADS + threadIdx.x, stride = gridDim.x * THREADS;
    uint32_t head = 0;
    if ((reinterpret_cast<uintptr_t>(in) & 15) == 0) {
        const uint32_t nv = n / VEC;
        const uint4* vin = reinterpret_cast<const uint4*>(in);
        uint32_t v = gtid;
        // four 128-bit loads in flight per thread before they are counted
        for (; (uint64_t)v + 3ull * stride < nv; v += 4 * stride) {
            uint4 w[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) w[q] = dev::ld_stream(vin + v + q * stride);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                T e[VEC];
                memcpy(e, &w[q], 16);
#pragma unroll
                for (int j = 0; j < VEC; ++j) count(e[j]);
            }
        }
        for (; v < nv; v += stride) {
            const uint4 w = dev::ld_stream(vin + v);
            T e[VEC];
            memcpy(e, &w, 16);
#pragma unroll
            for (int j = 0; j < VEC; ++j) count(e[j]);
        }
        head = nv * VEC;
    }
    for (uint32_t i = head + gtid; i < n; i += stride) count(in[i]);
    if (MODE != 2) {
        __syncthreads();
        for (uint32_t b = threadIdx.x; b < bins; b += THREADS) {
            uint32_t s = 0;
            for (uint32_t c = 0; c < copies; ++c) s += sh[c * bins + b];
            if (s != 0) atomicAdd(&hist[b], s);
        }
    }
}

// ---------------------------------------------------------------------------
// Bytes in pairs: one CTA per SM counts its share of the input into 65,536
// 16-bit counters, two to a word (128 KiB), and adds them up by value after
// every batch. The bin rule is applied to the 256 values' totals at the end.
//
// A counter may wrap, and carry into its neighbour: either loses 65,535 or
// 65,536 from the sum of all counters and nothing adds to it, so a batch whose
// counters do not add up to its pairs is counted again, by bytes, into per-warp
// 32-bit histograms, and so is the rest of the CTA's share.
//
// Pairs pay where a warp's words differ. Lanes with equal bytes add 1 to a counter
// together; their pairs' additions (1 or 2^16) meet on one address one after
// another, and so do all that meet in a bank, which the first byte chooses. So
// the warps look at one byte per lane (all of them before the first batch, some
// before the others), and the bytes are counted one by one from where the
// busiest bank makes the pairs the slower way (2^30 bytes, counted singly by k_histogram / always in pairs / now: runs of 256
// equal bytes 279 / 934 / 189 us, 16 values 279 / 336 / 189, normal with a
// deviation of 10 279 / 279 / 244, one value 279 / 204 / 188, uniform 385 / 270 / 267).
//
// 2^30 uniform bytes: 384 -> 269 us (one read at the copy rate 158; loading
// alone takes 150, the pairs' atomics 234, and with the counters' old values
// returned, to see them wrap, 293).
// ---------------------------------------------------------------------------
constexpr int PAIR_THREADS = 1024, PAIR_WARPS = PAIR_THREADS / 32;
constexpr int PAIR_BATCH = 64;   // 16-byte loads per thread in a batch: 524,288 pairs
constexpr std::size_t PAIR_SMEM = 32768 * 4;
// Below, the CTAs' 128 KiB to clear and add up cost too much where the pairs are
// given up (uniform / one value in nine places of ten / constant bytes, by
// k_histogram and here: 2^26, with a first batch in pairs always, 29.7 / 24.3 / 22.7
// and 27.6 / 36.9 / 36.5 us; 2^28 102.6 / 75.6 / 75.9 and 74.0 / 57.8 / 53.6).
constexpr std::size_t PAIR_MIN = std::size_t(1) << 28;

// What counting the warp's lanes' bytes in pairs costs, less what it costs byte by
// byte, in halves of an addition: those that the busiest bank takes, all of a
// counter's pairs or (by 1, as lanes with the same counter add together) one per
// counter, twice. An addition of 1 is about half the work of a pair's, and each
// has about one more around it (from the times above).
__device__ __forceinline__ int pairs_over_bytes(uint32_t byte)
{
    const uint32_t bank = __match_any_sync(dev::FULL_MASK, byte & 31u), same = __match_any_sync(dev::FULL_MASK, byte);
    const uint32_t once = __ballot_sync(dev::FULL_MASK, (int)(threadIdx.x & 31) == __ffs(same) - 1);
    const int pairs = (int)__reduce_max_sync(dev::FULL_MASK, (uint32_t)__popc(bank));
    const int bytes = (int)__reduce_max_sync(dev::FULL_MASK, (uint32_t)__popc(bank & once));
    return 2 * pairs - 2 * bytes - 2;
}

template <typename T> __global__ void __launch_bounds__(PAIR_THREADS, 1)
    k_histogram_pairs(const T* __restrict__ in, uint32_t n, uint32_t* __restrict__ hist, uint32_t bins, float lower, float upper)
{
    extern __shared__ __align__(16) uint32_t sh[];  // pair (a, b): half b / 128 of word (b % 128) * 256 + a
    __shared__ uint32_t s_value[256], s_sum;
    __shared__ int s_cost;  // the sum of pairs_over_bytes so far
    const int tid = threadIdx.x, warp = tid >> 5;
    const uint4* vin = reinterpret_cast<const uint4*>(in);
    const uint32_t nv = n / 16;
    const uint32_t first = (uint32_t)((uint64_t)nv * blockIdx.x / gridDim.x);
    const uint32_t last = (uint32_t)((uint64_t)nv * (blockIdx.x + 1) / gridDim.x);
    if (tid < 256) s_value[tid] = 0;
    if (tid == 0) s_cost = 0;
    auto clear = [&] {
        __syncthreads();
        for (int i = tid; i < (int)(PAIR_SMEM / 16); i += PAIR_THREADS) reinterpret_cast<uint4*>(sh)[i] = make_uint4(0, 0, 0, 0);
        __syncthreads();
    };
    // f(word) for the four words of every vector of [b, e), four loads in flight
    auto words = [&](uint32_t b, uint32_t e, auto f) {
        uint32_t v = b + tid;
        for (; v + 3 * PAIR_THREADS < e; v += 4 * PAIR_THREADS) {
            uint4 w[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) w[q] = dev::ld_stream(vin + v + q * PAIR_THREADS);
#pragma unroll
            for (int q = 0; q < 4; ++q) f(w[q].x), f(w[q].y), f(w[q].z), f(w[q].w);
        }
        for (; v < e; v += PAIR_THREADS) {
            const uint4 w = dev::ld_stream(vin + v);
            f(w.x), f(w.y), f(w.z), f(w.w);
        }
    };
    auto pair = [&](uint32_t x) { atomicAdd(&sh[x & 0x7FFFu], x & 0x8000u ? 0x10000u : 1u); };

    uint32_t b = first;  // what is left of the share
    auto look = [&](uint32_t v) { return v < last ? vin[v].x : 0u; };
    uint32_t seen = look(b + tid);  // of the next batch, one word per thread
    __syncthreads();
    for (int k = 0; b < last; ++k) {
        if ((k == 0 || warp < 8) && b + (tid | 31) < last) {  // every lane of the warp has a word
            const int cost = pairs_over_bytes(seen & 0xFFu);
            if ((tid & 31) == 0) atomicAdd(&s_cost, cost);
        }
        clear();
        if (s_cost >= 0) break;
        const uint32_t e = min(last, b + PAIR_BATCH * PAIR_THREADS);
        seen = look(e + tid);
        words(b, e, [&](uint32_t w) { pair(w & 0xFFFFu), pair(w >> 16); });
        if (tid == 0) s_sum = 0;
        __syncthreads();
        // by first value: a value and a quarter of the rows per thread
        uint32_t sum = 0;
        for (int r = 0; r < 32; ++r) {
            const uint32_t w = sh[((tid >> 8) * 32 + r) * 256 + (tid & 255)];
            sum += (w & 0xFFFFu) + (w >> 16);
        }
        const uint32_t warp_sum = __reduce_add_sync(dev::FULL_MASK, sum);
        if ((tid & 31) == 0) atomicAdd(&s_sum, warp_sum);
        __syncthreads();
        if (s_sum != (e - b) * 8) break;  // a counter has wrapped: this batch again
        if (sum != 0) atomicAdd(&s_value[tid & 255], sum);
        // by second value: eight threads per row, 32 words each, every lane of
        // a warp in a bank of its own
        uint32_t low = 0, high = 0;
        const int row = tid >> 3, seg = tid & 7;
        for (int i = 0; i < 32; ++i) {
            const uint32_t w = sh[row * 256 + seg * 32 + ((i + tid) & 31)];
            low += w & 0xFFFFu;
            high += w >> 16;
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            low += __shfl_down_sync(dev::FULL_MASK, low, o, 8);
            high += __shfl_down_sync(dev::FULL_MASK, high, o, 8);
        }
        if (seg == 0) {
            if (low != 0) atomicAdd(&s_value[row], low);
            if (high != 0) atomicAdd(&s_value[row + 128], high);
        }
        b = e;
    }
    if (b < last) {  // the rest by bytes
        clear();
        uint32_t* my = sh + warp * 256;
        words(b, last, [&](uint32_t w) {
            atomicAdd(&my[w & 0xFF], 1u);
            atomicAdd(&my[w >> 8 & 0xFF], 1u);
            atomicAdd(&my[w >> 16 & 0xFF], 1u);
            atomicAdd(&my[w >> 24], 1u);
        });
        __syncthreads();
        if (tid < 256) {
            uint32_t s = 0;
            for (int w = 0; w < PAIR_WARPS; ++w) s += sh[w * 256 + tid];
            s_value[tid] += s;
        }
    }
    __syncthreads();
    if (blockIdx.x == 0 && tid < (int)(n - 16 * nv))
        atomicAdd(&s_value[reinterpret_cast<const uint8_t*>(in)[16 * (std::size_t)nv + tid]], 1u);
    __syncthreads();
    if (tid < 256 && s_value[tid] != 0) {
        const float x = (float)(T)(uint8_t)tid, scale = (float)bins / (upper - lower);
        if (x >= lower && x < upper) {
            uint32_t bin = (uint32_t)((x - lower) * scale);
            if (bin >= bins) bin = bins - 1;
            atomicAdd(&hist[bin], s_value[tid]);
        }
    }
}

// True when, for every value v of T, the device's float rule gives exactly
// bin v - offset (or excludes v exactly when v - offset is outside [0, bins)).
// Evaluated over all 2^8 / 2^16 values with the same float operations the
// kernel performs.
template <typename T, typename ACC> bool offset_rule(uint32_t bins, ACC lo, ACC hi, int& offset)
{
    if (!std::is_integral<T>::value || sizeof(T) > 2) return false;
    if (!(std::floor((double)lo) == (double)lo) || std::fabs((double)lo) > 65536.0) return false;
    offset = (int)lo;
    const ACC scale = (ACC)bins / (hi - lo);
    const int64_t first = std::numeric_limits<T>::min(), last = std::numeric_limits<T>::max();
    for (int64_t v = first; v <= last; ++v) {
        const ACC x = (ACC)(T)v;
        int64_t fb = -1;
        if (x >= lo && x < hi) {
            volatile ACC d = x - lo;  // one rounding per operation, as on the device
            volatile ACC p = d * scale;
            uint32_t b = (uint32_t)p;
            if (b >= bins) b = bins - 1;
            fb = b;
        }
        const int64_t ib = v - offset;
        const int64_t want = (ib >= 0 && ib < (int64_t)bins) ? ib : -1;
        if (fb != want) return false;
    }
    return true;
}

template <typename T>
void launch(device_context& ctx, const void* in, uint32_t n, uint32_t* hist, uint32_t bins,
            double lower, double upper)
{
    using ACC = typename std::conditional<std::is_same<T, double>::value, double, float>::type;
    const ACC lo = static_cast<ACC>(lower), hi = static_cast<ACC>(upper);
    constexpr int VEC = 16 / sizeof(T);
    if constexpr (sizeof(T) == 1) {
        if (n >= PAIR_MIN && (reinterpret_cast<uintptr_t>(in) & 15) == 0 && ctx.smem_optin >= PAIR_SMEM + 4096) {
            auto kernel = &k_histogram_pairs<T>;
            if (first_use_on_device((const void*)kernel))
                check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PAIR_SMEM),
                           "cudaFuncSetAttribute");
            kernel_timer kt(ctx, "histogram.pairs");
            kernel<<<ctx.sm_count, PAIR_THREADS, PAIR_SMEM, ctx.stream>>>(static_cast<const T*>(in), n, hist, bins, lo, hi);
            check_cuda(cudaGetLastError(), "histogram launch");
            return;
        }
    }
    const std::size_t warp_bytes = (std::size_t)bins * 4 * WARPS;
    const std::size_t cta_bytes = (std::size_t)bins * 4;
    int m;
    std::size_t smem;
    if (warp_bytes <= 64 * 1024) m = 0, smem = warp_bytes;
    else if (cta_bytes + 1024 <= ctx.smem_optin) m = 1, smem = cta_bytes;
    else m = 2, smem = 0;
    int offset = 0;
    const bool use_offset = offset_rule<T, ACC>(bins, lo, hi, offset);
    void (*kernel)(const T*, uint32_t, uint32_t*, uint32_t, ACC, ACC, int) =
        use_offset ? (m == 0 ? &k_histogram<T, ACC, 0, true> : m == 1 ? &k_histogram<T, ACC, 1, true>
                                                                       : &k_histogram<T, ACC, 2, true>)
                   : (m == 0 ? &k_histogram<T, ACC, 0, false> : m == 1 ? &k_histogram<T, ACC, 1, false>
                                                                        : &k_histogram<T, ACC, 2, false>);
    if (smem > 0)  // static shared memory adds to this against the 48 KiB default
        check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                   "cudaFuncSetAttribute");
    int per_sm = 0;
    check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, THREADS, smem),
               "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
    const std::size_t work = ((std::size_t)n + (std::size_t)THREADS * VEC - 1) / ((std::size_t)THREADS * VEC);
    const int grid = (int)std::max<std::size_t>(1, std::min<std::size_t>(work, (std::size_t)ctx.sm_count * std::max(per_sm, 1)));
    kernel_timer kt(ctx, "histogram.even");
    kernel<<<grid, THREADS, smem, ctx.stream>>>(static_cast<const T*>(in), n, hist, bins, lo, hi, offset);
    check_cuda(cudaGetLastError(), "histogram launch");
}

}  // namespace

void histogram_even(device_context& ctx, const void* in, std::size_t n, elem t, uint32_t* hist,
                    std::size_t bins, double lower, double upper)
{
    if (bins == 0) return;
    if (!(lower < upper)) throw std::invalid_argument("histogram_even: lower must be below upper");
    check_size(n);
    if (bins > 0xFFFFFFFFu) throw std::invalid_argument("histogram_even: too many bins");
    ctx.activate();
    check_cuda(cudaMemsetAsync(hist, 0, bins * sizeof(uint32_t), ctx.stream), "cudaMemsetAsync");
    if (n == 0) return;
    const uint32_t nn = (uint32_t)n, b = (uint32_t)bins;
    switch (t) {
    case elem::i8: launch<int8_t>(ctx, in, nn, hist, b, lower, upper); break;
    case elem::u8: launch<uint8_t>(ctx, in, nn, hist, b, lower, upper); break;
    case elem::i16: launch<int16_t>(ctx, in, nn, hist, b, lower, upper); break;
    case elem::u16: launch<uint16_t>(ctx, in, nn, hist, b, lower, upper); break;
    case elem::i32: launch<int32_t>(ctx, in, nn, hist, b, lower, upper); break;
    case elem::u32: launch<uint32_t>(ctx, in, nn, hist, b, lower, upper); break;
    case elem::i64: launch<int64_t>(ctx, in, nn, hist, b, lower, upper); break;
    case elem::u64: launch<uint64_t>(ctx, in, nn, hist, b, lower, upper); break;
    case elem::f32: launch<float>(ctx, in, nn, hist, b, lower, upper); break;
    case elem::f64: launch<double>(ctx, in, nn, hist, b, lower, upper); break;
    }
}

}  // namespace gbc
