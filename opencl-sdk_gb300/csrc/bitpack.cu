// Bitpack compression of 32-bit integers: frame-of-reference bit packing per
// chunk, optionally after a delta + zigzag transform.
//
// Reference path replaced: compress_bitpack / decompress_bitpack
// (lib/src/Compute/Compression.cpp:139-200) with kernels clc_bitpack_analyze,
// clc_bitpack_pack and clc_bitpack_unpack (Compression.cpp:39-124). The
// device format is kept word for word, since compressed data outlives the
// library that wrote it (Compression.cpp:19-24): per chunk three words {base,
// width, offset of its packed words relative to the packed area}, then the
// packed area; element j of a chunk occupies bits [j * width, (j + 1) *
// width) of the chunk's words, least significant bits first; width = 32 -
// clz(max - min) of the chunk's encoded values (0 when they are all equal);
// delta mode stores zigzag(x[i] - x[i-1]) with wrapping arithmetic and
// x[-1] = 0, and decoding ends with a wrapping inclusive prefix sum over the
// whole array.
//
// How it runs here:
//   * analyze: one warp per chunk, 128-bit loads, warp min/max; the chunks'
//     word counts are turned into offsets by the library's single-pass scan
//     (the reference's scan client at Compression.cpp:178), which also
//     yields the total size;
//   * pack: one warp per chunk or part of it, in rounds of 1,024 elements, which
//     fill whole words: the encoded elements go to shared memory, and each lane puts
//     together every 32nd word of the round from the elements in it (the
//     reference ORs every element into global memory with atomics);
//   * unpack, delta mode with a mean width of at most 26 bits: one pass. A
//     thread decodes 32 consecutive elements from the `width` whole words
//     that hold them (width a compile-time constant: one funnel shift per
//     element), the tile publishes the sum of its deltas, and its prefix is
//     the sum of what the tiles before it have published;
//   * unpack, otherwise: one thread per 4 elements (a 128-bit store),
//     reading the 1-5 packed words that hold them; delta mode then runs the
//     library's scan in place.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <functional>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/compute_c.h"
#include "device_common.cuh"
#include "pipe.cuh"
#include "runtime.hpp"
#include "sort_internal.hpp"

namespace gbc {
namespace bitpack {

using dev::FULL_MASK;

constexpr int THREADS = 256;
constexpr int WARPS = THREADS / 32;
constexpr int PACK_ROWS = 8;                     // rows of 128 elements per round
constexpr uint32_t ROUND = PACK_ROWS * 128;      // elements per warp and round

__device__ __forceinline__ uint32_t zigzag(uint32_t d) { return (d << 1) ^ (0u - (d >> 31)); }
__device__ __forceinline__ uint32_t unzigzag(uint32_t v) { return (v >> 1) ^ (0u - (v & 1u)); }

// Encoded values in[i .. i+3] (i a multiple of 4; `prev` = in[i - 1], or 0).
template <bool DELTA> __device__ __forceinline__ void encode4(uint4 w, uint32_t prev, uint32_t (&e)[4])
{
    if (DELTA) {
        e[0] = zigzag(w.x - prev);
        e[1] = zigzag(w.y - w.x);
        e[2] = zigzag(w.z - w.y);
        e[3] = zigzag(w.w - w.z);
    } else {
        e[0] = w.x, e[1] = w.y, e[2] = w.z, e[3] = w.w;
    }
}

template <bool DELTA> __device__ __forceinline__ uint32_t encode_at(const uint32_t* in, uint32_t i)
{
    if (!DELTA) return in[i];
    return zigzag(in[i] - (i > 0 ? in[i - 1] : 0u));
}

// One warp per chunk: base and width into hdr[2c], hdr[2c + 1], the chunk's
// packed word count into words[c].
template <bool DELTA>
__global__ void __launch_bounds__(THREADS) k_bp_analyze(const uint32_t* __restrict__ in, uint32_t n, uint32_t chunk,
                                                        uint32_t chunks, uint32_t* __restrict__ hdr,
                                                        uint32_t* __restrict__ words)
{
    const int lane = threadIdx.x & 31;
    const bool vec = (reinterpret_cast<uintptr_t>(in) & 15) == 0;
    for (uint32_t c = blockIdx.x * WARPS + (threadIdx.x >> 5); c < chunks; c += gridDim.x * WARPS) {
        const uint32_t start = c * chunk, count = min(chunk, n - start);
        uint32_t lo = 0xFFFFFFFFu, hi = 0;
        uint32_t j = 0;
        if (vec) {
            for (; j + 4 * 32 <= count; j += 4 * 32) {
                const uint32_t i = start + j + 4 * lane;
                const uint4 w = dev::ld_stream(reinterpret_cast<const uint4*>(in + i));
                uint32_t e[4];
                encode4<DELTA>(w, DELTA && i > 0 ? in[i - 1] : 0u, e);
#pragma unroll
                for (int q = 0; q < 4; ++q) lo = min(lo, e[q]), hi = max(hi, e[q]);
            }
        }
        for (uint32_t k = j + lane; k < count; k += 32) {
            const uint32_t e = encode_at<DELTA>(in, start + k);
            lo = min(lo, e), hi = max(hi, e);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = min(lo, __shfl_xor_sync(FULL_MASK, lo, o));
            hi = max(hi, __shfl_xor_sync(FULL_MASK, hi, o));
        }
        if (lane == 0) {
            const uint32_t range = hi - lo;
            const uint32_t width = range == 0 ? 0u : 32u - __clz(range);
            hdr[2 * c] = lo;
            hdr[2 * c + 1] = width;
            words[c] = (uint32_t)(((uint64_t)count * width + 31) / 32);
        }
    }
}

// One warp per `span` elements (a chunk or a part of it, whole rounds): their packed
// words, and with a chunk's first part its header triple. Bound by DRAM where the
// loads are (8 x 16 bytes per lane in flight); lane-private runs of 64 elements,
// read 256 bytes apart, took 389 us for 2 10^8 timestamps, this 223 (0.64 of the copy
// rate).
template <bool DELTA>
__global__ void __launch_bounds__(THREADS) k_bp_pack(const uint32_t* __restrict__ in, uint32_t n, uint32_t chunk,
                                                     uint32_t chunks, const uint32_t* __restrict__ hdr,
                                                     const uint32_t* __restrict__ offsets, uint32_t* __restrict__ out,
                                                     uint32_t span)
{
    __shared__ __align__(16) uint32_t stage[WARPS][ROUND];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t* my = stage[warp];
    const bool vec = (reinterpret_cast<uintptr_t>(in) & 15) == 0;
    const uint32_t per_chunk = chunk / span, parts = chunks * per_chunk;  // powers of two; the last chunk's may be empty
    for (uint32_t u = blockIdx.x * WARPS + warp; u < parts; u += gridDim.x * WARPS) {
        const uint32_t c = u / per_chunk, part = u % per_chunk * span;  // the part's first element within the chunk
        const uint32_t start = c * chunk, count = min(min(chunk, n - start), part + span);
        if (part >= count) continue;
        const uint32_t base = hdr[2 * c], width = hdr[2 * c + 1], off = offsets[c];
        if (lane == 0 && part == 0) {
            out[3 * c] = base;
            out[3 * c + 1] = width;
            out[3 * c + 2] = off;
        }
        if (width == 0) continue;
        uint32_t* packed = out + 3 * (size_t)chunks + off;
        // x / width for x <= 32 * ROUND = 2^15: the quotient's error term stays below 1 / width
        const uint32_t inverse = (uint32_t)(((1ull << 32) + width - 1) / width);
        uint32_t before = DELTA && start + part > 0 ? in[start + part - 1] : 0u;  // the element before the round
        for (uint32_t r0 = part; r0 < count; r0 += ROUND) {
            const uint32_t rcount = min(ROUND, count - r0), i0 = start + r0 + 4 * lane;
            uint4 w[PACK_ROWS];
#pragma unroll
            for (int r = 0; r < PACK_ROWS; ++r) {
                const uint32_t j = r * 128 + 4 * lane, i = i0 + r * 128;
                if (vec && j + 4 <= rcount) {
                    w[r] = dev::ld_stream(reinterpret_cast<const uint4*>(in + i));
                } else {  // past the end: never packed
                    w[r].x = j < rcount ? in[i] : 0u;
                    w[r].y = j + 1 < rcount ? in[i + 1] : 0u;
                    w[r].z = j + 2 < rcount ? in[i + 2] : 0u;
                    w[r].w = j + 3 < rcount ? in[i + 3] : 0u;
                }
            }
#pragma unroll
            for (int r = 0; r < PACK_ROWS; ++r) {
                uint32_t prev = 0;
                if (DELTA) {
                    prev = __shfl_up_sync(FULL_MASK, w[r].w, 1);
                    if (lane == 0) prev = before;
                    before = __shfl_sync(FULL_MASK, w[r].w, 31);
                }
                uint32_t e[4];
                encode4<DELTA>(w[r], prev, e);
                reinterpret_cast<uint4*>(my)[r * 32 + lane] = make_uint4(e[0] - base, e[1] - base, e[2] - base, e[3] - base);
            }
            __syncwarp();
            const uint32_t rwords = (rcount * width + 31) / 32;
            uint32_t* dst = packed + (size_t)(r0 / 32) * width;  // r0 * width / 32 (r0 is a multiple of ROUND)
            for (uint32_t m = lane; m < rwords; m += 32) {
                uint32_t j = __umulhi(32 * m, inverse);  // the element holding the word's first bit (width 1: 2^32 wraps)
                if (width == 1) j = 32 * m;
                const uint32_t skip = 32 * m - j * width;
                uint32_t word = my[j] >> skip;
                for (uint32_t have = width - skip; have < 32 && ++j < rcount; have += width) word |= my[j] << have;
                dst[m] = word;
            }
            __syncwarp();
        }
    }
}

// One thread per 4 elements. Chunks hold a multiple of 4 elements (at least
// 256), so a group never straddles two chunks.
template <bool DELTA>
__global__ void __launch_bounds__(THREADS) k_bp_unpack(const uint32_t* __restrict__ data, uint32_t n,
                                                       uint32_t chunk_shift, uint32_t chunks,
                                                       uint32_t* __restrict__ out)
{
    const uint32_t groups = (n + 3) / 4;
    const bool vec = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    for (uint32_t g = blockIdx.x * THREADS + threadIdx.x; g < groups; g += gridDim.x * THREADS) {
        const uint32_t i = 4 * g;
        const uint32_t c = i >> chunk_shift, j = i & ((1u << chunk_shift) - 1u);
        const uint32_t base = __ldg(data + 3 * c), width = __ldg(data + 3 * c + 1);
        uint32_t v[4] = {base, base, base, base};
        if (width != 0) {
            const uint32_t* p = data + 3 * (size_t)chunks + __ldg(data + 3 * c + 2);
            const uint64_t first = (uint64_t)j * width;
            const uint32_t w0 = (uint32_t)(first >> 5);
            const uint32_t mask = width == 32 ? 0xFFFFFFFFu : ((1u << width) - 1u);
            // the group's elements below n lie in bits [first, first + valid
            // x width): at most 5 words from w0; words past the last of them
            // may lie beyond the chunk's packed words and are not read
            const uint32_t valid = min(4u, n - i);
            const uint32_t last_word = (uint32_t)((first + (uint64_t)valid * width - 1) >> 5);
            uint32_t wv[5];
#pragma unroll
            for (int q = 0; q < 5; ++q) wv[q] = (w0 + q <= last_word) ? __ldg(p + w0 + q) : 0u;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const uint64_t bit = first + (uint64_t)t * width;
                const uint32_t q = (uint32_t)(bit >> 5) - w0, sh = (uint32_t)(bit & 31);
                const uint64_t both = (uint64_t)wv[q] | ((uint64_t)(q + 1 < 5 ? wv[q + 1] : 0u) << 32);
                v[t] = (uint32_t)(both >> sh) & mask;
                v[t] += base;
            }
        }
        if (DELTA) {
#pragma unroll
            for (int t = 0; t < 4; ++t) v[t] = unzigzag(v[t]);
        }
        if (vec && i + 4 <= n) {
            *reinterpret_cast<uint4*>(out + i) = make_uint4(v[0], v[1], v[2], v[3]);
        } else {
            for (int t = 0; t < 4 && i + t < n; ++t) out[i + t] = v[t];
        }
    }
}

// ---- unpack by lane-private whole words ---------------------------------------
// A thread decodes 32 consecutive elements of one chunk, which occupy exactly
// `width` whole words of the packed area (element j sits at bit j * width and
// 32 * width bits are width words), so with the width as a compile-time
// constant every shift and word index is a constant (one funnel shift, a mask
// and an add per element). A CTA's 8,192 elements form one tile. In delta mode
// the tile's deltas are scanned in place (thread, warp, CTA), its sum is
// published at once, and its prefix is the sum of the published ones: every
// thread keeps its share of those before the CTA's last tile and adds its
// share of those since (about one per running CTA, read in one round trip).
// Nothing waits for another tile's prefix: the decoupled look-back that this
// replaces took 542 us for 2 10^8 timestamps, a first pass for the sums and a
// second one 350, this 319. The decoded tile is staged in shared memory at
// an odd stride and written out coalesced.
constexpr int UT = 256;             // threads per CTA
constexpr int UE = 32;              // elements per thread
constexpr int UTILE = UT * UE;      // elements per tile

// Elements of the lane's 32 (all in one chunk) from its W packed words at p;
// `words_left` bounds the reads at the end of the buffer.
template <int W>
__device__ __forceinline__ void decode32(const uint32_t* __restrict__ p, uint64_t words_left, uint32_t base,
                                         uint32_t (&v)[UE])
{
    if constexpr (W == 0) {
#pragma unroll
        for (int e = 0; e < UE; ++e) v[e] = base;
    } else {
        uint32_t w[W];
        if (words_left >= (uint64_t)W) {
#pragma unroll
            for (int k = 0; k < W; ++k) w[k] = __ldg(p + k);
        } else {
#pragma unroll
            for (int k = 0; k < W; ++k) w[k] = (uint64_t)k < words_left ? __ldg(p + k) : 0u;
        }
#pragma unroll
        for (int e = 0; e < UE; ++e) {
            constexpr uint32_t mask = W == 32 ? 0xFFFFFFFFu : ((1u << (W & 31)) - 1u);
            const int bit = e * W, q = bit >> 5, sh = bit & 31;
            uint32_t x;
            if (W == 32) x = w[e];
            else if (sh + W <= 32) x = (w[q] >> sh) & mask;
            else x = __funnelshift_r(w[q], w[q + 1 < W ? q + 1 : q], sh) & mask;
            v[e] = x + base;
        }
    }
}

template <int W0>
__device__ __forceinline__ void decode_dispatch(uint32_t width, const uint32_t* p, uint64_t words_left, uint32_t base,
                                                uint32_t (&v)[UE])
{
    if constexpr (W0 <= 32) {
        if (width == (uint32_t)W0) decode32<W0>(p, words_left, base, v);
        else decode_dispatch<W0 + 1>(width, p, words_left, base, v);
    }
}

template <bool DELTA>
__global__ void __launch_bounds__(UT)
    k_bp_unpack_tiles(const uint32_t* __restrict__ data, uint64_t words, uint32_t n, uint32_t chunk_shift,
                      uint32_t chunks, uint32_t* __restrict__ out, pipe::Tiles tiles)
{
    using Sum = pipe::Aggregate<uint32_t>;
    __shared__ uint32_t s_out[UT * (UE + 1)];
    __shared__ uint32_t s_warp[UT / 32], s_part[UT / 32];
    __shared__ uint32_t s_tile;
    uint32_t share = 0, done = 0;  // of the sums of the tiles before `done`
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t* packed = data + 3 * (size_t)chunks;
    for (;;) {
        if (tid == 0) s_tile = atomicAdd(tiles.counter, 1u);
        __syncthreads();
        const uint32_t t = s_tile;
        if (t >= tiles.num_tiles) break;
        const uint32_t i0 = t * UTILE + tid * UE;  // the thread's first element
        uint32_t v[UE];
        if (i0 < n) {
            const uint32_t c = i0 >> chunk_shift, j0 = i0 & ((1u << chunk_shift) - 1u);
            const uint32_t base = __ldg(data + 3 * c), width = __ldg(data + 3 * c + 1);
            const uint64_t first = (uint64_t)__ldg(data + 3 * c + 2) + (uint64_t)(j0 / UE) * width;
            const uint64_t avail = 3 * (uint64_t)chunks + first < words ? words - 3 * (uint64_t)chunks - first : 0;
            if (width > 32) {  // corrupt header: the caller validated the blob, nothing is decoded
#pragma unroll
                for (int e = 0; e < UE; ++e) v[e] = 0;
            } else {
                decode_dispatch<0>(width, packed + first, avail, base, v);
            }
#pragma unroll
            for (int e = 0; e < UE; ++e)
                if (i0 + e >= n) v[e] = DELTA ? zigzag(0u) : 0u;  // past the end: a zero delta
        } else {
#pragma unroll
            for (int e = 0; e < UE; ++e) v[e] = 0;
        }
        if (DELTA) {
            // undo the zigzag, then the thread's inclusive sums (wrapping)
#pragma unroll
            for (int e = 0; e < UE; ++e) v[e] = unzigzag(v[e]);
#pragma unroll
            for (int e = 1; e < UE; ++e) v[e] += v[e - 1];
        }
        bool abort = false;
        uint32_t add = 0;  // to the thread's sums
        if (DELTA) {
            uint32_t inc = v[UE - 1];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL_MASK, inc, o);
                if (lane >= o) inc += y;
            }
            if (lane == 31) s_warp[warp] = inc;
            __syncthreads();
            uint32_t sum = 0;
            add = inc - v[UE - 1];
#pragma unroll
            for (int w = 0; w < UT / 32; ++w) {
                const uint32_t x = s_warp[w];
                if (w < warp) add += x;
                sum += x;
            }
            if (tid == 0) Sum::publish(tiles.ring, tiles.seq0 + t, sum);
            for (uint32_t k = done + tid; k < t; k += UT) {
                uint32_t x;
                if (!Sum::read(tiles.ring, tiles.seq0 + k, x)) {
                    const unsigned long long start = dev::globaltimer();
                    for (uint32_t spin = 1; !Sum::read(tiles.ring, tiles.seq0 + k, x); ++spin) {
                        if ((spin & 63) == 0 && dev::globaltimer() - start > dev::SPIN_LIMIT_NS) {
                            dev::raise_error(tiles.err, dev::ERR_LOOKBACK_TIMEOUT);
                            abort = true;
                            break;
                        }
                        if (spin > 4) __nanosleep(64);
                    }
                    if (abort) break;
                }
                share += x;
            }
            done = t;
            const uint32_t part = __reduce_add_sync(FULL_MASK, share);
            if (lane == 0) s_part[warp] = part;
        }
        // after a timed-out wait the prefix is unknown: nothing is written any more
        if (__syncthreads_or(abort)) break;
        if (DELTA) {
#pragma unroll
            for (int w = 0; w < UT / 32; ++w) add += s_part[w];
#pragma unroll
            for (int e = 0; e < UE; ++e) v[e] += add;
        }
        {
            // stage at stride UE + 1 (conflict-free both ways) and write coalesced
#pragma unroll
            for (int e = 0; e < UE; ++e) s_out[tid * (UE + 1) + e] = v[e];
            __syncthreads();
            const uint32_t tb = t * UTILE;
            if (tb + UTILE <= n) {
#pragma unroll 8
                for (int k = 0; k < UE; ++k) {
                    const uint32_t idx = k * UT + tid;
                    out[tb + idx] = s_out[(idx / UE) * (UE + 1) + idx % UE];
                }
            } else {
                for (int k = 0; k < UE; ++k) {
                    const uint32_t idx = k * UT + tid;
                    if (tb + idx < n) out[tb + idx] = s_out[(idx / UE) * (UE + 1) + idx % UE];
                }
            }
            __syncthreads();
        }
    }
}

void check_chunk(std::size_t chunk)
{
    if (chunk < 256 || chunk > 65536 || (chunk & (chunk - 1)) != 0)
        throw std::invalid_argument("bitpack: chunk_size must be a power of two in [256, 65536]");
}

int grid_for(device_context& ctx, std::size_t work_warps, int warps_per_cta)
{
    const std::size_t ctas = (work_warps + warps_per_cta - 1) / warps_per_cta;
    return (int)std::max<std::size_t>(1, std::min<std::size_t>(ctas, (std::size_t)ctx.sm_count * 64 / warps_per_cta));
}

}  // namespace bitpack

std::size_t bitpack_words_bound(std::size_t n, std::size_t chunk)
{
    bitpack::check_chunk(chunk);
    return n == 0 ? 0 : 3 * ((n + chunk - 1) / chunk) + n;
}

std::size_t bitpack_compress(device_context& ctx, const uint32_t* in, std::size_t n, std::size_t chunk, bool delta,
                             const std::function<uint32_t*(std::size_t)>& make_output)
{
    using namespace bitpack;
    check_chunk(chunk);
    if (n == 0) return 0;
    check_size(n);
    if (in == nullptr) throw std::invalid_argument("bitpack: null input");
    ctx.activate();
    const uint32_t chunks = (uint32_t)((n + chunk - 1) / chunk);
    temp_buffer hdr(ctx.resource, (std::size_t)chunks * 2 * 4);
    temp_buffer words(ctx.resource, (std::size_t)chunks * 4);
    temp_buffer offs(ctx.resource, (std::size_t)chunks * 4);
    temp_buffer total(ctx.resource, 8);
    const int grid = grid_for(ctx, chunks, WARPS);
    {
        kernel_timer kt(ctx, "bitpack.analyze");
        if (delta)
            k_bp_analyze<true><<<grid, THREADS, 0, ctx.stream>>>(in, (uint32_t)n, (uint32_t)chunk, chunks,
                                                                 hdr.as<uint32_t>(), words.as<uint32_t>());
        else
            k_bp_analyze<false><<<grid, THREADS, 0, ctx.stream>>>(in, (uint32_t)n, (uint32_t)chunk, chunks,
                                                                  hdr.as<uint32_t>(), words.as<uint32_t>());
        check_cuda(cudaGetLastError(), "bitpack analyze launch");
    }
    const uint32_t zero = 0;
    scan(ctx, words.get(), offs.get(), chunks, elem::u32, op_kind::plus, &zero, true, total.get());
    uint64_t packed = 0;
    check_cuda(cudaMemcpyAsync(&packed, total.get(), 8, cudaMemcpyDeviceToHost, ctx.stream), "cudaMemcpyAsync");
    check_cuda(cudaStreamSynchronize(ctx.stream), "cudaStreamSynchronize");
    const std::size_t out_words = 3 * (std::size_t)chunks + packed;
    uint32_t* out = make_output(out_words);
    // Parts of a chunk where the chunks are too few to keep the SMs' warps busy several
    // times over (10^7 elements in chunks of 65,536: 474 -> 300 us for the call, 5,000 in
    // chunks of 2,048 45 -> 38); a whole chunk else, whose header is read once (10^8
    // elements in chunks of 2,048: 283 us, in rounds 294).
    std::size_t span = chunk;
    while (span > ROUND && n / span < (std::size_t(1) << 15)) span /= 2;
    {
        kernel_timer kt(ctx, "bitpack.pack");
        const int grid = grid_for(ctx, (n + span - 1) / span, WARPS);
        if (delta)
            k_bp_pack<true><<<grid, THREADS, 0, ctx.stream>>>(in, (uint32_t)n, (uint32_t)chunk, chunks,
                                                              hdr.as<uint32_t>(), offs.as<uint32_t>(), out, (uint32_t)span);
        else
            k_bp_pack<false><<<grid, THREADS, 0, ctx.stream>>>(in, (uint32_t)n, (uint32_t)chunk, chunks,
                                                               hdr.as<uint32_t>(), offs.as<uint32_t>(), out, (uint32_t)span);
        check_cuda(cudaGetLastError(), "bitpack pack launch");
    }
    return out_words;
}

void bitpack_decompress(device_context& ctx, const uint32_t* data, std::size_t words, std::size_t n,
                        std::size_t chunk, bool delta, uint32_t* out)
{
    using namespace bitpack;
    check_chunk(chunk);
    if (n == 0) return;
    check_size(n);
    if (data == nullptr || out == nullptr) throw std::invalid_argument("bitpack: null argument");
    const uint32_t chunks = (uint32_t)((n + chunk - 1) / chunk);
    if (words < 3 * (std::size_t)chunks) throw std::invalid_argument("bitpack: data shorter than its chunk headers");
    ctx.activate();
    uint32_t shift = 0;
    while ((std::size_t(1) << shift) < chunk) ++shift;
    // Delta mode with a mean packed width of at most 26 bits (known from the
    // compressed size): whole words per lane in one pass (2 10^8 elements, one
    // pass / two: 7 bits 0.32 / 0.56 ms, 18 bits 0.35 / 0.56, 25 bits 0.43 /
    // 0.56). Wider data, and plain mode, decode faster as 4-element groups (the
    // lane-private form issues W scattered loads per lane: 2^28 words, plain,
    // 1.1 ms against 0.42 at 32 bits).
    const uint64_t packed_words = words - 3 * (uint64_t)chunks;
    const bool one_pass = delta && packed_words * 32 <= (uint64_t)n * 26;
    launch_shape sh;
    const int forced = ctx.tuning.lookup("bitpack:unpack", sh) ? sh.variant : -1;  // 0: one pass, 1: two passes
    if (forced == 0 || (forced != 1 && one_pass)) {
        const uint32_t num_tiles = (uint32_t)((n + UTILE - 1) / UTILE);
        pipe::Tiles tiles;
        tiles.num_tiles = num_tiles;
        tiles.counter = reinterpret_cast<uint32_t*>(ctx.d_small + 3072);
        check_cuda(cudaMemsetAsync(tiles.counter, 0, 4, ctx.stream), "cudaMemsetAsync");
        tiles.ring = ctx.lookback_ring;
        tiles.seq0 = ctx.reserve_seq(num_tiles);
        tiles.err = ctx.d_error;
        auto kern = delta ? &k_bp_unpack_tiles<true> : &k_bp_unpack_tiles<false>;
        // asked once (one architecture): the query takes as long as a launch
        static std::atomic<int> known[2];
        int per_sm = known[delta].load(std::memory_order_relaxed);
        if (per_sm == 0) {
            check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, UT, 0), "cudaOccupancy");
            known[delta].store(per_sm = std::max(per_sm, 1), std::memory_order_relaxed);
        }
        const int grid = (int)std::min<std::size_t>(num_tiles, (std::size_t)ctx.sm_count * per_sm);
        kernel_timer kt(ctx, "bitpack.unpack");
        kern<<<grid, UT, 0, ctx.stream>>>(data, (uint64_t)words, (uint32_t)n, shift, chunks, out, tiles);
        check_cuda(cudaGetLastError(), "bitpack unpack launch");
        return;
    }
    const std::size_t groups = (n + 3) / 4;
    const int grid = (int)std::max<std::size_t>(
        1, std::min<std::size_t>((groups + THREADS - 1) / THREADS, (std::size_t)ctx.sm_count * 16));
    {
        kernel_timer kt(ctx, "bitpack.unpack");
        if (delta)
            k_bp_unpack<true><<<grid, THREADS, 0, ctx.stream>>>(data, (uint32_t)n, shift, chunks, out);
        else
            k_bp_unpack<false><<<grid, THREADS, 0, ctx.stream>>>(data, (uint32_t)n, shift, chunks, out);
        check_cuda(cudaGetLastError(), "bitpack unpack launch");
    }
    if (delta) {
        const uint32_t zero = 0;
        scan(ctx, out, out, n, elem::u32, op_kind::plus, &zero, false, nullptr);
    }
}

}  // namespace gbc
