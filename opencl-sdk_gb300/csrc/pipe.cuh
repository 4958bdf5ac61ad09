// Tiles of a large input as a pipeline inside each CTA, for operations whose
// output place or value depends on everything before it (scan, compaction).
//
// One CTA per SM runs four kinds of warps. The copying warp takes tiles from a
// counter and copies them to shared memory STAGES ahead (bulk copies). The
// folding warps reduce each tile as soon as it has landed and publish its
// aggregate. The prefix warp keeps the prefix of the CTA's last tile and adds
// the aggregates published since (about one per CTA). The writing warps, each
// with its own block of the tile and at its own pace, finish the tile.
//
// A tile's aggregate needs nothing but its own data, so nothing waits for
// another tile's prefix; and tiles are taken in order, so a CTA only waits for
// tiles that running CTAs hold: the kernel needs no co-residency. Waits are
// bounded: a prefix warp that waits too long for an aggregate records
// ERR_LOOKBACK_TIMEOUT, and its CTA writes nothing from then on.
//
// The reference's counterpart is the multi-launch scan of tile totals
// (lib/src/Compute/Algorithm.cpp:280-318).
#pragma once

#include <cstring>

#include "device_common.cuh"
#include "sort_internal.hpp"

namespace gbc {
namespace pipe {

using dev::FULL_MASK;

// Warps. Measured as writers / folders / stages (scan of 2^30 int32 with its
// total, scan of 2^28 int64, copy_if of 10^8 floats): 16/8/6 1.26 ms, 0.89 ms,
// 141 us; 20/10/5 1.21, 0.75, 117; 24/6/4 1.26, 0.69, 119; 21/7/5 1.22, 0.75, 117;
// 20/5/5 1.30, 0.75, 120; 24/4/4 1.47, 0.70, 127; 16/4/6 1.39, 0.87, 122. What
// bounds a tile is the chain of one writing warp, so more of them pay.
constexpr int WRITERS = 20, FOLDERS = 10;
constexpr int THREADS = (WRITERS + FOLDERS + 2) * 32;  // and the prefix warp and the copying warp
constexpr int PREFIX_WARP = WRITERS + FOLDERS, COPY_WARP = PREFIX_WARP + 1;
constexpr int ROWS = 4;  // rows of 512 bytes per writing warp and tile
constexpr int STAGES = 5;
constexpr int PER = 8;  // aggregates read per lane and round trip: 256, more than there are CTAs
constexpr int BLOCKS = WRITERS / FOLDERS;  // a tile's blocks (one per writing warp) per folding warp
constexpr uint32_t BLOCK_BYTES = ROWS * 512, TILE_BYTES = WRITERS * BLOCK_BYTES;
constexpr std::size_t SMEM = (std::size_t)STAGES * TILE_BYTES;
constexpr uint32_t END = 0xFFFFFFFFu;
// Waits inside a CTA outlast its wait for other CTAs, so that the latter gives
// up first and is what is reported.
constexpr unsigned long long INNER_LIMIT_NS = 4 * dev::SPIN_LIMIT_NS;

constexpr uint64_t FLAG_AGG = 1;
constexpr uint64_t TAG_MASK = (1ull << 30) - 1;

// The published aggregate of one tile: a word of (flag | tag | 32 bits of the
// value) per four bytes of it; every word carries its tag, so they are read in
// one round trip with no order between them.
template <typename T> struct Aggregate {
    static constexpr int WORDS = sizeof(T) / 4;
    static constexpr uint64_t SLOTS = onesweep::RING_BYTES / 8 / (WORDS <= 2 ? WORDS : 4);
    __device__ static uint64_t* at(uint64_t* ring, uint64_t seq)
    {
        return ring + (seq & (SLOTS - 1)) * (WORDS <= 2 ? WORDS : 4);
    }
    __device__ static uint64_t head(uint64_t seq) { return (FLAG_AGG << 62) | ((seq & TAG_MASK) << 32); }
    __device__ static void publish(uint64_t* ring, uint64_t seq, const T& v)
    {
        uint32_t bits[WORDS];
        memcpy(bits, &v, sizeof(T));
#pragma unroll
        for (int i = 0; i < WORDS; ++i) dev::st_relaxed(at(ring, seq) + i, head(seq) | bits[i]);
    }
    __device__ static bool read(uint64_t* ring, uint64_t seq, T& v)
    {
        uint32_t bits[WORDS];
        bool ok = true;
#pragma unroll
        for (int i = 0; i < WORDS; ++i) {
            const uint64_t w = dev::ld_relaxed(at(ring, seq) + i);
            ok &= (w >> 32) == (head(seq) >> 32);
            bits[i] = (uint32_t)w;
        }
        memcpy(&v, bits, sizeof(T));
        return ok;
    }
};

template <typename T> __device__ __forceinline__ T shfl_down(const T& x, int o)
{
    uint32_t w[sizeof(T) / 4];
    memcpy(w, &x, sizeof(T));
#pragma unroll
    for (auto& v : w) v = __shfl_down_sync(FULL_MASK, v, o);
    T y;
    memcpy(&y, w, sizeof(T));
    return y;
}
template <typename T> __device__ __forceinline__ T shfl_up(const T& x, int o)
{
    uint32_t w[sizeof(T) / 4];
    memcpy(w, &x, sizeof(T));
#pragma unroll
    for (auto& v : w) v = __shfl_up_sync(FULL_MASK, v, o);
    T y;
    memcpy(&y, w, sizeof(T));
    return y;
}
template <typename T> __device__ __forceinline__ T shfl(const T& x, int lane)
{
    uint32_t w[sizeof(T) / 4];
    memcpy(w, &x, sizeof(T));
#pragma unroll
    for (auto& v : w) v = __shfl_sync(FULL_MASK, v, lane);
    T y;
    memcpy(&y, w, sizeof(T));
    return y;
}

// op over lanes 0 .. count - 1 in order, to every lane (count >= 1).
template <typename T, typename Op> __device__ __forceinline__ T fold_lanes(T x, int count, Op op)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T y = shfl_down(x, o);
        if ((lane & (2 * o - 1)) == 0 && lane + o < count) x = op(x, y);
    }
    return shfl(x, 0);
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(dev::smem_addr(bar)) : "memory");
}
// Barrier of the folding warps.
__device__ __forceinline__ void fold_sync() { asm volatile("bar.sync 1, %0;" ::"n"(FOLDERS * 32) : "memory"); }

// What a launch's CTAs share.
struct Tiles {
    uint32_t num_tiles;
    uint32_t* counter;
    uint64_t* ring;
    uint64_t seq0;  // sequence number of tile 0's aggregate
    int* err;
};

// A CTA's state in shared memory. Iteration k of every role works on stage
// k % STAGES; T: the aggregate's type.
template <typename T> struct Shared {
    uint64_t full[STAGES];   // the tile's index is known and its copy has landed
    uint64_t empty[STAGES];  // every writing warp is done with the stage
    uint64_t ready[STAGES];  // the prefix and what the folding warps leave are there
    uint32_t tile[STAGES];   // or END
    T prefix[STAGES];        // of the tiles before it
    T total[2][WRITERS];     // the folding warps' block totals
    volatile int abort;

    // Every thread of the CTA calls it.
    __device__ void init()
    {
        if (threadIdx.x == 0) {
            for (int s = 0; s < STAGES; ++s) {
                dev::mbar_init(&full[s], 1);
                dev::mbar_init(&empty[s], WRITERS);
                dev::mbar_init(&ready[s], 2);  // prefix warp, first folding warp
                tile[s] = END;
            }
            abort = 0;
            dev::fence_mbar_init();
        }
        __syncthreads();
    }
    __device__ void wait(uint64_t* bar, uint32_t k, int* err)
    {
        const uint32_t parity = (k / STAGES) & 1;
        if (dev::mbar_try_wait(bar, parity)) return;
        const unsigned long long start = dev::globaltimer();
        for (uint32_t spin = 1; !dev::mbar_try_wait(bar, parity); ++spin)
            if ((spin & 63) == 0 && dev::globaltimer() - start > INNER_LIMIT_NS) {
                dev::raise_error(err, dev::ERR_LOOKBACK_TIMEOUT);
                abort = 1;
                return;
            }
    }
    // Waits for iteration k's tile: its index, or END.
    __device__ uint32_t next(uint32_t k, int* err)
    {
        wait(&full[k % STAGES], k, err);
        return *(volatile uint32_t*)&tile[k % STAGES];
    }
};

// Iterations of every role, at most.
__device__ __forceinline__ uint32_t limit(const Tiles& a) { return a.num_tiles + STAGES; }

// The copying warp: whole tiles of TILE_BYTES from `in` (16-byte aligned); a
// last partial tile is announced without a copy. SIDE: bytes per tile of a
// second array, copied along into side_stages.
template <uint32_t SIDE = 0, typename T>
__device__ void copy_role(const Tiles& a, Shared<T>& sh, unsigned char* stages, const void* in, uint64_t bytes,
                          unsigned char* side_stages = nullptr, const void* side = nullptr)
{
    static_assert(SIDE % 16 == 0, "bulk copies");
    if ((threadIdx.x & 31) != 0) return;
    for (uint32_t k = 0; k < limit(a); ++k) {
        const int s = k % STAGES;
        if (k >= STAGES) sh.wait(&sh.empty[s], k - STAGES, a.err);
        const uint32_t t = atomicAdd(a.counter, 1u);
        if (t >= a.num_tiles) {
            sh.tile[s] = END;
            mbar_arrive(&sh.full[s]);
            return;
        }
        sh.tile[s] = t;
        if ((uint64_t)(t + 1) * TILE_BYTES <= bytes) {
            dev::mbar_arrive_expect_tx(&sh.full[s], TILE_BYTES + SIDE);
            dev::bulk_g2s(stages + (std::size_t)s * TILE_BYTES, static_cast<const unsigned char*>(in) + (std::size_t)t * TILE_BYTES,
                          TILE_BYTES, &sh.full[s]);
            if (SIDE > 0)
                dev::bulk_g2s(side_stages + (std::size_t)s * SIDE, static_cast<const unsigned char*>(side) + (std::size_t)t * SIDE,
                              SIDE, &sh.full[s]);
        } else {
            mbar_arrive(&sh.full[s]);
        }
    }
}

// The prefix warp: prefix[s] = first, combined with the aggregates of all tiles
// before the stage's. ANY_ORDER: no order changes the operator's result, and the
// lanes read neighbouring words, a quarter of the sectors (scan of 2^30 int32
// 1.31 -> 1.26 ms); else each lane reads PER consecutive ones, so that they
// combine in order. (Two prefix warps taking the CTA's tiles in turn read twice
// as many words and were slower: 2^30 int32 1.31 -> 1.55 ms.)
template <bool ANY_ORDER, typename T, typename Op> __device__ void prefix_role(const Tiles& a, Shared<T>& sh, T first, Op op)
{
    const int lane = threadIdx.x & 31;
    T run = first;  // over the tiles before `done`
    uint32_t done = 0;
    for (uint32_t k = 0; k < limit(a); ++k) {
        const uint32_t t = sh.next(k, a.err);
        if (t == END) return;
        // windows of 32 * PER tiles, all read before any is waited for
        for (uint32_t w = done; w < t; w += 32 * PER) {
            const uint32_t count = min(32u * PER, t - w);
            auto index = [&](int q) { return (uint32_t)(ANY_ORDER ? q * 32 + lane : lane * PER + q); };
            T val[PER];
            uint32_t missing = 0;
#pragma unroll
            for (int q = 0; q < PER; ++q)
                if (index(q) < count && !Aggregate<T>::read(a.ring, a.seq0 + w + index(q), val[q]))
                    missing |= 1u << q;
            const unsigned long long start = missing ? dev::globaltimer() : 0;
            for (uint32_t spin = 1; missing != 0 && !sh.abort; ++spin) {
#pragma unroll
                for (int q = 0; q < PER; ++q)
                    if ((missing >> q & 1u) && Aggregate<T>::read(a.ring, a.seq0 + w + index(q), val[q]))
                        missing &= ~(1u << q);
                if ((spin & 63) == 0 && dev::globaltimer() - start > dev::SPIN_LIMIT_NS) {
                    dev::raise_error(a.err, dev::ERR_LOOKBACK_TIMEOUT);
                    sh.abort = 1;
                }
            }
            __syncwarp();
            T mine = val[0];
#pragma unroll
            for (int q = 1; q < PER; ++q)
                if (index(q) < count) mine = op(mine, val[q]);
            run = op(run, fold_lanes(mine, (int)(ANY_ORDER ? min(count, 32u) : (count + PER - 1) / PER), op));
        }
        done = t;
        if (lane == 0) {
            sh.prefix[k % STAGES] = run;
            mbar_arrive(&sh.ready[k % STAGES]);  // releases the store
        }
        __syncwarp();
    }
}

// The folding warps, after each has put its blocks' totals into
// sh.total[k & 1]: publishes tile t's aggregate; block b > 0 finds the
// combination of the blocks before it in before[b].
template <typename T, typename Op>
__device__ __forceinline__ void publish_tile(const Tiles& a, Shared<T>& sh, uint32_t k, uint32_t t, T (&before)[WRITERS], Op op)
{
    const int lane = threadIdx.x & 31;
    fold_sync();
    if ((threadIdx.x >> 5) != WRITERS) return;  // the first folding warp
    T x = sh.total[k & 1][lane % WRITERS];
#pragma unroll
    for (int o = 1; o < WRITERS; o <<= 1) {
        const T y = shfl_up(x, o);
        if (lane >= o) x = op(y, x);
    }
    if (lane == WRITERS - 1) Aggregate<T>::publish(a.ring, a.seq0 + t, x);
    if (lane < WRITERS - 1) before[lane + 1] = x;
    __syncwarp();
    if (lane == 0) mbar_arrive(&sh.ready[k % STAGES]);
}

}  // namespace pipe
}  // namespace gbc
