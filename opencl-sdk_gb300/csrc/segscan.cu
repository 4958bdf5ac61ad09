// Segmented scan: one single-pass decoupled look-back scan whose running value
// restarts at every segment start. No reference counterpart (the reference
// scans one array per call, lib/src/Compute/Algorithm.cpp:280-318); within a
// segment the semantics are the reference scan's: canonical operator combined
// in sequence order, exclusive output begins with the identity.
//
// Each element carries a head flag (it starts a segment); pairs combine as
//   (fa, va) (+) (fb, vb) = (fa | fb, fb ? vb : op(va, vb)),
// which is associative, so the tile machinery of the plain scan applies. A
// predecessor tile that contains a head already holds a complete prefix, so
// the look-back also stops there.
//
// Head flags come from the offsets: one binary search per tile for the first
// segment starting in the tile, then the tile's starts are set in a shared
// bitmask.
#include <cstring>
#include <memory>

#include "device_common.cuh"
#include "ops.cuh"
#include "pipe.cuh"
#include "runtime.hpp"
#include "segmented.hpp"
#include "sort_internal.hpp"

namespace gbc {
namespace {

using dev::FULL_MASK;
constexpr int THREADS = 256;
constexpr uint64_t FLAG_AGG = 1, FLAG_PRE = 2;
constexpr uint64_t TAG_MASK = (1ull << 29) - 1;
constexpr uint64_t HEAD_BIT = 1ull << 61;

template <typename T> __device__ __forceinline__ uint64_t to_bits(T v)
{
    uint64_t b = 0;
    memcpy(&b, &v, sizeof(T));
    return b;
}
template <typename T> __device__ __forceinline__ T from_bits(uint64_t b)
{
    T v;
    memcpy(&v, &b, sizeof(T));
    return v;
}

template <typename T, bool WIDE = (sizeof(T) == 8)> struct SStatus;
template <typename T> struct SStatus<T, false> {
    static constexpr uint64_t SLOTS = onesweep::RING_BYTES / 8;
    __device__ static void publish(uint64_t* ring, uint64_t seq, uint64_t flag, bool head, T v)
    {
        dev::st_relaxed(&ring[seq & (SLOTS - 1)], (flag << 62) | (head ? HEAD_BIT : 0) |
                                                      ((seq & TAG_MASK) << 32) | (uint32_t)to_bits(v));
    }
    __device__ static bool read(const uint64_t* ring, uint64_t seq, uint64_t& flag, bool& head, T& v)
    {
        const uint64_t w = dev::ld_relaxed(&ring[seq & (SLOTS - 1)]);
        flag = w >> 62;
        if (flag == 0 || ((w >> 32) & TAG_MASK) != (seq & TAG_MASK)) return false;
        head = (w & HEAD_BIT) != 0;
        v = from_bits<T>((uint32_t)w);
        return true;
    }
};
template <typename T> struct SStatus<T, true> {  // halves of the value, as in the scan's status
    static constexpr uint64_t SLOTS = onesweep::RING_BYTES / 32;
    static constexpr uint64_t HEAD = HEAD_BIT >> 32;
    __device__ static uint64_t front(uint64_t flag, uint64_t seq) { return (flag << 30) | (seq & TAG_MASK); }
    __device__ static void publish(uint64_t* ring, uint64_t seq, uint64_t flag, bool head, T v)
    {
        uint64_t* s = ring + (seq & (SLOTS - 1)) * 4 + (flag == FLAG_PRE ? 2 : 0);
        const uint64_t bits = to_bits(v), h = (front(flag, seq) | (head ? HEAD : 0)) << 32;
        dev::st_relaxed2(s, h | (uint32_t)bits, h | (bits >> 32));
    }
    __device__ static bool read(const uint64_t* ring, uint64_t seq, uint64_t& flag, bool& head, T& v)
    {
        const uint64_t* s = ring + (seq & (SLOTS - 1)) * 4;
        uint64_t w[4];
        dev::ld_relaxed2(s, w[0], w[1]);
        dev::ld_relaxed2(s + 2, w[2], w[3]);
        const uint64_t pre = front(FLAG_PRE, seq), agg = front(FLAG_AGG, seq);
        const bool done = ((w[2] >> 32) & ~HEAD) == pre && ((w[3] >> 32) & ~HEAD) == pre;
        const uint64_t lo = done ? w[2] : w[0], hi = done ? w[3] : w[1];
        flag = done ? FLAG_PRE : FLAG_AGG;
        head = (lo & HEAD_BIT) != 0;
        v = from_bits<T>((hi << 32) | (uint32_t)lo);
        return done || (((lo >> 32) & ~HEAD) == agg && ((hi >> 32) & ~HEAD) == agg);
    }
};

template <typename T> struct SegScanArgs {
    const T* in;
    T* out;
    uint32_t n;
    T identity;
    int exclusive;
    int aligned;
    const uint32_t* off;
    uint32_t nseg;
    uint32_t num_tiles;
    uint64_t* ring;
    uint64_t seq0;
    uint32_t* tile_ctr;
    int* err;
};

// Inclusive scan of (flag, value) pairs across a warp, sequence order.
template <typename T, typename Op>
__device__ __forceinline__ void warp_seg_scan(uint32_t& f, T& v, Op op)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T yv = __shfl_up_sync(FULL_MASK, v, o);
        const uint32_t yf = __shfl_up_sync(FULL_MASK, f, o);
        if (lane >= o) {
            if (!f) v = op(yv, v);
            f |= yf;
        }
    }
}

template <typename T, typename Op>
__global__ void __launch_bounds__(THREADS) k_segscan(SegScanArgs<T> a)
{
    constexpr int VEC = 16 / sizeof(T);
    constexpr int ROWS = sizeof(T) == 4 ? 4 : 8;
    constexpr int TILE = THREADS * VEC * ROWS;
    constexpr int RW = ROWS * (THREADS / 32);
    constexpr int PER = RW / 32;

    __shared__ uint32_t s_head[TILE / 32];
    __shared__ T s_rw[RW];
    __shared__ uint32_t s_rwf[RW];
    __shared__ T s_prefix;
    __shared__ uint32_t s_tile, s_lo;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Op op;
    const T identity = a.identity;

    for (;;) {
        if (tid == 0) s_tile = atomicAdd(a.tile_ctr, 1u);
        for (int i = tid; i < TILE / 32; i += THREADS) s_head[i] = 0;
        __syncthreads();
        const uint32_t t = s_tile;
        if (t >= a.num_tiles) break;
        const uint32_t base = t * TILE;
        const bool full = base + TILE <= a.n;

        // Segment starts inside [base, base + TILE).
        if (tid == 0) {
            uint32_t lo = 0, hi = a.nseg;  // first i in [0, nseg) with off[i] >= base, else nseg
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (a.off[mid] < base) lo = mid + 1;
                else hi = mid;
            }
            s_lo = lo;
            if (base == 0) s_head[0] = 1u;  // position 0 always starts a segment
        }
        __syncthreads();
        for (uint32_t i = s_lo + tid; i < a.nseg; i += THREADS) {
            const uint32_t o = a.off[i];
            if (o >= base + TILE) break;
            if (o < base) continue;  // only with non-monotone offsets
            const uint32_t local = o - base;
            atomicOr(&s_head[local >> 5], 1u << (local & 31));
        }
        __syncthreads();

        T x[ROWS][VEC];
        uint32_t hb[ROWS];  // head bits of the thread's VEC elements, per row
        if (full && a.aligned) {
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                const uint4 w = dev::ld_stream(reinterpret_cast<const uint4*>(a.in + base + (r * THREADS + tid) * VEC));
                memcpy(x[r], &w, 16);
            }
        } else {
#pragma unroll
            for (int r = 0; r < ROWS; ++r)
#pragma unroll
                for (int j = 0; j < VEC; ++j) {
                    const uint32_t idx = base + (r * THREADS + tid) * VEC + j;
                    x[r][j] = idx < a.n ? a.in[idx] : identity;
                }
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const uint32_t l0 = (r * THREADS + tid) * VEC;
            hb[r] = (s_head[l0 >> 5] >> (l0 & 31)) & ((1u << VEC) - 1);
        }

        // Thread totals per row, then warp scans of the pairs.
        T wv[ROWS];
        uint32_t wf[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            T v = x[r][0];
#pragma unroll
            for (int j = 1; j < VEC; ++j) v = ((hb[r] >> j) & 1) ? x[r][j] : op(v, x[r][j]);
            uint32_t f = hb[r] != 0;
            warp_seg_scan(f, v, op);
            wv[r] = v;
            wf[r] = f;
            if (lane == 31) {
                s_rw[r * (THREADS / 32) + warp] = v;
                s_rwf[r * (THREADS / 32) + warp] = f;
            }
        }
        __syncthreads();

        if (warp == 0) {
            T v[PER];
            uint32_t f[PER];
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                v[k] = s_rw[lane * PER + k];
                f[k] = s_rwf[lane * PER + k];
            }
            T lv = v[0];
            uint32_t lf = f[0];
#pragma unroll
            for (int k = 1; k < PER; ++k) {
                lv = f[k] ? v[k] : op(lv, v[k]);
                lf |= f[k];
            }
            T iv = lv;
            uint32_t iff = lf;
            warp_seg_scan(iff, iv, op);
            const T uv = __shfl_up_sync(FULL_MASK, iv, 1);
            const uint32_t uf = __shfl_up_sync(FULL_MASK, iff, 1);
            // exclusive prefix of each row-warp (entry 0 has none)
            T rv = uv;
            uint32_t rf = lane == 0 ? 0u : uf;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                s_rw[lane * PER + k] = rv;
                s_rwf[lane * PER + k] = rf;
                if (lane == 0 && k == 0) {
                    rv = v[0];
                    rf = f[0];
                } else {
                    rv = f[k] ? v[k] : op(rv, v[k]);
                    rf |= f[k];
                }
            }
            const T agg = __shfl_sync(FULL_MASK, iv, 31);
            const bool agg_head = __shfl_sync(FULL_MASK, iff, 31) != 0;
            const uint64_t my_seq = a.seq0 + t;
            if (lane == 0) SStatus<T>::publish(a.ring, my_seq, t == 0 ? FLAG_PRE : FLAG_AGG, agg_head, agg);

            T excl = identity;
            if (t > 0) {
                bool have = false;
                int64_t w_end = t;
                for (;;) {
                    const int64_t k = w_end - 32 + lane;
                    uint64_t flag = FLAG_PRE;
                    bool head = true;
                    T val = identity;
                    bool gave_up = false;
                    if (k >= 0) {
                        if (!SStatus<T>::read(a.ring, a.seq0 + (uint64_t)k, flag, head, val)) {
                            const unsigned long long start = dev::globaltimer();
                            for (uint32_t spin = 1;; ++spin) {
                                if (SStatus<T>::read(a.ring, a.seq0 + (uint64_t)k, flag, head, val)) break;
                                if ((spin & 255) == 0 && dev::globaltimer() - start > dev::SPIN_LIMIT_NS) {
                                    gave_up = true;
                                    flag = FLAG_PRE;
                                    head = true;
                                    val = identity;
                                    break;
                                }
                                if (spin > 32) __nanosleep(64);
                            }
                        }
                    }
                    if (__any_sync(FULL_MASK, gave_up) && lane == 0) dev::raise_error(a.err, dev::ERR_LOOKBACK_TIMEOUT);
                    const bool stop = flag == FLAG_PRE || head;
                    const uint32_t stops = __ballot_sync(FULL_MASK, stop);
                    const int L = stops ? 31 - __clz(stops) : 0;
                    uint32_t cf = lane >= L ? (uint32_t)head : 0u;
                    T cv = lane >= L ? val : identity;
                    warp_seg_scan(cf, cv, op);
                    const T wsum = __shfl_sync(FULL_MASK, cv, 31);
                    const bool wflag = __shfl_sync(FULL_MASK, cf, 31) != 0;
                    (void)wflag;
                    // Nearer windows held no head and no prefix (else the walk
                    // would have stopped), so the farther window folds in
                    // front of what has been gathered so far.
                    excl = have ? op(wsum, excl) : wsum;
                    have = true;
                    if (stops) break;
                    w_end -= 32;
                }
                if (lane == 0)
                    SStatus<T>::publish(a.ring, my_seq, FLAG_PRE, true, agg_head ? agg : op(excl, agg));
            }
            if (lane == 0) s_prefix = excl;
        }
        __syncthreads();

        const T prefix = s_prefix;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const int rw = r * (THREADS / 32) + warp;
            const T wexc = __shfl_up_sync(FULL_MASK, wv[r], 1);
            const uint32_t wexf = __shfl_up_sync(FULL_MASK, wf[r], 1);
            T run = prefix;  // placeholder when nothing precedes (position 0 is a head)
            if (rw != 0) run = s_rwf[rw] ? s_rw[rw] : op(run, s_rw[rw]);
            if (lane > 0) run = wexf ? wexc : op(run, wexc);
            T o[VEC];
#pragma unroll
            for (int j = 0; j < VEC; ++j) {
                const bool head = (hb[r] >> j) & 1;
                const T inc = head ? x[r][j] : op(run, x[r][j]);
                o[j] = a.exclusive ? (head ? identity : run) : inc;
                run = inc;
            }
            if (full && a.aligned) {
                uint4 w;
                memcpy(&w, o, 16);
                *reinterpret_cast<uint4*>(a.out + base + (r * THREADS + tid) * VEC) = w;
            } else {
#pragma unroll
                for (int j = 0; j < VEC; ++j) {
                    const uint32_t idx = base + (r * THREADS + tid) * VEC + j;
                    if (idx < a.n) a.out[idx] = o[j];
                }
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Large inputs of 4-byte elements: the same scan as a pipeline inside each CTA
// (pipe.cuh), with a tile's (head, value) pair as its aggregate. The look-back
// form above is bound by the chain of publish and look-back from tile to tile
// (int32 over 200,000 lognormal segments, 3.8e8 elements: 1186 us, this one 649
// with its head bits).
//
// Head flags come as one bit per element, set in memory beforehand and copied
// with the tile: finding a tile's segments inside the kernel would cost a
// search (four dependent loads at least) per tile.
// ---------------------------------------------------------------------------
template <typename T> struct HeadValue {
    uint32_t head;  // a segment starts among the elements
    T v;            // their combination from the last start on
};
template <typename T, typename Op> struct HeadOp {
    Op op;
    __device__ HeadValue<T> operator()(const HeadValue<T>& a, const HeadValue<T>& b) const
    {
        return {a.head | b.head, b.head ? b.v : op(a.v, b.v)};
    }
};

// Sets the bit of every segment start below n, and of position 0. Neighbouring
// starts share a word: one atomic per word and warp.
__global__ void __launch_bounds__(256) k_heads(const uint32_t* off, uint32_t nseg, uint32_t n, uint32_t* heads)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&heads[0], 1u);
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < nseg; i0 += stride) {
        const uint64_t i = i0 + lane;
        const uint32_t o = i < nseg ? off[i] : 0xFFFFFFFFu;
        const uint32_t word = o < n ? o >> 5 : 0xFFFFFFFFu;
        const uint32_t peers = __match_any_sync(FULL_MASK, word);
        const uint32_t bits = __reduce_or_sync(peers, 1u << (o & 31));
        if (o < n && lane == (uint32_t)__ffs(peers) - 1) atomicOr(&heads[word], bits);
    }
}

template <typename T> struct SegPipeArgs {
    const T* in;
    T* out;
    const uint32_t* heads;
    uint32_t n;
    T identity;
    int exclusive;
    pipe::Tiles tiles;
};

constexpr uint32_t HEAD_TILE_BYTES = pipe::TILE_BYTES / 4 / 8;
constexpr std::size_t SEG_PIPE_SMEM = pipe::SMEM + pipe::STAGES * HEAD_TILE_BYTES;

template <typename T, typename Op>
__global__ void __launch_bounds__(pipe::THREADS, 1) k_segscan_pipe(SegPipeArgs<T> a)
{
    using namespace pipe;
    static_assert(sizeof(T) == 4, "four elements per lane and row");
    constexpr int VEC = 4;
    constexpr uint32_t TILE = TILE_BYTES / 4;
    using Pair = HeadValue<T>;
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char* head_stages = smem + pipe::SMEM;
    __shared__ Shared<Pair> sh;
    __shared__ Pair s_before[STAGES][WRITERS];
    const Tiles& tiles = a.tiles;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Op op;
    const HeadOp<T, Op> pair_op{};
    sh.init();
    if (warp == COPY_WARP)
        return copy_role<HEAD_TILE_BYTES>(tiles, sh, smem, a.in, (uint64_t)a.n * 4, head_stages, a.heads);
    // position 0 is a start, so nothing of `first` reaches an output
    if (warp == PREFIX_WARP) return prefix_role<false>(tiles, sh, Pair{0u, a.identity}, pair_op);

    // This lane's elements of a row of the tile and their head bits.
    auto load_row = [&](uint32_t t, int s, bool whole, int row, T (&x)[VEC]) -> uint32_t {
        const uint32_t word = row * 4 + lane / 8;
        uint32_t h;
        if (whole) {
            const uint4 v = reinterpret_cast<const uint4*>(smem + (std::size_t)s * TILE_BYTES)[row * 32 + lane];
            memcpy(x, &v, 16);
            h = reinterpret_cast<const uint32_t*>(head_stages + s * HEAD_TILE_BYTES)[word];
        } else {
#pragma unroll
            for (int j = 0; j < VEC; ++j) {
                const uint64_t at = (uint64_t)t * TILE + (row * 32 + lane) * VEC + j;
                x[j] = at < a.n ? a.in[at] : a.identity;
            }
            h = a.heads[(std::size_t)t * (TILE / 32) + word];
        }
        return (h >> (lane * 4 & 31)) & 15u;
    };
    // The lane's combination from its last head (or its first element) on,
    // then the same from the row's start to the lane; returns the lanes with
    // heads. A lane combines with lanes back to the last one with a head only.
    auto scan_row = [&](const T (&x)[VEC], uint32_t h, T& v) -> uint32_t {
        v = x[0];
#pragma unroll
        for (int j = 1; j < VEC; ++j) v = (h >> j & 1u) ? x[j] : op(v, x[j]);
        const uint32_t lanes = __ballot_sync(FULL_MASK, h != 0);
        const uint32_t mine = lanes & (0xFFFFFFFFu >> (31 - lane));
        const int from = mine != 0 ? 31 - __clz((int)mine) : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const T y = __shfl_up_sync(FULL_MASK, v, o);
            if (lane - o >= from) v = op(y, v);
        }
        return lanes;
    };

    if (warp >= WRITERS) {  // folding
        const int f = warp - WRITERS;
        for (uint32_t k = 0; k < limit(tiles); ++k) {
            const uint32_t t = sh.next(k, tiles.err);
            if (t == END) break;
            const bool whole = (uint64_t)(t + 1) * TILE <= a.n;
#pragma unroll
            for (int b = 0; b < BLOCKS; ++b) {
                Pair total{0u, a.identity};
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    T x[VEC], v;
                    const uint32_t h = load_row(t, k % STAGES, whole, (f * BLOCKS + b) * ROWS + r, x);
                    const uint32_t lanes = scan_row(x, h, v);
                    const Pair row{lanes != 0 ? 1u : 0u, v};
                    total = r == 0 ? row : pair_op(total, row);  // lane 31's
                }
                if (lane == 31) sh.total[k & 1][f * BLOCKS + b] = total;
            }
            publish_tile(tiles, sh, k, t, s_before[k % STAGES], pair_op);
        }
        return;
    }

    for (uint32_t k = 0; k < limit(tiles); ++k) {  // scanning and writing
        const int s = k % STAGES;
        const uint32_t t = sh.next(k, tiles.err);
        if (t == END) return;
        const bool whole = (uint64_t)(t + 1) * TILE <= a.n;
        T x[ROWS][VEC], incl[ROWS];
        uint32_t h[ROWS], lanes[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) h[r] = load_row(t, s, whole, warp * ROWS + r, x[r]);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) lanes[r] = scan_row(x[r], h[r], incl[r]);
        sh.wait(&sh.ready[s], k, tiles.err);
        T before = const_cast<const volatile Pair&>(sh.prefix[s]).v;  // since the last start before the block, then each row
        if (warp > 0) {
            const Pair p = s_before[s][warp];
            before = p.head ? p.v : op(before, p.v);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.empty[s]);  // the warp is done with the stage and its slots
        if (sh.abort) continue;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const T left = __shfl_up_sync(FULL_MASK, incl[r], 1);
            T run = before;
            if (lane > 0) run = (lanes[r] & dev::lanemask_lt()) != 0 ? left : op(before, left);
            const T last = __shfl_sync(FULL_MASK, incl[r], 31);
            before = lanes[r] != 0 ? last : op(before, last);
            T o[VEC];
#pragma unroll
            for (int j = 0; j < VEC; ++j) {
                const bool head = (h[r] >> j & 1u) != 0;
                const T inc = head ? x[r][j] : op(run, x[r][j]);
                o[j] = a.exclusive ? (head ? a.identity : run) : inc;
                run = inc;
            }
            const uint32_t at = t * TILE + ((warp * ROWS + r) * 32 + lane) * VEC;
            if (whole) {
                uint4 w;
                memcpy(&w, o, 16);
                *reinterpret_cast<uint4*>(a.out + at) = w;
            } else {
#pragma unroll
                for (int j = 0; j < VEC; ++j)
                    if (at + j < a.n) a.out[at + j] = o[j];
            }
        }
    }
}

// From here the pipeline wins for every segment length (int32, look-back /
// pipeline in us, segments of 20, 1000 and 100,000 elements): 2^26 elements 324 /
// 184, 229 / 137, 180 / 138; 2^24 74 / 66, 62 / 55, 51 / 55; 2^23 39 / 42, 34 / 38, 28 / 37.
constexpr std::size_t PIPE_MIN = std::size_t(1) << 25;

struct SegScanLaunch {
    device_context& ctx;
    const void* in;
    void* out;
    std::size_t n;
    const void* identity;
    bool exclusive;
    const uint32_t* off;
    std::size_t nseg;

    template <typename T, typename Op> void run()
    {
        if constexpr (sizeof(T) == 4) {
            if (n >= PIPE_MIN && ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0 &&
                ctx.smem_optin >= SEG_PIPE_SMEM + 8192 && run_pipe<T, Op>())
                return;
        }
        run_lookback<T, Op>();
    }

    // False when there is no memory for the head bits (or, under capture, none
    // in the pool): the look-back form needs none.
    template <typename T, typename Op> bool run_pipe()
    {
        constexpr uint32_t TILE = pipe::TILE_BYTES / sizeof(T);
        SegPipeArgs<T> a;
        a.tiles.num_tiles = (uint32_t)((n + TILE - 1) / TILE);
        const std::size_t head_bytes = (std::size_t)a.tiles.num_tiles * HEAD_TILE_BYTES;
        std::unique_ptr<temp_buffer> heads;
        try {
            heads = std::make_unique<temp_buffer>(ctx.resource, head_bytes);
        } catch (const out_of_memory&) {
            return false;
        } catch (const unsupported_error&) {
            return false;
        }
        check_cuda(cudaMemsetAsync(heads->get(), 0, head_bytes, ctx.stream), "cudaMemsetAsync");
        kernel_timer kt(ctx, "segscan.pipe");
        const int hgrid = (int)std::max<std::size_t>(1, std::min<std::size_t>((nseg + 255) / 256, (std::size_t)ctx.sm_count * 8));
        k_heads<<<hgrid, 256, 0, ctx.stream>>>(off, (uint32_t)nseg, (uint32_t)n, heads->as<uint32_t>());
        a.in = static_cast<const T*>(in);
        a.out = static_cast<T*>(out);
        a.heads = heads->as<uint32_t>();
        a.n = (uint32_t)n;
        std::memcpy(&a.identity, identity, sizeof(T));
        a.exclusive = exclusive ? 1 : 0;
        a.tiles.ring = ctx.lookback_ring;
        a.tiles.seq0 = ctx.reserve_seq(a.tiles.num_tiles);
        a.tiles.err = ctx.d_error;
        unsigned char* ctl = ctx.d_small + 256;
        check_cuda(cudaMemsetAsync(ctl, 0, 64, ctx.stream), "cudaMemsetAsync");
        a.tiles.counter = reinterpret_cast<uint32_t*>(ctl);
        auto kernel = &k_segscan_pipe<T, Op>;
        check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SEG_PIPE_SMEM),
                   "cudaFuncSetAttribute");
        const int grid = (int)std::min<std::size_t>(a.tiles.num_tiles, (std::size_t)ctx.sm_count);
        kernel<<<grid, pipe::THREADS, SEG_PIPE_SMEM, ctx.stream>>>(a);
        check_cuda(cudaGetLastError(), "segmented scan launch");
        return true;
    }

    template <typename T, typename Op> void run_lookback()
    {
        constexpr int VEC = 16 / sizeof(T);
        constexpr int ROWS = sizeof(T) == 4 ? 4 : 8;
        constexpr uint32_t TILE = THREADS * VEC * ROWS;
        SegScanArgs<T> a;
        a.in = static_cast<const T*>(in);
        a.out = static_cast<T*>(out);
        a.n = (uint32_t)n;
        std::memcpy(&a.identity, identity, sizeof(T));
        a.exclusive = exclusive ? 1 : 0;
        a.aligned = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
        a.off = off;
        a.nseg = (uint32_t)nseg;
        a.num_tiles = (uint32_t)((n + TILE - 1) / TILE);
        a.ring = ctx.lookback_ring;
        a.seq0 = ctx.reserve_seq(a.num_tiles);
        a.err = ctx.d_error;
        unsigned char* ctl = ctx.d_small + 256;
        check_cuda(cudaMemsetAsync(ctl, 0, 64, ctx.stream), "cudaMemsetAsync");
        a.tile_ctr = reinterpret_cast<uint32_t*>(ctl);
        auto kernel = &k_segscan<T, Op>;
        int per_sm = 0;
        check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, THREADS, 0),
                   "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
        const int grid = (int)std::min<std::size_t>(a.num_tiles, (std::size_t)ctx.sm_count * std::max(per_sm, 1));
        kernel_timer kt(ctx, "segscan.lookback");
        kernel<<<grid, THREADS, 0, ctx.stream>>>(a);
        check_cuda(cudaGetLastError(), "segmented scan launch");
    }
};

}  // namespace

void segmented_scan(device_context& ctx, const void* in, void* out, std::size_t n, elem t, op_kind op,
                    const void* identity, bool exclusive, const uint32_t* offsets, std::size_t num_segments)
{
    if (n == 0) return;
    check_size(n);
    if (in == nullptr || out == nullptr || identity == nullptr || (num_segments > 0 && offsets == nullptr))
        throw std::invalid_argument("segmented_scan: null argument");
    if (num_segments > 0x7FFFFFFFu) throw std::length_error("segmented_scan: too many segments");
    ctx.activate();
    SegScanLaunch l{ctx, in, out, n, identity, exclusive, offsets, num_segments};
    ops::dispatch(t, op, l);
}

}  // namespace gbc
