// Batched (segmented) sort and scan: entry points and tunables.
#pragma once

#include <cstddef>
#include <cstdint>

#include "runtime.hpp"

namespace gbc {

//! Launch-shape choices of the segmented sort (picked by the autotuner).
struct seg_options {
    int cta_cap = 0;  // largest segment a single CTA sorts in shared memory (0: the type's maximum)
    // device, one byte per segment or null: nonzero marks a segment already in
    // order (every key equal), left untouched; only for in-place calls
    const uint8_t* skip = nullptr;
    // MSD route: a large segment whose highest varying digit splits it into
    // buckets that fit a one-CTA sort of msd_cap keys (with room for a window
    // of neighbouring buckets) takes one pass on that digit, then the one-CTA
    // sorts finish the buckets; 0: every large segment takes all digit
    // passes; -1: the default (the tuning table's entry, else off for
    // 32-bit keys up to 2^26 of them and the one-CTA maximum otherwise: the
    // batch of 200,000 lognormal segments of u64 pairs takes 11.1 ms with its
    // scan, 27.0 with the one-CTA sorts of every digit and the route off)
    int msd_cap = -1;
    // threads of the one-CTA sorts of up to 4,096 keys: 256 (16 keys per
    // thread) or 512 (8). 0: the tuning table's entry for this workload (the
    // segmented key with ":threads", stored by the autotuner), else its
    // "segsort:cta_threads" entry, else 256. The longer classes have 512 or
    // 1,024 threads.
    int cta_threads = 0;
    // the keys of a segment differ in this many of their lowest 8-bit digits at
    // most (0: in any); the passes over the others are not launched
    int low_digits = 0;
    // few launches, all on the context's stream: for calls that mostly have
    // little to do or nothing
    bool sparse = false;
    // scratch of the call's n keys (and values), or null: from the context's arena
    void* alt_keys = nullptr;
    uint32_t* alt_vals = nullptr;
};

//! Sorts every segment [offsets[i], offsets[i+1]) independently and stably.
//! offsets has num_segments + 1 monotone entries (device memory); keys_in ==
//! keys_out sorts in place. Asynchronous; graph-capturable once the pool is
//! warm (every temporary then comes from the cache).
void segmented_sort(device_context& ctx, const void* keys_in, void* keys_out, int key_bytes, int key_kind,
                    const uint32_t* vals_in, uint32_t* vals_out, std::size_t n, const uint32_t* offsets,
                    std::size_t num_segments, bool descending, const seg_options& opt);

//! The same in place for 64-bit keys (and values, or null) whose order is that
//! of dev::KeyXform{xf_a, xf_b} applied to them.
void segmented_sort_xf(device_context& ctx, uint64_t* keys, uint32_t* vals, uint64_t xf_a, uint64_t xf_b, std::size_t n,
                       const uint32_t* offsets, std::size_t num_segments, const seg_options& opt);

//! Scan restarted at every segment start (offsets as for segmented_sort;
//! position 0 always starts a segment). Exclusive: a segment's first output
//! is the identity.
void segmented_scan(device_context& ctx, const void* in, void* out, std::size_t n, elem t, op_kind op,
                    const void* identity, bool exclusive, const uint32_t* offsets, std::size_t num_segments);

std::string segsort_tuning_key(int key_bytes, bool has_values, std::size_t n, std::size_t num_segments);
//! The tuning-table key of the batch's launch form. There is one form, the launch
//! sequence; entries that older tables hold for others change nothing.
std::string segsort_batch_tuning_key(int key_bytes, bool has_values, std::size_t n, std::size_t num_segments);
//! The tuning-table key of the one-CTA sorts' thread count (256 or 512; one
//! entry for every segmented sort of the context).
std::string segsort_cta_threads_tuning_key();
//! The tuning-table key of the one-CTA sorts' thread count for one workload
//! class (the segmented key with ":threads").
std::string segsort_threads_tuning_key(int key_bytes, bool has_values, std::size_t n, std::size_t num_segments);
//! The tuning-table key of the MSD route's bucket capacity (0: off).
std::string segsort_msd_tuning_key(int key_bytes, bool has_values, std::size_t n, std::size_t num_segments);

//! Largest segment the segmented sort finishes in one CTA's shared memory.
uint32_t segsort_cta_cap(int key_bytes, bool has_values);

}  // namespace gbc
