// Onesweep-style LSD radix sort of (u64 key, u32 index) pairs (sort.cu).
#pragma once

#include <algorithm>

#include "common.cuh"

namespace nbody {

// Histogram and status slots of one sort scratch. A slot holds the digit counts
// of one pass and that pass's tile status words and ticket; every pass of one
// build takes a different slot. The passes of a plan take slots 0 .. 15, those of
// the full sort (k_full_sort) kFullSlot onwards.
constexpr int kSortSlots = 34;
constexpr int kFullSlot = 16;
constexpr uint32_t kSortTile = 4096;  // keys per tile

// Right shift of pass q (0-based, least significant digit first) when `passes`
// 8-bit digits sort a 63-bit key word from its top bit down: all 64 bits,
// byte-aligned, for 8 passes; otherwise bits [63 - 8 passes, 63), the word's
// top 8 passes key bits (bit 63 is always zero).
__host__ __device__ inline int digit_shift(int passes, int q) { return passes >= 8 ? 8 * q : 63 - 8 * passes + 8 * q; }
// The same for a full 64-bit key (the system's number above the first key word).
__host__ __device__ inline int digit_shift64(int passes, int q) { return 64 - 8 * passes + 8 * q; }

// Layout of a sort scratch of 32-bit words: the digit counts of every slot, 128
// counters (a ticket per slot, then the full sort's), the status words per slot.
constexpr size_t kSortCounters = kSortSlots * 256;
constexpr size_t kSortStatus = kSortCounters + 128;
constexpr int kFullCounters = 64;  // first of the full sort's counters

// Bytes of device scratch for sorting n pairs.
size_t sort_scratch_bytes(uint32_t n);
// Words from the start of the scratch to be zero before the sorts of `passes` slots
// (a multiple of 4). The full sort zeroes its own status words.
size_t sort_zero_words(uint32_t n, int passes);

// Zeroes the scratch for `passes` slots.
cudaError_t sort_reset(uint32_t *scratch, uint32_t n, int passes, cudaStream_t st);

// Digit counts of a 63-bit word (8 passes) into slots slot ...
cudaError_t sort_histograms(const uint64_t *w, int slot, uint32_t n, uint32_t *scratch, cudaStream_t st,
                            unsigned *launches);

// One stable pass by the 8-bit digit (key >> shift) & 255, with the digit
// counts, status words and ticket of `slot` (the counts of that slot must have
// been taken with the same shift). A look-back that gives up waiting ORs err_bit
// into *err.
cudaError_t sort_pass(const uint64_t *kin, const uint32_t *iin, uint64_t *kout, uint32_t *iout, uint32_t n, int slot,
                      int shift, uint32_t *scratch, uint32_t *err, uint32_t err_bit, cudaStream_t st,
                      unsigned *launches);

// The full sort by (system,) first and second key words, in one launch that
// returns at once unless *run_if is non-zero (null: always runs). k1 and k2 are in
// user order; k2 is computed here unless have_k2. Results: idx_a, the words in that
// order in key_b (first) and key_a (second), and sys_sorted.
struct FullSort {
    uint64_t *key_a, *key_b;
    const uint64_t *k1;
    uint64_t *k2;
    uint32_t *idx_a, *idx_b;
    const uint32_t *sys_id;  // null: one system
    uint32_t *sys_sorted;
    uint32_t n;
    uint32_t *scratch;
    uint32_t *err, err_bit;
    const uint32_t *run_if;
    int have_k2;
    const double *pos;
    const DevScalars *sc;
    const double *sys_root;
    int single;
};
cudaError_t sort_full(const FullSort &f, cudaStream_t st, unsigned *launches);

}  // namespace nbody
