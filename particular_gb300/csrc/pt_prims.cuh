// Device-wide primitives used by the Barnes-Hut build: scratch for the scans of pt_scan.cuh
// and a stable radix sort of u64 keys and their indices.
#pragma once

#include "pt_common.cuh"

namespace pt {

// Scratch for the primitives; grow-only, owned by a subsystem.
struct PrimScratch {
    DevBuf scan;   // tile totals of a scan
    DevBuf hist;   // radix histograms / offsets, the flags of a sort
    DevBuf keys2;  // ping-pong keys
    DevBuf vals2;  // ping-pong values
};

// Sorting n keys takes two calls: radix_sort_prepare before the keys are produced tells the
// producer where to put them (first->keys, or the caller's own array where that is null) and,
// for small n, to count their first digits: hist[(i / tile) * 256 + (key >> shift & 255)]
// for key i where hist is not null. radix_sort_u64 then leaves the keys ascending by
// their low `bits` bits in keys, equal ones in the order of their index, and their indices in
// vals.
struct RadixFirst {
    uint64_t *keys;
    uint32_t *hist;
    int shift, tile;
    // n large, else null: the producer sets it where many keys share their bits from shift on
    int *deep;
    uint32_t *zero;  // words that have to be zero before the keys are produced
    int zero_words;
};
int radix_sort_prepare(pt_ctx *ctx, PrimScratch &s, int n, int bits, RadixFirst *first);
int radix_sort_u64(pt_ctx *ctx, PrimScratch &s, uint64_t *keys, uint32_t *vals, int n, int bits);

void prim_free(pt_ctx *ctx, PrimScratch &s);

}  // namespace pt
