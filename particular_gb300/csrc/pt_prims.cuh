// Device-wide primitives used by the Barnes-Hut build: scratch for the scans of pt_scan.cuh
// and a stable LSD radix sort of (u64 key, u32 value) pairs.
#pragma once

#include "pt_common.cuh"

namespace pt {

// Scratch for the primitives; grow-only, owned by a subsystem.
struct PrimScratch {
    DevBuf scan;   // tile totals of a scan
    DevBuf hist;   // radix histograms / offsets
    DevBuf keys2;  // ping-pong keys
    DevBuf vals2;  // ping-pong values
};

// Sorts keys (and their values) ascending by the low `bits` bits, stably. The
// result ends in keys/vals.
int radix_sort_u64(pt_ctx *ctx, PrimScratch &s, uint64_t *keys, uint32_t *vals, int n, int bits);

void prim_free(pt_ctx *ctx, PrimScratch &s);

}  // namespace pt
