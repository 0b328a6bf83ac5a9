// Small decisions of the search kernels that depend on numbers alone, kept
// apart from the device code so that they compile and can be checked on the
// host too.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define DDP_RULE __host__ __device__ __forceinline__
#else
#define DDP_RULE static inline
#endif

namespace ddp {

// Entries of a one-CTA phase list (m pushed, at most list_cap of them in
// shared memory) that go back to a near queue of cap_q entries.  Entries past
// the shared list were written to the queue at once, with a check of their own;
// m > cap_q is an overflow of the queue.
DDP_RULE int local_handback(int m, int list_cap, int64_t cap_q) {
    const int k = m < list_cap ? m : list_cap;
    return k < cap_q ? k : (int)cap_q;
}

// Threads of a CTA for opts.block = want (> 0): whole warps, at most top (a
// multiple of 32).  The engines deal work out by warps: with part of a warp
// over, warps of the grid would not be warps of the hardware, and with fewer
// than 32 threads there would be none.
DDP_RULE int block_threads(int want, int top) { return want >= top ? top : (want + 31) & ~31; }

// Whether a graph's degrees are skewed: rows of more than 256 arcs hold a
// sixteenth of its arcs or more (of 2e, forward and reverse).  The bidirectional
// search opens no buckets ahead there (WAVE_AHEAD).
DDP_RULE int64_t long_row_arcs(int64_t len) { return len > 256 ? len : 0; }
DDP_RULE bool skewed_rows(int64_t in_long, int64_t arcs) { return in_long > 0 && in_long >= arcs / 16; }

}  // namespace ddp
