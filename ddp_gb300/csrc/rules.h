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

}  // namespace ddp
