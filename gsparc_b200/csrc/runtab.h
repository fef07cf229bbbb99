// runtab.h -- the run lookup table of a group of jobs: for every 32 contract
// keys of a job the keys that have a run of Y (bits) and the first of these
// runs (first).  Written by k_y_runs (rows.cu), read by k_bmatch (batch.cu).
#pragma once

#include <cstdint>

#include "hd.h"

namespace gs {

// Whether a run of contract part c enters the table of a job of `ncbits`
// contract bits.  A Y index outside its mode can leave a part above that width
// where another job of the group has wider keys.  No X nonzero matches such a
// run, and it has no word of its own job: folded onto one, its run number would
// become the word's first one, and runs counted from there reach into the next
// job.  The parts of a job ascend, so the ones left out follow all its others
// and a word's first run is found among keys that are in.
GS_HD bool run_in_table(uint64_t c, int ncbits) { return ncbits >= 64 || c >> ncbits == 0; }

// Run of contract key c (of its job's width) from its word, `none` where it has none.
GS_HD uint64_t run_of_key(uint32_t bits, uint32_t first, uint64_t c, uint64_t none) {
    const uint32_t bit = 1u << (c & 31);
    if (!(bits & bit)) return none;
#ifdef __CUDA_ARCH__
    return (uint64_t)first + __popc(bits & (bit - 1u));
#else
    return (uint64_t)first + (uint64_t)__builtin_popcount(bits & (bit - 1u));
#endif
}

}  // namespace gs
