// lv_sym.h -- symmetry check of a level's entries, shared by the kernels that
// sum it and the host tests.
#pragma once
#include "lv_rng.h"

namespace lv {

// A 64-bit mix of one directed entry.  The pair is mixed in full before the
// weight joins, and the two are mixed in full again, so that the difference of
// two weights' mixes depends on the pair in every bit (a weight added before a
// single round cancelled against its mirror entry's other weight for one pair
// in 2^24).
LVRNG_HD uint64_t sym_mix(uint32_t a, uint32_t b, uint64_t w) {
    return lvrng::mix64(lvrng::mix64((uint64_t)a << 32 | b) + w);
}

// One entry's share: the sum over all entries of mix(row, col, w) -
// mix(col, row, w) is zero when the entries and their mirror images are the
// same multiset.  The mix is fixed; for entries that were not made to cancel
// under it the sum is otherwise zero by a chance of about 2^-64.
LVRNG_HD uint64_t sym_share(int32_t v, int32_t j, uint64_t w) {
    return sym_mix((uint32_t)v, (uint32_t)j, w) - sym_mix((uint32_t)j, (uint32_t)v, w);
}

}  // namespace lv
