// tri.h -- rows of an M x M vector X(p, q) = X[p + M q] with X^T = +-X that a
// sum needs: the entries p <= q, those off the diagonal twice.
//
// Slot i of tri_slots(M) pairs column v with column M-1-v, so that every
// M + 1 slots hold two contiguous runs: (w, v) for w <= v, then (w - v - 1,
// M-1-v).  For odd M the middle column pairs with itself and its second run
// is void.
#pragma once
#include <cstdint>

namespace de {

inline int64_t tri_slots(int64_t m) { return (m + 1) / 2 * (m + 1); }

// Row of slot i and its weight (2 off the diagonal); false for a void slot.
__device__ __forceinline__ bool tri_row(unsigned i, unsigned m, int64_t &row, double &weight)
{
    const unsigned v = i / (m + 1), w = i - v * (m + 1);
    const bool first = w <= v;
    const unsigned p = first ? w : w - v - 1, q = first ? v : m - 1 - v;
    row = p + (int64_t)m * q;
    weight = p == q ? 1.0 : 2.0;
    return first || q != v;
}

}  // namespace de
