// order.cuh -- spatial order of a caller's point queries.
#pragma once

#include "common.cuh"

namespace dwg {

// buffers of one owner's calls (grown on demand, one call at a time)
struct QueryOrder {
    DevBuf<int> key, order, hist, fill;
    DevBuf<unsigned char> scratch;
};

// *order[j] = index of the j-th query when the queries q (packed xyz) are
// taken by the Morton code of their cell in the cube root (centre, width),
// coarse cells in any order inside; null when they are to be taken as they
// come: while `s` is being captured (a graph must not hold buffers that a
// later call may grow), or beyond 2^31 queries.
int query_order(QueryOrder& w, const float* q, long long nq, const double root[4], cudaStream_t s, const int** order);

}  // namespace dwg
