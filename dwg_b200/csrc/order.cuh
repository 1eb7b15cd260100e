// order.cuh -- spatial order of a caller's point queries.
#pragma once

#include "common.cuh"

namespace dwg {

// One call's buffers, allocated and released in the order of the call's stream:
// calls on several streams share nothing.
struct QueryOrder {
    QueryOrder() = default;
    ~QueryOrder() {
        if (mem) cudaFreeAsync(mem, stream);
    }
    QueryOrder(const QueryOrder&) = delete;
    QueryOrder& operator=(const QueryOrder&) = delete;
    void* mem = nullptr;
    cudaStream_t stream = nullptr;
    unsigned int* counter = nullptr;  // 0, for a launch's work
};

// *order[j] = index of the j-th query when the queries q (packed xyz) are
// taken by the Morton code of their cell in the cube root (centre, width),
// coarse cells in any order inside, valid for work queued on s while w lives;
// null when they are to be taken as they come: while `s` is being captured (a
// graph would hold memory of this call), beyond 2^31 queries, or when there is
// no memory for it.
//
// w.counter comes with an order; work_counter gives one alone (null in the same cases).
int work_counter(QueryOrder& w, cudaStream_t s);
int query_order(QueryOrder& w, const float* q, long long nq, const double root[4], cudaStream_t s, const int** order);

}  // namespace dwg
