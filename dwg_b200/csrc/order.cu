// order.cu -- spatial order of a caller's point queries: one counting sort by
// the Morton code of a coarse cell.  A warp that walks the octree for 32
// queries shares the walk only as far as they lie together; a caller's points
// come in any order.
#include <cub/cub.cuh>

#include "order.cuh"

namespace dwg {

namespace {

// the low 10 bits of v, two zero bits between them
__device__ __forceinline__ unsigned spread3(unsigned v) {
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    return (v | (v << 2)) & 0x09249249u;
}

struct Cube {
    float lo[3], scale;
    int cells;
};

__device__ __forceinline__ unsigned cube_cell(float x, float lo, float scale, int cells) {
    const int c = (int)((x - lo) * scale);  // (a NaN gives 0, beyond the range the end)
    return (unsigned)(c < 0 ? 0 : c >= cells ? cells - 1 : c);
}

__global__ void k_query_key(const float* __restrict__ q, long long nq, Cube c, int* __restrict__ key,
                            int* __restrict__ hist) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nq;
         i += (long long)gridDim.x * blockDim.x) {
        const unsigned k = spread3(cube_cell(q[i * 3], c.lo[0], c.scale, c.cells)) |
                           (spread3(cube_cell(q[i * 3 + 1], c.lo[1], c.scale, c.cells)) << 1) |
                           (spread3(cube_cell(q[i * 3 + 2], c.lo[2], c.scale, c.cells)) << 2);
        key[i] = (int)k;
        atomicAdd(&hist[k], 1);
    }
}

__global__ void k_query_place(const int* __restrict__ key, long long nq, int* __restrict__ fill,
                              int* __restrict__ order) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nq;
         i += (long long)gridDim.x * blockDim.x)
        order[atomicAdd(&fill[key[i]], 1)] = (int)i;
}

}  // namespace

static int call_memory(QueryOrder& w, size_t bytes, cudaStream_t s) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    DWG_CHECK_CUDA(cudaStreamIsCapturing(s, &cs));
    if (cs != cudaStreamCaptureStatusNone) return DWG_OK;
    const cudaError_t e = cudaMallocAsync(&w.mem, bytes, s);
    if (e != cudaSuccess) w.mem = nullptr;
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        return DWG_OK;
    }
    DWG_CHECK_CUDA(e);
    w.stream = s;
    return DWG_OK;
}

int work_counter(QueryOrder& w, cudaStream_t s) {
    DWG_TRY(call_memory(w, sizeof(int), s));
    if (!w.mem) return DWG_OK;
    DWG_CHECK_CUDA(cudaMemsetAsync(w.mem, 0, sizeof(int), s));
    w.counter = (unsigned int*)w.mem;
    return DWG_OK;
}

int query_order(QueryOrder& w, const float* q, long long nq, const double root[4], cudaStream_t s, const int** order) {
    *order = nullptr;
    if (nq >= (1ll << 31) || !(root[3] > 0)) return DWG_OK;
    // ~4 queries of a surface per cell, at most 2^21 cells (clearing and
    // scanning their counts takes 10 us)
    int bits = 4;
    while (bits < 7 && (4ll << (2 * bits)) < nq) ++bits;
    const int cells = 1 << bits, buckets = 1 << (3 * bits);
    Cube c;
    for (int d = 0; d < 3; ++d) c.lo[d] = (float)(root[d] - 0.5 * root[3]);
    c.scale = (float)(cells / root[3]);
    c.cells = cells;
    size_t scan = 0;
    DWG_CHECK_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, scan, (int*)nullptr, (int*)nullptr, buckets, s));
    // keys, order, counts and the counter, places, the scan's storage
    const size_t keys = ((size_t)nq * sizeof(int) + 255) / 256 * 256, counts = (size_t)buckets * sizeof(int);
    DWG_TRY(call_memory(w, 2 * keys + 2 * counts + 256 + scan, s));
    if (!w.mem) return DWG_OK;
    char* const at = (char*)w.mem;
    int *key = (int*)at, *out = (int*)(at + keys), *hist = (int*)(at + 2 * keys), *fill = hist + buckets + 64;
    DWG_CHECK_CUDA(cudaMemsetAsync(hist, 0, counts + sizeof(int), s));
    w.counter = (unsigned int*)(hist + buckets);
    long long blocks = (nq + 255) / 256;
    if (blocks > (long long)num_sms() * 8) blocks = (long long)num_sms() * 8;
    k_query_key<<<(unsigned)blocks, 256, 0, s>>>(q, nq, c, key, hist);
    DWG_CHECK_LAUNCH();
    DWG_CHECK_CUDA(cub::DeviceScan::ExclusiveSum(at + 2 * keys + 2 * counts + 256, scan, hist, fill, buckets, s));
    k_query_place<<<(unsigned)blocks, 256, 0, s>>>(key, nq, fill, out);
    DWG_CHECK_LAUNCH();
    *order = out;
    return DWG_OK;
}

}  // namespace dwg
