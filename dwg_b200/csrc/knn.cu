// knn.cu -- exact kNN over a uniform cell grid.
//
// The reference builds a left-balanced kd-tree with log2(N) thrust sorts and
// walks it per query with a 30-entry stack (src/KNN_GWN.cu:42-66,490-715,
// include/cudaKDTree/cukd/traverse-cct.h:25-101).  Point clouds here are
// surfaces, so a uniform grid sized for 3 to 4 points per occupied cell is
// built with one counting sort (histogram, scan, scatter).  Up to k = 16 a
// query reads the points within a trial radius of it (k_knn_near) and the
// queries far from the points walk an occupancy pyramid in groups
// (k_knn_far); above, a thread per query visits shells of cells and then the
// pyramid (k_knn_thread).  Candidates are ranked by the cukd key (float bits
// of dist^2) << 32 | index (include/cudaKDTree/cukd/knn.h:279-282), with
// dist^2 = (dx*dx + dy*dy) + dz*dz in round-to-nearest single precision.
#include <cub/cub.cuh>

#include <cfloat>
#include <climits>
#include <type_traits>
#include <vector>

#include "knn.cuh"
#include "octree.cuh"

namespace dwg {

// work that runs only when a device count exceeds a minimum
struct Gate {
    const int* count = nullptr;
    int min = 0;
    __device__ __forceinline__ bool closed() const { return count && *count <= min; }
};

// The searches compare a query with cells and nodes in coordinates relative
// to the grid's corner lo: a point's cell is that of fl(p - lo), so the
// rounding of every step is a part of the grid's extent, however far from the
// origin the cloud lies (faces at lo + i h would be rounded at |lo|, which
// moves them by cells).  In units of 2^-24 extents, a point's cell carries at
// most 3 (the difference, 1 / h, the product), a face i h - eps 2 and a
// query's difference 1, and the extent is at most max(G) cells: eps widens
// boxes and reaches by 8 of them, and 1e-4 cells: below a thousandth of a cell
// (max(G) <= 1024) whatever the cloud's size, so a reach stays a few cells.
struct KnnGrid {
    int G0, G1, G2;
    float lo0, lo1, lo2, h, inv_h, eps;
};

static KnnGrid grid_of(const KnnIndex& ix) {
    const int most = max(ix.G[0], max(ix.G[1], ix.G[2]));
    const float eps = (1e-4f + (float)most * (1.f / 2097152.f)) * ix.h;  // (8 * 2^-24 = 2^-21)
    return KnnGrid{ix.G[0], ix.G[1], ix.G[2], ix.lo[0], ix.lo[1], ix.lo[2], ix.h, ix.inv_h, eps};
}

// the cell of a relative coordinate, and of a point's
__device__ __forceinline__ int cell_at(float u, float inv_h, int G) {
    const int c = (int)floorf(__fmul_rn(u, inv_h));
    return c < 0 ? 0 : (c >= G ? G - 1 : c);
}
__device__ __forceinline__ int cell_coord(float p, float lo, float inv_h, int G) {
    return cell_at(__fsub_rn(p, lo), inv_h, G);
}

__global__ void k_knn_hist(const float* __restrict__ P, int n, KnnGrid g, int* __restrict__ counts,
                           int* __restrict__ cell_of) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int cx = cell_coord(P[(size_t)i * 3], g.lo0, g.inv_h, g.G0);
    int cy = cell_coord(P[(size_t)i * 3 + 1], g.lo1, g.inv_h, g.G1);
    int cz = cell_coord(P[(size_t)i * 3 + 2], g.lo2, g.inv_h, g.G2);
    int c = cx + g.G0 * (cy + g.G1 * cz);
    cell_of[i] = c;
    atomicAdd(&counts[c], 1);
}

__global__ void k_knn_scatter(const float* __restrict__ P, int n, const int* __restrict__ cell_of,
                              int* __restrict__ fill, float4* __restrict__ pts) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int slot = atomicAdd(&fill[cell_of[i]], 1);
    pts[slot] = make_float4(P[(size_t)i * 3], P[(size_t)i * 3 + 1], P[(size_t)i * 3 + 2], __int_as_float(i));
}

// The occupancy pyramid: node c of level l >= 1 holds the mask of its
// occupied children (bit t for the child 2 * (i, j, k) + (t & 1, t >> 1 & 1,
// t >> 2), cells at level 1), so a node is occupied iff its byte is nonzero
// and a walk skips empty children without loading them.  One launch fills
// every level of a zeroed pyramid: a thread per level-1 node ORs in its mask,
// then climbs while it is the first child to make its parent nonzero (the old
// byte of the OR), so every occupied node's bit reaches its parent once and
// no thread waits for another.
struct PyrDims {
    int levels;
    int ldim[KnnIndex::kMaxLevels][3];
    long long loff[KnnIndex::kMaxLevels];
};

// OR v into the byte at p (a 32-bit atomic on its word; the buffer is padded
// to whole words); returns the byte before
__device__ __forceinline__ unsigned atomic_or_byte(unsigned char* p, unsigned v) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    unsigned* w = reinterpret_cast<unsigned*>(a & ~(uintptr_t)3);
    const unsigned sh = (unsigned)(a & 3) * 8u;
    return (atomicOr(w, v << sh) >> sh) & 0xffu;
}

__global__ void k_pyr_fill(const int* __restrict__ cell_start, int G0, int G1, int G2, PyrDims pd,
                           unsigned char* __restrict__ occ, Gate gate) {
    if (gate.closed()) return;
    const int D0 = pd.ldim[1][0], D1 = pd.ldim[1][1], D2 = pd.ldim[1][2];
    const long long m = (long long)D0 * D1 * D2;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < m;
         c += (long long)gridDim.x * blockDim.x) {
        int i = (int)(c % D0), j = (int)((c / D0) % D1), k = (int)(c / ((long long)D0 * D1));
        unsigned o = 0;
        for (int t = 0; t < 8; ++t) {
            const int x = 2 * i + (t & 1), y = 2 * j + ((t >> 1) & 1), z = 2 * k + (t >> 2);
            if (x >= G0 || y >= G1 || z >= G2) continue;
            const long long f = x + (long long)G0 * (y + (long long)G1 * z);
            o |= (cell_start[f + 1] > cell_start[f] ? 1u : 0u) << t;
        }
        if (!o) continue;
        atomic_or_byte(occ + pd.loff[1] + c, o);
        for (int l = 2; l <= pd.levels; ++l) {
            const int t = (i & 1) | ((j & 1) << 1) | ((k & 1) << 2);
            i >>= 1;
            j >>= 1;
            k >>= 1;
            const long long p = pd.loff[l] + i + (long long)pd.ldim[l][0] * (j + (long long)pd.ldim[l][1] * k);
            if (atomic_or_byte(occ + p, 1u << t) != 0) break;  // the parent was occupied: its ancestors know
        }
    }
}

// level dimensions and offsets of the occupancy pyramid of ix's grid
static int pyramid_dims(KnnIndex& ix) {
    ix.levels = 0;
    int d[3] = {ix.G[0], ix.G[1], ix.G[2]};
    ix.ldim[0][0] = d[0];
    ix.ldim[0][1] = d[1];
    ix.ldim[0][2] = d[2];
    long long total = 0;
    int L = 0;
    while (d[0] > 1 || d[1] > 1 || d[2] > 1) {
        DWG_REQUIRE(L + 1 < KnnIndex::kMaxLevels, "knn: grid too large for the occupancy pyramid");
        ++L;
        for (int t = 0; t < 3; ++t) {
            d[t] = (d[t] + 1) / 2;
            ix.ldim[L][t] = d[t];
        }
        ix.loff[L] = total;
        total += (long long)d[0] * d[1] * d[2];
    }
    ix.levels = L;
    // padded to whole 32-bit words (the fill ORs bytes through word atomics)
    if (L > 0) DWG_TRY(ix.occ.reserve((size_t)total + 4));
    return DWG_OK;
}

// the occupancy masks of every level from ix.cell_start (stream-ordered)
static int pyramid_fill(KnnIndex& ix, Gate gate, cudaStream_t s) {
    if (ix.levels < 1) return DWG_OK;
    PyrDims pd;
    pd.levels = ix.levels;
    for (int l = 0; l < KnnIndex::kMaxLevels; ++l) {
        pd.loff[l] = ix.loff[l];
        for (int d = 0; d < 3; ++d) pd.ldim[l][d] = ix.ldim[l][d];
    }
    DWG_CHECK_CUDA(cudaMemsetAsync(ix.occ.ptr, 0, ix.occ.n, s));
    const long long m = (long long)ix.ldim[1][0] * ix.ldim[1][1] * ix.ldim[1][2];
    long long blocks = div_up(m, 256);
    const long long cap = (long long)num_sms() * 8;
    if (blocks > cap) blocks = cap;
    k_pyr_fill<<<(unsigned)blocks, 256, 0, s>>>(ix.cell_start.ptr, ix.G[0], ix.G[1], ix.G[2], pd, ix.occ.ptr,
                                                  gate);
    DWG_CHECK_LAUNCH();
    return DWG_OK;
}

static int build_pyramid(KnnIndex& ix, cudaStream_t s) {
    DWG_TRY(pyramid_dims(ix));
    return pyramid_fill(ix, Gate{}, s);
}

int knn_build(KnnIndex& ix, const float* P, int n, cudaStream_t s) {
    DWG_REQUIRE(P != nullptr && n >= 1, "knn: need at least one point (n=%d)", n);
    FreeScope on_s(s, false);  // the temporaries are used on s alone
    DWG_TRY(require_finite(P, 3ll * n, "knn", s));
    ix.n = n;
    DWG_TRY(ix.bbox.reserve(6));
    DWG_TRY(bbox_device(P, n, ix.bbox.ptr, s));
    float bb[6];
    DWG_CHECK_CUDA(cudaMemcpyAsync(bb, ix.bbox.ptr, sizeof(bb), cudaMemcpyDeviceToHost, s));
    DWG_CHECK_CUDA(cudaStreamSynchronize(s));
    float ext[3], emax = 0.f;
    for (int d = 0; d < 3; ++d) {
        ext[d] = bb[3 + d] - bb[d];
        emax = fmaxf(emax, ext[d]);
    }
    if (!(emax > 0.f)) emax = 1.f;
    // ~3 points per occupied cell for a surface sample
    double gm = ceil(sqrt((double)n / 14.0));
    if (gm < 1) gm = 1;
    if (gm > 1024) gm = 1024;
    // (no cell below 1e-12: eps and the radii, thousandths of a cell, keep
    // normal squares; the points of a cloud that small share a few cells)
    float h = fmaxf((float)(emax / gm) * 1.0001f, 1e-12f);
    for (;;) {
        long long tot = 1;
        for (int d = 0; d < 3; ++d) {
            int G = (int)ceil(ext[d] / h);
            if (G < 1) G = 1;
            ix.G[d] = G;
            tot *= G;
        }
        if (tot <= (1ll << 27)) break;
        h *= 1.25f;
    }
    ix.h = h;
    ix.inv_h = 1.0f / h;
    for (int d = 0; d < 3; ++d) ix.lo[d] = bb[d];
    long long ncell = (long long)ix.G[0] * ix.G[1] * ix.G[2];
    const KnnGrid g = grid_of(ix);
    DevBuf<int> counts, cell_of;
    DWG_TRY(counts.reserve(ncell + 1));
    DWG_TRY(cell_of.reserve(n));
    DWG_TRY(ix.cell_start.reserve(ncell + 1));
    DWG_TRY(ix.cell_fill.reserve(ncell + 1));
    DWG_TRY(ix.pts.reserve(n));
    DWG_CHECK_CUDA(cudaMemsetAsync(counts.ptr, 0, sizeof(int) * (ncell + 1), s));
    k_knn_hist<<<div_up(n, 256), 256, 0, s>>>(P, n, g, counts.ptr, cell_of.ptr);
    DWG_CHECK_LAUNCH();
    size_t bytes = 0;
    int* cin = counts.ptr;
    int* cout = ix.cell_start.ptr;
    DWG_CHECK_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, bytes, cin, cout, (int)(ncell + 1), s));
    DWG_TRY(ix.scratch.reserve(bytes + 256));
    bytes = ix.scratch.n;
    DWG_CHECK_CUDA(cub::DeviceScan::ExclusiveSum(ix.scratch.ptr, bytes, cin, cout, (int)(ncell + 1), s));
    DWG_CHECK_CUDA(cudaMemcpyAsync(ix.cell_fill.ptr, ix.cell_start.ptr, sizeof(int) * (ncell + 1),
                                   cudaMemcpyDeviceToDevice, s));
    k_knn_scatter<<<div_up(n, 256), 256, 0, s>>>(P, n, cell_of.ptr, ix.cell_fill.ptr, ix.pts.ptr);
    DWG_CHECK_LAUNCH();
    DWG_TRY(build_pyramid(ix, s));
    DWG_CHECK_CUDA(cudaStreamSynchronize(s));
    return DWG_OK;
}

struct KnnArgs {
    KnnGrid g;
    const float4* __restrict__ pts;
    const int* __restrict__ cell_start;
    const float* __restrict__ q;
    const int* __restrict__ q_index;
    const float* __restrict__ q_source;
    long long nq;
    const unsigned long long* nq_dev;
    const int* nq_dev_i32;
    const int* gate_count;
    int gate_min;
    int k;
    int* __restrict__ out;
    const int* __restrict__ order;  // query processing order (spatially bucketed)
    int* __restrict__ q_key;
    int* __restrict__ q_hist;
    int morton_shift;
    // the queries that k_knn_far finishes, a bound on the k-th squared
    // distance of each, the groups (first entry, entries), and the counts of
    // entries and groups
    int* __restrict__ far_list;
    float* __restrict__ far_bound;
    int2* __restrict__ far_group;
    unsigned int* __restrict__ far_count;
    // per query (null: none): a key above its k-th nearest key, ~0 for none
    const unsigned long long* __restrict__ seed;
    // occupancy pyramid
    const unsigned char* __restrict__ occ;
    int levels;
    int ldim[KnnIndex::kMaxLevels][3];
    long long loff[KnnIndex::kMaxLevels];
};

__device__ __forceinline__ long long knn_count(const KnnArgs& a) {
    long long nq = a.nq;
    if (a.nq_dev) {
        unsigned long long d = *a.nq_dev;
        if ((long long)d < nq) nq = (long long)d;
    }
    if (a.nq_dev_i32) {
        long long d = *a.nq_dev_i32;
        if (d < nq) nq = d;
    }
    return nq;
}

__device__ __forceinline__ void knn_load_query(const KnnArgs& a, long long qi, float& qx, float& qy, float& qz) {
    if (a.q_index) {
        long long src = a.q_index[qi];
        qx = a.q_source[src * 3];
        qy = a.q_source[src * 3 + 1];
        qz = a.q_source[src * 3 + 2];
    } else {
        qx = a.q[qi * 3];
        qy = a.q[qi * 3 + 1];
        qz = a.q[qi * 3 + 2];
    }
}

// the low 10 bits of v, two zero bits between them
__device__ __forceinline__ unsigned spread10(unsigned v) {
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

// bucket the queries by the Morton code of their coarse cell
__global__ void k_knn_qkey(KnnArgs a) {
    if (a.gate_count && *a.gate_count <= a.gate_min) return;
    const long long nq = knn_count(a);
    for (long long qi = blockIdx.x * (long long)blockDim.x + threadIdx.x; qi < nq;
         qi += (long long)gridDim.x * blockDim.x) {
        float qx, qy, qz;
        knn_load_query(a, qi, qx, qy, qz);
        unsigned cx = cell_coord(qx, a.g.lo0, a.g.inv_h, a.g.G0) >> a.morton_shift;
        unsigned cy = cell_coord(qy, a.g.lo1, a.g.inv_h, a.g.G1) >> a.morton_shift;
        unsigned cz = cell_coord(qz, a.g.lo2, a.g.inv_h, a.g.G2) >> a.morton_shift;
        int key = (int)(spread10(cx) | (spread10(cy) << 1) | (spread10(cz) << 2));
        a.q_key[qi] = key;
        atomicAdd(&a.q_hist[key], 1);
    }
}

__global__ void k_knn_qscatter(KnnArgs a, int* __restrict__ fill, int* __restrict__ order) {
    if (a.gate_count && *a.gate_count <= a.gate_min) return;
    const long long nq = knn_count(a);
    for (long long qi = blockIdx.x * (long long)blockDim.x + threadIdx.x; qi < nq;
         qi += (long long)gridDim.x * blockDim.x)
        order[atomicAdd(&fill[a.q_key[qi]], 1)] = (int)qi;
}

// top-k state of one lane: an unsorted set of KMAX keys and its maximum
// (value, slot) of the largest of v[LO, LO + N), the lowest slot among equal
// values (what a scan from LO with a strict comparison finds), by a
// tournament: depth log2 N instead of a chain of N - 1 dependent compares
template <int LO, int N, typename T, int M>
__device__ __forceinline__ void tour_max(const T (&v)[M], T& m, int& p) {
    if constexpr (N == 1) {
        m = v[LO];
        p = LO;
    } else {
        T m1, m2;
        int p1, p2;
        tour_max<LO, N / 2>(v, m1, p1);
        tour_max<LO + N / 2, N - N / 2>(v, m2, p2);
        const bool r = m2 > m1;
        m = r ? m2 : m1;
        p = r ? p2 : p1;
    }
}

// Batcher's odd-even merge sort on 16 inputs, 63 comparators in 10 layers
// (the iterative form: for p = 1, 2, 4, 8, for d = p, p/2, ..., 1, for j =
// d mod p, step 2d, for i < d, join i + j and i + j + d when both lie in the
// same block of 2p); comparator t orders slots kSortLo[t] < kSortHi[t]
constexpr int kSortNet = 63;
constexpr unsigned char kSortLo[kSortNet] = {0, 2, 4, 6, 8, 10, 12, 14, 0, 1, 4, 5, 8, 9, 12, 13, 1, 5, 9, 13, 0, 1, 2, 3, 8, 9, 10, 11, 2, 3, 10, 11, 1, 3, 5, 9, 11, 13, 0, 1, 2, 3, 4, 5, 6, 7, 4, 5, 6, 7, 2, 3, 6, 7, 10, 11, 1, 3, 5, 7, 9, 11, 13};
constexpr unsigned char kSortHi[kSortNet] = {1, 3, 5, 7, 9, 11, 13, 15, 2, 3, 6, 7, 10, 11, 14, 15, 2, 6, 10, 14, 4, 5, 6, 7, 12, 13, 14, 15, 4, 5, 12, 13, 2, 4, 6, 10, 12, 14, 8, 9, 10, 11, 12, 13, 14, 15, 8, 9, 10, 11, 4, 5, 8, 9, 12, 13, 2, 4, 6, 8, 10, 12, 14};

template <int KMAX>
struct TopK {
    unsigned long long e[KMAX];
    unsigned long long mx;  // the k-th key (max of the set) or NONE
    int mpos;
    int fill;  // keys entered so far, up to k: the slots fill in order before any maximum search
    __device__ __forceinline__ void init(int k) {
#pragma unroll
        for (int q = 0; q < KMAX; ++q) e[q] = q < k ? ~0ull : 0ull;  // unused slots never become the max
        mx = ~0ull;
        mpos = 0;
        fill = 0;
    }
    // enter v (v < mx): the first k keys take the slots in turn (the
    // maximum stays the initial key until the last slot is taken, then it is
    // searched once), later keys replace the maximum
    __device__ __forceinline__ void push(unsigned long long v, int k) {
        if (fill < k) {
#pragma unroll
            for (int q = 0; q < KMAX; ++q)
                if (q == fill) e[q] = v;
            if (++fill == k) {
                max_slot();
            }
        } else {
            replace_max(v);
        }
    }
    __device__ __forceinline__ void order(int lo, int hi) {
        const unsigned long long a = e[lo], b = e[hi];
        e[lo] = a < b ? a : b;
        e[hi] = a < b ? b : a;
    }
    // the 16 slots from LO
    template <int LO, int T = 0>
    __device__ __forceinline__ void sort_net() {
        if constexpr (T < kSortNet) {
            constexpr int lo = LO + kSortLo[T], hi = LO + kSortHi[T];
            order(lo, hi);
            sort_net<LO, T + 1>();
        }
    }
    // sorted runs of RUN slots from LO on, merged in pairs: the first layer
    // joins each slot with its mirror image, the others are half-cleaners
    template <int RUN>
    __device__ __forceinline__ void merge_runs() {
        if constexpr (RUN < KMAX) {
#pragma unroll
            for (int lo = 0; lo < KMAX; lo += 2 * RUN) {
#pragma unroll
                for (int q = 0; q < RUN; ++q) order(lo + q, lo + 2 * RUN - 1 - q);
#pragma unroll
                for (int d = RUN / 2; d > 0; d >>= 1)
#pragma unroll
                    for (int q = 0; q < 2 * RUN; ++q)
                        if (!(q & d)) order(lo + q, lo + q + d);
            }
            merge_runs<2 * RUN>();
        }
    }
    template <int LO = 0>
    __device__ __forceinline__ void sort_blocks() {
        if constexpr (LO < KMAX) {
            sort_net<LO>();
            sort_blocks<LO + 16>();
        }
    }
    // mx and mpos: the largest key and its lowest slot
    __device__ __forceinline__ void max_slot() {
        if constexpr (KMAX <= 32) {
            tour_max<0, KMAX>(e, mx, mpos);
        } else {
            mx = e[0];
            mpos = 0;
#pragma unroll
            for (int q = 1; q < KMAX; ++q)
                if (e[q] > mx) {
                    mx = e[q];
                    mpos = q;
                }
        }
    }
    // replace the maximum by v (v < mx) and find the new maximum (a warp's
    // lanes take the same steps whether or not their slots are all filled)
    __device__ __forceinline__ void replace_max(unsigned long long v) {
#pragma unroll
        for (int q = 0; q < KMAX; ++q)
            if (q == mpos) e[q] = v;
        max_slot();
    }
    // ascending order (once per query): up to 32 slots the networks, more
    // slots an insertion sort in local memory
    __device__ __forceinline__ void sort() {
        if constexpr (KMAX <= 32) {
            static_assert(KMAX > 32 || KMAX % 16 == 0, "blocks of 16 slots, merged in pairs");
            sort_blocks();
            merge_runs<16>();
        } else {
            unsigned long long t[KMAX];
#pragma unroll
            for (int q = 0; q < KMAX; ++q) t[q] = e[q];
#pragma unroll 1
            for (int q = 1; q < KMAX; ++q) {
                const unsigned long long v = t[q];
                int p = q - 1;
                while (p >= 0 && t[p] > v) {
                    t[p + 1] = t[p];
                    --p;
                }
                t[p + 1] = v;
            }
#pragma unroll
            for (int q = 0; q < KMAX; ++q) e[q] = t[q];
        }
    }
};

// Exact continuation of a query's search over the occupancy pyramid, after
// the Chebyshev shells 0 and 1 around its cell (cx, cy, cz) were scanned.
// Depth-first from the 1x1x1 top level, the children of a node in the order
// of their octant's distance from the query's octant (same octant, then the
// three face neighbours, the three edge neighbours, the opposite one); a
// node is skipped when it is empty (its bit in the parent's child mask: no
// load) or its (eps-widened) box is farther than the current k-th candidate.
// The walk is stackless: a 4-bit child counter per level in one 64-bit word,
// the child masks of the nodes on the path (a byte per level in two 64-bit
// words) and the current node's coordinates.
template <int KMAX>
__device__ __forceinline__ void knn_pyramid(const KnnArgs& a, float qx, float qy, float qz, int cx, int cy, int cz,
                                            TopK<KMAX>& top) {
    const unsigned long long NONE = ~0ull;
    const float h = a.g.h;
    const float eps = a.g.eps;
    const float ux = __fsub_rn(qx, a.g.lo0), uy = __fsub_rn(qy, a.g.lo1), uz = __fsub_rn(qz, a.g.lo2);
    const int top_l = a.levels;
    int lvl = top_l, ci = 0, cj = 0, ck = 0;
    unsigned long long ctr = 0;
    // byte l of (mk1:mk0): the child mask of the path's node at level l
    unsigned long long mk0 = 0ull, mk1 = 0ull;
    {
        const unsigned long long tm = (unsigned long long)a.occ[a.loff[top_l]] << (8 * (top_l & 7));
        if (top_l < 8) mk0 = tm;
        else mk1 = tm;
    }
    for (;;) {
        const int sh = 4 * lvl;
        const int c = (int)((ctr >> sh) & 15ull);
        if (c == 8) {
            if (lvl == top_l) break;
            ctr &= ~(15ull << sh);
            ++lvl;
            ci >>= 1;
            cj >>= 1;
            ck >>= 1;
            continue;
        }
        ctr += 1ull << sh;
        // octant of the query about the node's midpoint
        const int half = 1 << (lvl - 1);
        const float mx = (float)((ci << lvl) + half) * h;
        const float my = (float)((cj << lvl) + half) * h;
        const float mz = (float)((ck << lvl) + half) * h;
        const int qo = (ux >= mx ? 1 : 0) | (uy >= my ? 2 : 0) | (uz >= mz ? 4 : 0);
        const int oc = qo ^ (int)((0x76534210u >> (4 * c)) & 7u);
        // empty or outside the grid (such children have no bit)
        if (!(((lvl < 8 ? mk0 : mk1) >> (8 * (lvl & 7) + oc)) & 1ull)) continue;
        const int nl = lvl - 1;
        const int ni = (ci << 1) | (oc & 1), nj = (cj << 1) | ((oc >> 1) & 1), nk = (ck << 1) | (oc >> 2);
        const float kd2 = top.mx == NONE ? INFINITY : __uint_as_float((unsigned)(top.mx >> 32)) * 1.00001f;
        const float x0 = (float)(ni << nl) * h - eps, x1 = (float)((ni + 1) << nl) * h + eps;
        const float y0 = (float)(nj << nl) * h - eps, y1 = (float)((nj + 1) << nl) * h + eps;
        const float z0 = (float)(nk << nl) * h - eps, z1 = (float)((nk + 1) << nl) * h + eps;
        const float ddx = fmaxf(0.f, fmaxf(x0 - ux, ux - x1));
        const float ddy = fmaxf(0.f, fmaxf(y0 - uy, uy - y1));
        const float ddz = fmaxf(0.f, fmaxf(z0 - uz, uz - z1));
        if (ddx * ddx + ddy * ddy + ddz * ddz > kd2) continue;
        if (nl == 0) {
            if (abs(ni - cx) <= 1 && abs(nj - cy) <= 1 && abs(nk - cz) <= 1) continue;  // scanned already
            const int cell = ni + a.g.G0 * (nj + a.g.G1 * nk);
            const int e = a.cell_start[cell + 1];
            for (int t = a.cell_start[cell]; t < e; ++t) {
                const float4 pp = a.pts[t];
                const int id = __float_as_int(pp.w);
                const float d2 = sq3_rn(__fsub_rn(pp.x, qx), __fsub_rn(pp.y, qy), __fsub_rn(pp.z, qz));
                const unsigned long long v = ((unsigned long long)__float_as_uint(d2) << 32) | (unsigned)id;
                if (v < top.mx) top.push(v, a.k);
            }
            continue;
        }
        const int* D = a.ldim[nl];
        const unsigned long long cm = a.occ[a.loff[nl] + ni + (long long)D[0] * (nj + (long long)D[1] * nk)];
        const int bs = 8 * (nl & 7);
        if (nl < 8) mk0 = (mk0 & ~(0xffull << bs)) | (cm << bs);
        else mk1 = (mk1 & ~(0xffull << bs)) | (cm << bs);
        lvl = nl;
        ci = ni;
        cj = nj;
        ck = nk;
    }
}

// k > 16: one thread per query; queries are processed in the order of their coarse
// Morton bucket so that neighbouring threads search neighbouring cells.  A
// query visits Chebyshev shells of cells around its own cell; a cell is
// skipped when its box is farther than the current k-th candidate; the k best
// keys are an unsorted register set whose maximum is kept in a register
// (replace-the-maximum on insertion, one sort at the end).  The search stops
// when the k-th key is closer than the boundary of the visited block.
template <int KMAX>
__global__ void __launch_bounds__(128) k_knn_thread(KnnArgs a) {
    if (a.gate_count && *a.gate_count <= a.gate_min) return;
    const long long nq = knn_count(a);
    const unsigned long long NONE = ~0ull;
    const int k = a.k;
    const float h = a.g.h;
    const float eps = a.g.eps;
    for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < nq;
         j += (long long)gridDim.x * blockDim.x) {
        const long long qi = a.order ? a.order[j] : j;
        float qx, qy, qz;
        knn_load_query(a, qi, qx, qy, qz);
        const float ux = __fsub_rn(qx, a.g.lo0), uy = __fsub_rn(qy, a.g.lo1), uz = __fsub_rn(qz, a.g.lo2);
        const int cx = cell_at(ux, a.g.inv_h, a.g.G0);
        const int cy = cell_at(uy, a.g.inv_h, a.g.G1);
        const int cz = cell_at(uz, a.g.inv_h, a.g.G2);
        TopK<KMAX> top;
        top.init(k);
        for (int r = 0;; ++r) {
            const float kd2 = top.mx == NONE ? INFINITY : __uint_as_float((unsigned)(top.mx >> 32)) * 1.00001f;
            for (int dz = -r; dz <= r; ++dz) {
                const int z = cz + dz;
                if (z < 0 || z >= a.g.G2) continue;
                const float z0 = (float)z * h - eps, z1 = z0 + h + 2.f * eps;
                const float ddz = fmaxf(0.f, fmaxf(z0 - uz, uz - z1));
                for (int dy = -r; dy <= r; ++dy) {
                    const int y = cy + dy;
                    if (y < 0 || y >= a.g.G1) continue;
                    const float y0 = (float)y * h - eps, y1 = y0 + h + 2.f * eps;
                    const float ddy = fmaxf(0.f, fmaxf(y0 - uy, uy - y1));
                    const float dyz = ddy * ddy + ddz * ddz;
                    if (dyz > kd2) continue;
                    const bool face = (dz == -r || dz == r || dy == -r || dy == r);
                    const int step = face ? 1 : (r > 0 ? 2 * r : 1);
                    for (int dx = -r; dx <= r; dx += step) {
                        const int x = cx + dx;
                        if (x < 0 || x >= a.g.G0) continue;
                        const float x0 = (float)x * h - eps, x1 = x0 + h + 2.f * eps;
                        const float ddx = fmaxf(0.f, fmaxf(x0 - ux, ux - x1));
                        if (ddx * ddx + dyz > kd2) continue;
                        const int c = x + a.g.G0 * (y + a.g.G1 * z);
                        const int e = a.cell_start[c + 1];
                        for (int t = a.cell_start[c]; t < e; ++t) {
                            const float4 pp = a.pts[t];
                            const int id = __float_as_int(pp.w);
                            const float d2 =
                                sq3_rn(__fsub_rn(pp.x, qx), __fsub_rn(pp.y, qy), __fsub_rn(pp.z, qz));
                            const unsigned long long v = ((unsigned long long)__float_as_uint(d2) << 32) | (unsigned)id;
                            if (v < top.mx) top.push(v, k);
                        }
                    }
                }
            }
            if (cx - r <= 0 && cy - r <= 0 && cz - r <= 0 && cx + r >= a.g.G0 - 1 && cy + r >= a.g.G1 - 1 &&
                cz + r >= a.g.G2 - 1)
                break;
            if (top.mx != NONE) {
                float bd = INFINITY;
                if (cx - r > 0) bd = fminf(bd, ux - (float)(cx - r) * h);
                if (cx + r < a.g.G0 - 1) bd = fminf(bd, (float)(cx + r + 1) * h - ux);
                if (cy - r > 0) bd = fminf(bd, uy - (float)(cy - r) * h);
                if (cy + r < a.g.G1 - 1) bd = fminf(bd, (float)(cy + r + 1) * h - uy);
                if (cz - r > 0) bd = fminf(bd, uz - (float)(cz - r) * h);
                if (cz + r < a.g.G2 - 1) bd = fminf(bd, (float)(cz + r + 1) * h - uz);
                bd -= eps;
                if (bd > 0.f && __uint_as_float((unsigned)(top.mx >> 32)) < bd * bd * 0.9999f) break;
            }
            if (r == 1 && a.levels > 0) {
                knn_pyramid<KMAX>(a, qx, qy, qz, cx, cy, cz, top);
                break;
            }
        }
        top.sort();
        // slots >= k hold 0 (below every key) and sort first; results start at KMAX - k
#pragma unroll
        for (int t = 0; t < KMAX; ++t) {
            const int o = t - (KMAX - k);
            if (o >= 0) a.out[qi * k + o] = top.e[t] == NONE ? -1 : (int)(unsigned)(top.e[t] & 0xffffffffu);
        }
    }
}

// -------------------------------------------------------- near queries --
// k <= 16: kNearLanes lanes per query.  A query reads the points within a
// trial radius of it: cells are x-fastest, so the cells of one row (y, z)
// within the radius hold one contiguous run of points.  The lanes list the
// rows' runs, join them into one list and walk it a point each; the keys
// within the radius go to shared memory, and when there are k a bitonic sort
// over the query's lanes orders them.  The first radius: a query a short way
// from one that has its k points finds k within that one's radius and the
// way; else it follows the density around the query's cell, ~1.35 k points.
// A round that finds fewer than k is followed by one that reads the shell up
// to 1.5 times the radius, and past the widest the query goes to k_knn_far, as
// does one with more keys than are kept (from its radius).  A query with a
// seed within reach starts from the seed's radius.  Instructions bound it
// (80 % of issue slots): 305,000 queries of a uniform sphere of 10,000 points,
// up to a cell off it, took 2,310 per warp and 4 queries with the keys' ranks
// counted (807 of them the ranks), 280 us with the queries' order; sorted
// 241 us.  250,000 on 100,000 points 242 -> 221 us (430 us with one warp per
// cell streaming the cell's ball; a thread per query keeping a sorted set
// waited on its loads).
constexpr int kNearThreads = 128;
constexpr int kNearLanes = 8;  // lanes per query
constexpr int kNearRuns = 4;   // rows a lane lists before it reads their points
constexpr int kNearKeys = 64;  // keys kept per query
constexpr int kNearUnit = 64;  // queries a warp takes at a time, at most
constexpr float kNearFirst = 1.35f * 11.f / 3.14159265f;  // first radius^2 in cells^2: this k / points near
constexpr float kNearMost = 4.f;                          // at most this
constexpr float kNearWay = 0.4f;                          // a way to a query with its points, in their radius
// the widest radius, in cells
constexpr float kNearWidest = 3.3f;
// a window of cells about a query is at most 15 wide then, so a row's number
// stays below 2^8
static_assert(kNearWidest < 6.9f, "rows of a window are numbered below 2^8");

// the KMAX smallest keys, ascending (k < KMAX: the first KMAX - k slots hold
// 0); an insertion is 2 compares and 2 selects of 64 bits per slot, without
// branches, and leaves the set sorted for the output
template <int KMAX>
struct SortedK {
    unsigned long long e[KMAX];
    __device__ __forceinline__ void init(int k, unsigned long long T) {
#pragma unroll
        for (int q = 0; q < KMAX; ++q) e[q] = q < KMAX - k ? 0ull : T;
    }
    __device__ __forceinline__ unsigned long long last() const { return e[KMAX - 1]; }
    // the largest squared distance kept (NaN while a slot is empty)
    __device__ __forceinline__ float last_d2() const { return __uint_as_float((unsigned)(e[KMAX - 1] >> 32)); }
    __device__ __forceinline__ void insert(unsigned long long v) {
#pragma unroll
        for (int q = KMAX - 1; q > 0; --q) e[q] = v < e[q] ? (v < e[q - 1] ? e[q - 1] : v) : e[q];
        e[0] = v < e[0] ? v : e[0];
    }
    // the k keys' indices (-1 in empty slots)
    __device__ __forceinline__ void store(int* __restrict__ out, int k) const {
#pragma unroll
        for (int t = 0; t < KMAX; ++t) {
            const int o = t - (KMAX - k);
            if (o >= 0) out[o] = e[t] == ~0ull ? -1 : (int)(unsigned)(e[t] & 0xffffffffu);
        }
    }
};

// Far queries waiting in a warp: position and query, bound
struct FarWait {
    float4 q[64];
    float bound[64];
};

// a square root rounded up (1e-4 over: the approximation's error is below 1e-6)
__device__ __forceinline__ float sqrt_up(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y * 1.0001f;
}

// n (1 to 32) of them go to the far list, split into groups of queries near
// each other: within 4 cells, or an eighth of the bound, of the group's first
__device__ __forceinline__ void far_groups(const KnnArgs& a, const FarWait& f, int n, int lane) {
    const unsigned FULL = 0xffffffffu;
    unsigned pos = 0;
    if (lane == 0) pos = atomicAdd(a.far_count, (unsigned)n);
    pos = __shfl_sync(FULL, pos, 0);
    const float4 q = f.q[lane];
    const float b = f.bound[lane];
    unsigned left = n == 32 ? FULL : (1u << n) - 1u;
    while (left) {
        const int first = __ffs(left) - 1;
        const float dx = q.x - __shfl_sync(FULL, q.x, first), dy = q.y - __shfl_sync(FULL, q.y, first),
                    dz = q.z - __shfl_sync(FULL, q.z, first);
        const float b0 = __shfl_sync(FULL, b, first);
        const float reach = fmaxf(16.f * a.g.h * a.g.h, b0 < INFINITY ? b0 * (1.f / 64.f) : 0.f);
        const bool in = lane == first || (((left >> lane) & 1u) && dx * dx + dy * dy + dz * dz <= reach);
        const unsigned m = __ballot_sync(FULL, in);
        if (in) {
            const unsigned o = pos + __popc(m & ((1u << lane) - 1u));
            a.far_list[o] = __float_as_int(q.w);
            a.far_bound[o] = b;
        }
        if (lane == 0) a.far_group[atomicAdd(a.far_count + 1, 1u)] = make_int2((int)pos, __popc(m));
        pos += __popc(m);
        left &= ~m;
    }
    __syncwarp();
}

// Keys of a query over its lanes, U to a lane (place = lane U + slot).
// key_none comes after every key.
__device__ __forceinline__ double key_none() { return __hiloint2double(0x7ff00000, 0); }

// bitonic merge of runs of N places: ascending where (place & N) is 0 or N is
// everything, descending elsewhere
template <int U, int N>
__device__ __forceinline__ void merge_keys(double (&v)[U], int sub) {
    constexpr unsigned FULL = 0xffffffffu;
    const bool down = N < U * kNearLanes && N >= U && ((sub * U) & N);
#pragma unroll
    for (int d = N / 2; d > 0; d >>= 1) {
        if (d >= U) {
            const bool high = (sub & (d / U)) != 0;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const double x = __shfl_xor_sync(FULL, v[u], d / U);
                v[u] = (x < v[u]) != (high != down) ? x : v[u];
            }
        } else {
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (!(u & d)) {
                    const bool swap = (v[u + d] < v[u]) != (N < U ? (u & N) != 0 : down);
                    const double x = v[u];
                    v[u] = swap ? v[u + d] : x;
                    v[u + d] = swap ? x : v[u + d];
                }
        }
    }
}
template <int U, int N = 2>
__device__ __forceinline__ void sort_keys(double (&v)[U], int sub) {
    merge_keys<U, N>(v, sub);
    if constexpr (N < U * kNearLanes) sort_keys<U, 2 * N>(v, sub);
}

__global__ void __launch_bounds__(kNearThreads) k_knn_near(KnnArgs a, unsigned int* __restrict__ work) {
    constexpr int G = kNearLanes, QW = 32 / G;  // lanes per query, queries per warp
    // a key's bits read as a double order like the key (d2 <= +inf: the
    // exponent stays below the NaNs'), and compare in one instruction
    __shared__ __align__(16) double keys[kNearThreads / G][kNearKeys];
    __shared__ int2 runs[kNearThreads / G][G * kNearRuns];
    __shared__ FarWait far[kNearThreads / 32];
    if (a.gate_count && *a.gate_count <= a.gate_min) return;
    const long long nq = knn_count(a);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int sub = lane & (G - 1);
    const unsigned FULL = 0xffffffffu;
    const unsigned mine = ((1u << G) - 1u) << (lane & ~(G - 1));  // the query's lanes
    const unsigned before = mine & ((1u << lane) - 1u);
    double* const key = keys[tid / G];
    int2* const run = runs[tid / G];
    const unsigned long long NONE = ~0ull;
    const int k = a.k;
    const float h = a.g.h;
    const float eps = a.g.eps;
    const float widest = kNearWidest * h;
    // a warp takes a run of consecutive queries at a time, short when the
    // launch's warps (one per 4 queries, up to a full GPU) would be left idle;
    // the far ones among them form the groups of the far search
    const long long warps = (long long)gridDim.x * (kNearThreads / 32);
    const unsigned unit = (unsigned)(max((long long)QW, min((long long)kNearUnit, nq / (2 * warps))) / QW * QW);
    unsigned base = 0, end = 0;
    int nfar = 0;  // queries waiting (warp-uniform)
    // the slot's last query and the radius of its k points
    float lx = 0.f, ly = 0.f, lz = 0.f, lr = INFINITY;
    for (;;) {
        if (base == end || (long long)base >= nq) {
            if (nfar > 0) {
                far_groups(a, far[w], nfar, lane);
                nfar = 0;
            }
            if (lane == 0) base = atomicAdd(work, unit);
            base = __shfl_sync(FULL, base, 0);
            end = base + unit;
        }
        if ((long long)base >= nq) break;
        const long long j = (long long)base + lane / G;
        const bool has = j < nq;
        const long long qi = !has ? 0 : a.order ? a.order[j] : j;
        base += QW;
        float qx = 0.f, qy = 0.f, qz = 0.f, seed2 = INFINITY;
        bool search = has, wait = false;
        if (has) {
            knn_load_query(a, qi, qx, qy, qz);
            if (a.seed) {
                const unsigned long long T = a.seed[qi];
                if (T != NONE) seed2 = __uint_as_float((unsigned)(T >> 32));
            }
            // a NaN has no neighbours
            search = !(isnan(qx) || isnan(qy) || isnan(qz));
        }
        int found = 0;  // keys of the query
        // The first radius: a surface through the 3x3x3 block around the
        // query's cell covers ~11 faces of cells, so 1.35 k points lie within
        // r^2 = 1.35 k 11 / (pi N) cells^2 for N points in the block
        const float ux = __fsub_rn(qx, a.g.lo0), uy = __fsub_rn(qy, a.g.lo1), uz = __fsub_rn(qz, a.g.lo2);
        const int cx = cell_at(ux, a.g.inv_h, a.g.G0), cy = cell_at(uy, a.g.inv_h, a.g.G1),
                  cz = cell_at(uz, a.g.inv_h, a.g.G2);
        float hi2 = INFINITY;
        // A query a short way from one that has its k points finds k within
        // their radius and the way; the last four queries are asked
        if (a.levels > 0) {
            float r = INFINITY;
#pragma unroll
            for (int s = 0; s < 32; s += G) {
                const float dx = qx - __shfl_sync(FULL, lx, s), dy = qy - __shfl_sync(FULL, ly, s),
                            dz = qz - __shfl_sync(FULL, lz, s), rs = __shfl_sync(FULL, lr, s);
                const float way = sqrt_up(dx * dx + dy * dy + dz * dz);
                if (way <= kNearWay * rs) r = fminf(r, rs + way);
            }
            hi2 = r * r;
            bool need = search && !(hi2 <= widest * widest) && !(seed2 <= widest * widest);
            if (__any_sync(FULL, need)) {
                int near = 0;
                if (need) {
                    const int x0 = max(cx - 1, 0), x1 = min(cx + 1, a.g.G0 - 1) + 1;
#pragma unroll
                    for (int u = 0; u < (9 + G - 1) / G; ++u) {
                        const int i = u * G + sub, y = cy + i % 3 - 1, z = cz + i / 3 - 1;
                        if (i < 9 && y >= 0 && y < a.g.G1 && z >= 0 && z < a.g.G2) {
                            const int* row = a.cell_start + a.g.G0 * (y + a.g.G1 * z);
                            near += row[x1] - row[x0];
                        }
                    }
                }
#pragma unroll
                for (int o = G / 2; o > 0; o >>= 1) near += __shfl_xor_sync(FULL, near, o);
                if (need) hi2 = fminf(__fdividef(kNearFirst * (float)k, (float)near), kNearMost) * (h * h);
            }
        }
        if (seed2 <= widest * widest) hi2 = seed2;
        // (cells so wide that their squares overflow: the far search reads no
        // rows of a square's width)
        if (search && a.levels > 0 && !(widest * widest < INFINITY)) {
            wait = true;
            search = false;
        }
        float lo2 = -1.f;  // the round reads the points with lo2 < d2 <= hi2
        while (__any_sync(FULL, search)) {
            // the rows (y, z) of cells within the radius
            const float out2 = hi2 * 1.00001f, reach = sqrt_up(hi2) + eps;
            const int y0 = cell_at(uy - reach, a.g.inv_h, a.g.G1);
            const int ny = cell_at(uy + reach, a.g.inv_h, a.g.G1) - y0 + 1;
            const int z0 = cell_at(uz - reach, a.g.inv_h, a.g.G2);
            const int nrow = search ? ny * (cell_at(uz + reach, a.g.inv_h, a.g.G2) - z0 + 1) : 0;
            // row i is (i % ny, i / ny), i / ny = i * inv >> 16 (exact for
            // ny <= 15, i < 2^8)
            const unsigned inv = (unsigned)__fdividef(65536.f, (float)ny) + 1u;
            const float by = (float)y0 * h - eps - uy, bz = (float)z0 * h - eps - uz;
            const float wide = h + 2.f * eps;
            for (int rb = 0; __any_sync(FULL, rb < nrow); rb += G * kNearRuns) {
                // the lane's runs of this batch of rows
                int s[kNearRuns], e[kNearRuns];
#pragma unroll
                for (int u = 0; u < kNearRuns; ++u) {
                    const int i = rb + u * G + sub;
                    s[u] = e[u] = 0;
                    if (i < nrow) {
                        const int iz = (int)((unsigned)i * inv >> 16), iy = i - iz * ny;
                        // distance of the row's (eps-widened) face
                        const float fy = by + (float)iy * h, fz = bz + (float)iz * h;
                        const float ddy = fmaxf(0.f, fmaxf(fy, -fy - wide));
                        const float ddz = fmaxf(0.f, fmaxf(fz, -fz - wide));
                        const float rest = out2 - (ddy * ddy + ddz * ddz);
                        // (all rows within an infinite radius, whose rest
                        // is a NaN for a query at infinity)
                        if (!(rest < 0.f)) {
                            const float hx = sqrt_up(rest) + eps;
                            const int* row = a.cell_start + a.g.G0 * (y0 + iy + a.g.G1 * (z0 + iz));
                            s[u] = row[cell_at(ux - hx, a.g.inv_h, a.g.G0)];
                            e[u] = row[cell_at(ux + hx, a.g.inv_h, a.g.G0) + 1];
                        }
                    }
                }
                // the query's runs as one list, walked by its lanes a point
                // each: run r holds the points up to run[r].y of the list, at
                // their position in it + run[r].x
                int nr = 0, np = 0;
#pragma unroll
                for (int u = 0; u < kNearRuns; ++u) {
                    nr += s[u] < e[u] ? 1 : 0;
                    np += e[u] - s[u];
                }
                int r = nr, all = np;
#pragma unroll
                for (int o = 1; o < G; o <<= 1) {
                    const int pr = __shfl_up_sync(FULL, r, o, G), pp = __shfl_up_sync(FULL, all, o, G);
                    if (sub >= o) {
                        r += pr;
                        all += pp;
                    }
                }
                r -= nr;
                int at = all - np;
                all = __shfl_sync(FULL, all, G - 1, G);
#pragma unroll
                for (int u = 0; u < kNearRuns; ++u)
                    if (s[u] < e[u]) {
                        run[r++] = make_int2(s[u] - at, at + e[u] - s[u]);
                        at += e[u] - s[u];
                    }
                __syncwarp();
                // the next point is loaded while one is tested
                int i = sub;
                float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
                const int2* in_run = run;
                int2 g = make_int2(0, 0);
                if (i < all) {
                    g = *in_run;
                    while (i >= g.y) g = *++in_run;
                    p = a.pts[i + g.x];
                }
                while (__any_sync(FULL, i < all)) {
                    const float4 c = p;
                    const bool have = i < all;
                    i += G;
                    if (i < all) {
                        while (i >= g.y) g = *++in_run;
                        p = a.pts[i + g.x];
                    }
                    const float d2 = sq3_rn(__fsub_rn(c.x, qx), __fsub_rn(c.y, qy), __fsub_rn(c.z, qz));
                    const bool in = have && d2 > lo2 && d2 <= hi2;
                    const unsigned m = __ballot_sync(FULL, in);
                    const int pos = found + __popc(m & before);
                    if (in && pos < kNearKeys)
                        key[pos] = __hiloint2double(__float_as_int(d2), __float_as_int(c.w));
                    found += __popc(m & mine);
                }
                __syncwarp();  // the list is read before the next batch's
            }
            if (search) {
                // k points within the radius, or everything was read
                search = found < k && hi2 < INFINITY;
                if (search) {
                    lo2 = hi2;
                    hi2 = fmaxf(hi2 * 2.25f, eps * eps);  // (a radius of 0 grows too)
                    if (hi2 > widest * widest) {
                        wait = true;
                        search = false;
                    }
                } else if (found > kNearKeys) {
                    // more than the buffer holds: the far search, from this radius
                    wait = true;
                    seed2 = fminf(seed2, hi2);
                }
            }
        }
        __syncwarp();
        if (wait) found = 0;
        // the keys in order: 2, 4 or twice 4 to a lane
        float kth = INFINITY;
        const int most = __reduce_max_sync(FULL, found);
        auto put = [&](auto& v) {
            constexpr int U = sizeof(v) / sizeof(double);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (sub * U + u < min(found, k)) {
                    a.out[qi * k + sub * U + u] = __double2loint(v[u]);
                    if (sub * U + u == k - 1) kth = __int_as_float(__double2hiint(v[u]));
                }
        };
        auto get = [&](auto& v, int b) {
            constexpr int U = sizeof(v) / sizeof(double);
#pragma unroll
            for (int u = 0; u < U; u += 2) {
                const double2 o = *reinterpret_cast<const double2*>(key + b + sub * U + u);
                v[u] = b + sub * U + u < found ? o.x : key_none();
                v[u + 1] = b + sub * U + u + 1 < found ? o.y : key_none();
            }
        };
        if (most <= 2 * G) {
            double v[2];
            get(v, 0);
            sort_keys<2>(v, sub);
            put(v);
        } else {
            double v[4];
            get(v, 0);
            sort_keys<4>(v, sub);
            if (most > 4 * G) {
                double o[4];
                get(o, 4 * G);
                sort_keys<4>(o, sub);
                // the smaller of each pair (i, 31 - i) are the smallest 32
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const double x = __shfl_xor_sync(FULL, o[3 - u], G - 1);
                    v[u] = x < v[u] ? x : v[u];
                }
                merge_keys<4, 4 * G>(v, sub);
            }
            put(v);
        }
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) kth = fminf(kth, __shfl_xor_sync(FULL, kth, o));
        lx = qx;
        ly = qy;
        lz = qz;
        lr = sqrt_up(kth);
        if (has && !wait)
            for (int i = found + sub; i < k; i += G) a.out[qi * k + i] = -1;
        const unsigned wm = __ballot_sync(FULL, wait && sub == 0);
        if (wm) {
            if (wait && sub == 0) {
                const int o = nfar + __popc(wm & ((1u << lane) - 1u));
                far[w].q[o] = make_float4(qx, qy, qz, __int_as_float((int)qi));
                far[w].bound[o] = seed2;
            }
            nfar += __popc(wm);
            __syncwarp();
            if (nfar >= 32) {
                far_groups(a, far[w], 32, lane);
                nfar -= 32;
                if (lane < nfar) {
                    far[w].q[lane] = far[w].q[32 + lane];
                    far[w].bound[lane] = far[w].bound[32 + lane];
                }
                __syncwarp();
            }
        }
        __syncwarp();  // the keys are read before the next queries'
    }
}

// --------------------------------------------------------- far queries --
// The queries that k_knn_near passed on, in groups of up to 32 near each
// other, a warp per group and a lane per query.  The warp walks the occupancy
// pyramid once for the group, depth first, the children nearest to the
// group's centre first: a node is opened when its (eps-widened) box lies
// within the k-th distance of some lane's query, tested when it is popped,
// with the bounds reached by then.  Below level 2 the points of the node's
// 4x4x4 cells (16 runs, a lane each) are gathered at once, those within the
// group's reach staged in shared memory, and every lane ranks them for its
// own query: the walk is a chain of dependent loads, and fewer, wider steps
// shorten it.  Groups stay narrow (far_groups) because a wide one opens the
// nodes of all its queries in turn, and the longest group is the launch's
// time.  A million queries around a 1 M-point torus, a quarter of them off the
// surface: 5.6 ms here and 1.1 ms in k_knn_near (125 ms with a warp per cell).
constexpr int kFarWarps = 4;
constexpr int kFarStack = 8 * KnnIndex::kMaxLevels;  // 7 siblings left per level, and the last 8
constexpr int kFarLeaf = 2;                          // the level whose nodes are read whole

// (level, child mask) and coordinates (10 bits each) of a node
__device__ __forceinline__ int2 far_entry(int i, int j, int k, int level, unsigned mask) {
    return make_int2(i | (j << 10) | (k << 20), level | (int)(mask << 8));
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

template <int KMAX>
__global__ void __launch_bounds__(kFarWarps * 32) k_knn_far(KnnArgs a, unsigned int* __restrict__ work) {
    __shared__ int2 stack[kFarWarps][kFarStack];
    __shared__ float4 stage[kFarWarps][32];
    if (a.gate_count && *a.gate_count <= a.gate_min) return;
    const unsigned FULL = 0xffffffffu;
    const unsigned long long NONE = ~0ull;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    const unsigned ng = a.far_count[1];
    const int k = a.k;
    const float h = a.g.h;
    const float eps = a.g.eps;
    for (;;) {
        unsigned g = 0;
        if (lane == 0) g = atomicAdd(work, 1u);
        g = __shfl_sync(FULL, g, 0);
        if (g >= ng) break;
        const int2 gr = a.far_group[g];
        const bool has = lane < gr.y;
        // lanes without a query stand on the group's first
        const unsigned at = (unsigned)gr.x + (has ? lane : 0);
        const long long qi = a.far_list[at];
        float qx, qy, qz;
        knn_load_query(a, qi, qx, qy, qz);
        const float U2 = a.far_bound[at];
        SortedK<KMAX> top;
        // (a lane without a query takes no key)
        top.init(k, !has ? 0ull
                         : U2 < INFINITY ? ((unsigned long long)__float_as_uint(U2) << 32) | 0xffffffffull : NONE);
        const float ux = __fsub_rn(qx, a.g.lo0), uy = __fsub_rn(qy, a.g.lo1), uz = __fsub_rn(qz, a.g.lo2);
        // the group's box, relative to the grid's too (rl, rh), and its centre
        float lo[3] = {qx, qy, qz}, hi[3] = {qx, qy, qz};
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                lo[d] = fminf(lo[d], __shfl_xor_sync(FULL, lo[d], o));
                hi[d] = fmaxf(hi[d], __shfl_xor_sync(FULL, hi[d], o));
            }
        const float rl[3] = {lo[0] - a.g.lo0, lo[1] - a.g.lo1, lo[2] - a.g.lo2};
        const float rh[3] = {hi[0] - a.g.lo0, hi[1] - a.g.lo1, hi[2] - a.g.lo2};
        const float mx = 0.5f * (rl[0] + rh[0]), my = 0.5f * (rl[1] + rh[1]), mz = 0.5f * (rl[2] + rh[2]);
        // (a grid of one cell has no pyramid: the cell is the root)
        if (lane == 0) stack[w][0] = far_entry(0, 0, 0, a.levels, a.levels > 0 ? a.occ[a.loff[a.levels]] : 0);
        int sp = 1;
        float kd2 = U2 * 1.00001f;  // the lane's bound, and the widest of the group
        float wide = warp_max(has ? kd2 : 0.f);
        while (sp > 0) {
            __syncwarp();  // the entries pushed last, and the stage's readers
            const int2 en = stack[w][--sp];
            const int lvl = en.y & 0xff;
            const int ci = en.x & 1023, cj = (en.x >> 10) & 1023, ck = en.x >> 20;
            {
                const float x0 = (float)(ci << lvl) * h - eps, x1 = (float)((ci + 1) << lvl) * h + eps;
                const float y0 = (float)(cj << lvl) * h - eps, y1 = (float)((cj + 1) << lvl) * h + eps;
                const float z0 = (float)(ck << lvl) * h - eps, z1 = (float)((ck + 1) << lvl) * h + eps;
                const float dx = fmaxf(0.f, fmaxf(x0 - ux, ux - x1));
                const float dy = fmaxf(0.f, fmaxf(y0 - uy, uy - y1));
                const float dz = fmaxf(0.f, fmaxf(z0 - uz, uz - z1));
                if (!__any_sync(FULL, has && dx * dx + dy * dy + dz * dz <= kd2)) continue;
            }
            if (lvl > kFarLeaf) {
                // push the occupied children within the group's reach, the
                // nearest to its centre last; a lane per child
                const int oc = lane & 7;
                const float half = (float)(1 << (lvl - 1));
                const int ni = 2 * ci + (oc & 1), nj = 2 * cj + ((oc >> 1) & 1), nk = 2 * ck + (oc >> 2);
                bool push = lane < 8 && ((en.y >> (8 + oc)) & 1);
                unsigned cm = 0;
                float away = -1.f;
                if (push) {
                    const int* D = a.ldim[lvl - 1];
                    cm = a.occ[a.loff[lvl - 1] + ni + (long long)D[0] * (nj + (long long)D[1] * nk)];
                    const float side = half * h;
                    const float x0 = (float)ni * side - eps, x1 = (float)(ni + 1) * side + eps;
                    const float y0 = (float)nj * side - eps, y1 = (float)(nj + 1) * side + eps;
                    const float z0 = (float)nk * side - eps, z1 = (float)(nk + 1) * side + eps;
                    const float dx = fmaxf(0.f, fmaxf(x0 - rh[0], rl[0] - x1));
                    const float dy = fmaxf(0.f, fmaxf(y0 - rh[1], rl[1] - y1));
                    const float dz = fmaxf(0.f, fmaxf(z0 - rh[2], rl[2] - z1));
                    push = dx * dx + dy * dy + dz * dz <= wide;
                    const float ax = 0.5f * (x0 + x1) - mx, ay = 0.5f * (y0 + y1) - my, az = 0.5f * (z0 + z1) - mz;
                    // (the limit takes a NaN too, of coordinates whose sums
                    // overflow: it has to order like the others)
                    if (push) away = fminf(ax * ax + ay * ay + az * az, FLT_MAX);
                }
                int place = sp;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const float o = __shfl_sync(FULL, away, u);
                    place += o > away || (o == away && u < lane) ? 1 : 0;
                }
                if (push) stack[w][place] = far_entry(ni, nj, nk, lvl - 1, cm);
                sp += __popc(__ballot_sync(FULL, push));
                continue;
            }
            // the rows of the node's cells, a lane each
            const int side = 1 << lvl;
            int s0 = 0, cnt = 0;
            if (lane < side * side) {
                const int x = ci << lvl, y = (cj << lvl) + (lane & (side - 1)), z = (ck << lvl) + (lane >> lvl);
                if (y < a.g.G1 && z < a.g.G2) {
                    const int row = a.g.G0 * (y + a.g.G1 * z);
                    s0 = a.cell_start[row + x];
                    cnt = a.cell_start[row + min(x + side, a.g.G0)] - s0;
                }
            }
            int incl = cnt;
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) {
                const int v = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += v;
            }
            const int excl = incl - cnt, tot = __shfl_sync(FULL, incl, 15);
            for (int b = 0; b < tot; b += 32) {
                const int t = b + lane;
                // the run that holds point t: the last one that starts at or before it
                int own = 0;
#pragma unroll
                for (int st = 8; st > 0; st >>= 1) {
                    const int e = __shfl_sync(FULL, excl, own + st);
                    if (e <= t) own += st;
                }
                const int ps = __shfl_sync(FULL, s0, own), po = __shfl_sync(FULL, excl, own);
                bool keep = false;
                float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
                if (t < tot) {
                    p = a.pts[ps + (t - po)];
                    const float dx = fmaxf(0.f, fmaxf(lo[0] - p.x, p.x - hi[0]));
                    const float dy = fmaxf(0.f, fmaxf(lo[1] - p.y, p.y - hi[1]));
                    const float dz = fmaxf(0.f, fmaxf(lo[2] - p.z, p.z - hi[2]));
                    keep = dx * dx + dy * dy + dz * dz <= wide;
                }
                const unsigned km = __ballot_sync(FULL, keep);
                if (keep) stage[w][__popc(km & below)] = p;
                __syncwarp();
                // four at a time: their distances do not wait for one another
                const int m = __popc(km);
                if (lane < 4 && m < 32) stage[w][m + lane < 32 ? m + lane : 31] = make_float4(INFINITY, 0.f, 0.f, 0.f);
                __syncwarp();
                for (int i = 0; i < m; i += 4) {
                    float d2[4];
                    int id[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const float4 c = stage[w][i + u];
                        d2[u] = sq3_rn(__fsub_rn(c.x, qx), __fsub_rn(c.y, qy), __fsub_rn(c.z, qz));
                        id[u] = __float_as_int(c.w);
                    }
                    if (fminf(fminf(d2[0], d2[1]), fminf(d2[2], d2[3])) <= kd2) {
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const unsigned long long v =
                                ((unsigned long long)__float_as_uint(d2[u]) << 32) | (unsigned)id[u];
                            if (i + u < m && v < top.last()) top.insert(v);
                        }
                        kd2 = top.last() == NONE ? INFINITY : top.last_d2() * 1.00001f;
                    }
                }
                __syncwarp();
            }
            wide = warp_max(has ? kd2 : 0.f);
        }
        if (has) top.store(a.out + qi * k, k);
    }
}

template <int KMAX>
static int knn_launch(const KnnArgs& a, long long nq, cudaStream_t s) {
    static int bps = 0;
    if (!bps) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_knn_thread<KMAX>, 128, 0);
        if (bps <= 0) bps = 1;
    }
    long long blocks = (nq + 127) / 128;
    long long cap = (long long)num_sms() * bps;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    k_knn_thread<KMAX><<<(unsigned)blocks, 128, 0, s>>>(a);
    DWG_CHECK_LAUNCH();
    return DWG_OK;
}

template <int KMAX>
static int near_launch(const KnnIndex& ix, const KnnArgs& a, long long nq, cudaStream_t s) {
    static int bps = 0;
    if (!bps) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_knn_near, kNearThreads, 0);
        if (bps <= 0) bps = 1;
    }
    // a block holds 16 queries at a time (2,000 queries on 1 M points that fill
    // a cube, k = 16: 1,407 us with a block per 128, 123 us; 2,000 of 20,000
    // surface points among themselves, k = 10: 73 and 38 us)
    constexpr int each = kNearThreads / kNearLanes;
    long long blocks = (nq + each - 1) / each;
    if (blocks > (long long)num_sms() * bps) blocks = (long long)num_sms() * bps;
    k_knn_near<<<(unsigned)blocks, kNearThreads, 0, s>>>(a, (unsigned int*)ix.q_misc.ptr);
    DWG_CHECK_LAUNCH();
    // the queries far from the points, or in sparse neighbourhoods
    static int fbps = 0;
    if (!fbps) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fbps, k_knn_far<KMAX>, kFarWarps * 32, 0);
        if (fbps <= 0) fbps = 1;
    }
    // (their number is the device's: a warp each if all are far and alone)
    blocks = (nq + kFarWarps - 1) / kFarWarps;
    if (blocks > (long long)num_sms() * fbps) blocks = (long long)num_sms() * fbps;
    k_knn_far<KMAX><<<(unsigned)blocks, kFarWarps * 32, 0, s>>>(a, (unsigned int*)ix.q_misc.ptr + 3);
    DWG_CHECK_LAUNCH();
    return DWG_OK;
}

// ------------------------------------------------------------- subsets --
__global__ void k_sub_count(long long ncell, const int* __restrict__ cs, const float4* __restrict__ pts,
                            const unsigned char* __restrict__ exclude, int* __restrict__ count, Gate gate) {
    if (gate.closed()) return;
    const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (c > ncell) return;
    int m = 0;
    if (c < ncell) {
        const int e = cs[c + 1];
        for (int t = cs[c]; t < e; ++t) m += exclude[__float_as_int(pts[t].w)] ? 0 : 1;
    }
    count[c] = m;  // count[ncell] = 0 closes the scan
}

__global__ void k_sub_fill(long long ncell, const int* __restrict__ cs, const float4* __restrict__ pts,
                           const unsigned char* __restrict__ exclude, const int* __restrict__ sub_start,
                           float4* __restrict__ sub_pts, Gate gate) {
    if (gate.closed()) return;
    const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (c >= ncell) return;
    int o = sub_start[c];
    const int e = cs[c + 1];
    for (int t = cs[c]; t < e; ++t) {
        const float4 p = pts[t];
        if (!exclude[__float_as_int(p.w)]) sub_pts[o++] = p;
    }
}

int knn_build_subset(const KnnIndex& full, const unsigned char* exclude, KnnIndex& sub, const int* gate_count,
                     int gate_min, cudaStream_t s) {
    const Gate gate{gate_count, gate_min};
    DWG_REQUIRE(exclude && full.n >= 1, "knn subset: bad arguments");
    const long long ncell = (long long)full.G[0] * full.G[1] * full.G[2];
    if (sub.n != full.n || sub.G[0] != full.G[0] || sub.G[1] != full.G[1] || sub.G[2] != full.G[2]) {
        sub.n = full.n;  // an upper bound; the kept count stays on the device
        for (int d = 0; d < 3; ++d) {
            sub.G[d] = full.G[d];
            sub.lo[d] = full.lo[d];
        }
        sub.h = full.h;
        sub.inv_h = full.inv_h;
        DWG_TRY(sub.cell_start.reserve(ncell + 1));
        DWG_TRY(sub.cell_fill.reserve(ncell + 1));
        DWG_TRY(sub.pts.reserve(full.n));
        DWG_TRY(sub.bbox.reserve(6));
        DWG_CHECK_CUDA(cudaMemcpyAsync(sub.bbox.ptr, full.bbox.ptr, sizeof(float) * 6, cudaMemcpyDeviceToDevice, s));
        DWG_TRY(pyramid_dims(sub));
        size_t bytes = 0;
        DWG_CHECK_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, bytes, sub.cell_fill.ptr, sub.cell_start.ptr,
                                                     (int)(ncell + 1), s));
        DWG_TRY(sub.scratch.reserve(bytes + 256));
    }
    k_sub_count<<<div_up(ncell + 1, 256), 256, 0, s>>>(ncell, full.cell_start.ptr, full.pts.ptr, exclude,
                                                       sub.cell_fill.ptr, gate);
    DWG_CHECK_LAUNCH();
    size_t bytes = sub.scratch.n;
    DWG_CHECK_CUDA(cub::DeviceScan::ExclusiveSum(sub.scratch.ptr, bytes, sub.cell_fill.ptr, sub.cell_start.ptr,
                                                 (int)(ncell + 1), s));
    k_sub_fill<<<div_up(ncell, 256), 256, 0, s>>>(ncell, full.cell_start.ptr, full.pts.ptr, exclude,
                                                  sub.cell_start.ptr, sub.pts.ptr, gate);
    DWG_CHECK_LAUNCH();
    DWG_TRY(pyramid_fill(sub, gate, s));
    return DWG_OK;
}

int knn_query(const KnnIndex& ix, const KnnQuery& q, int k, int* out, cudaStream_t s) {
    DWG_REQUIRE(k >= 1 && k <= 64, "knn: k must be in [1, 64] (got %d)", k);
    DWG_REQUIRE(out != nullptr, "knn: output is null");
    DWG_REQUIRE(q.q || (q.q_index && q.q_source), "knn: no queries");
    if (q.nq <= 0) return DWG_OK;
    KnnArgs a;
    a.g = grid_of(ix);
    a.pts = ix.pts.ptr;
    a.cell_start = ix.cell_start.ptr;
    a.q = q.q;
    a.q_index = q.q_index;
    a.q_source = q.q_source;
    a.nq = q.nq;
    a.nq_dev = q.nq_dev;
    a.nq_dev_i32 = q.nq_dev_i32;
    a.gate_count = q.gate_count;
    a.gate_min = q.gate_min;
    a.k = k;
    a.out = out;
    a.morton_shift = 0;
    a.occ = ix.occ.ptr;
    a.levels = ix.levels;
    for (int l = 0; l < KnnIndex::kMaxLevels; ++l) {
        a.loff[l] = ix.loff[l];
        for (int t = 0; t < 3; ++t) a.ldim[l][t] = ix.ldim[l][t];
    }
    a.order = nullptr;
    a.q_key = nullptr;
    a.q_hist = nullptr;
    a.far_list = nullptr;
    a.far_bound = nullptr;
    a.far_group = nullptr;
    a.far_count = nullptr;
    a.seed = q.seed;
    // few queries are done sooner than ordered (the far side of a ball of 20,000
    // points: 1 query 96 us with, 75 without; on its surface 42 and 20)
    if (!q.coherent && q.nq > 512) {
        // bucket the queries spatially (counting sort on device counts, no host sync)
        DWG_TRY(ix.q_key.reserve(q.nq));
        DWG_TRY(ix.q_order.reserve(q.nq));
        // buckets per axis: the grid's cells, at most 128 (32 for few queries,
        // whose buckets then hold several: clearing and scanning 2^21 counts
        // takes 10 us)
        const int gm = max(ix.G[0], max(ix.G[1], ix.G[2]));
        const int most = q.nq > (1 << 16) ? 7 : 5;
        int bits = 0;
        while ((1 << bits) < gm && bits < most) ++bits;
        a.morton_shift = 0;
        while ((gm - 1) >> (bits + a.morton_shift)) ++a.morton_shift;
        const int buckets = 1 << (3 * bits);
        DWG_TRY(ix.q_hist.reserve(buckets));
        DWG_TRY(ix.q_fill.reserve(buckets));
        a.q_key = ix.q_key.ptr;
        a.q_hist = ix.q_hist.ptr;
        DWG_CHECK_CUDA(cudaMemsetAsync(ix.q_hist.ptr, 0, sizeof(int) * buckets, s));
        long long blocks = (q.nq + 255) / 256;
        const long long cap = (long long)num_sms() * 8;
        if (blocks > cap) blocks = cap;
        k_knn_qkey<<<(unsigned)blocks, 256, 0, s>>>(a);
        DWG_CHECK_LAUNCH();
        size_t bytes = 0;
        int* hin = ix.q_hist.ptr;
        int* hout = ix.q_fill.ptr;
        DWG_CHECK_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, bytes, hin, hout, buckets, s));
        DWG_TRY(ix.q_scratch.reserve(bytes + 256));
        bytes = ix.q_scratch.n;
        DWG_CHECK_CUDA(cub::DeviceScan::ExclusiveSum(ix.q_scratch.ptr, bytes, hin, hout, buckets, s));
        k_knn_qscatter<<<(unsigned)blocks, 256, 0, s>>>(a, ix.q_fill.ptr, ix.q_order.ptr);
        DWG_CHECK_LAUNCH();
        a.order = ix.q_order.ptr;
    }
    if (k <= kKnnNearK) {
        DWG_TRY(ix.q_misc.reserve(4));
        DWG_TRY(ix.q_far.reserve(q.nq));
        DWG_TRY(ix.q_far_bound.reserve(q.nq));
        DWG_TRY(ix.q_far_group.reserve(q.nq));
        DWG_CHECK_CUDA(cudaMemsetAsync(ix.q_misc.ptr, 0, sizeof(int) * 4, s));
        a.far_list = ix.q_far.ptr;
        a.far_bound = ix.q_far_bound.ptr;
        a.far_group = ix.q_far_group.ptr;
        a.far_count = (unsigned int*)ix.q_misc.ptr + 1;
        // k = 15 (the triangle queries) keeps 15 slots per lane instead of 16
        // and k <= 10 (the zero repair) 10: shorter insertions, fewer registers
        if (k == 15) return near_launch<15>(ix, a, q.nq, s);
        if (k <= 10) return near_launch<10>(ix, a, q.nq, s);
        return near_launch<16>(ix, a, q.nq, s);
    }
    if (k <= 32) return knn_launch<32>(a, q.nq, s);
    return knn_launch<64>(a, q.nq, s);
}

}  // namespace dwg
