// gwn_eval.cu -- the winding-number sums and their gradients in FP64, one
// thread per query, with the Barnes-Hut decisions of the warp kernels
// (gwn.cu, which also has the FP32-term gradients): the yardstick a caller
// checks the FP32 sums against on the GPU, as the CPU oracle does on the
// host.  Terms and sums are in double, from the FP64 moments (cm_d, ec_d) and
// the points' float data; the terms' formulas are in gwn.cu (grad_term).
//
// Decisions: a child record is far when sq3_rn(CM_f - q) > its open
// threshold (exactly the warp kernels' test, so the same terms are taken);
// leaves are always summed point by point.  The traversal walks the level-
// order records with a per-level (first child, count, next) stack; point
// queries beyond a few hundred are taken in spatial order.
#include <algorithm>

#include "gwn.cuh"

namespace dwg {

constexpr double kFourPiD = 12.566370614359172953850573533118;

struct ThreadArgs {
    const float4* __restrict__ node_a;
    const float4* __restrict__ node_b;
    const int* __restrict__ level_nodes;
    const double* __restrict__ cm_d;
    const double* __restrict__ ec_d;
    const float4* __restrict__ pa;
    const float4* __restrict__ nr;
    float sigma, screen;
    int use_radii;
    const float* __restrict__ q;
    const int* order;  // point queries in spatial order (null: as they come)
    long long nq;
    int rx, ry, rz, zoff;
    float ox, oy, oz, h;
    int num_nodes, num_points;
    double* out_w;
    double* out_g;
    unsigned int* err;
};

// One term and its gradient.
template <bool SCREENED, bool GRAD>
__device__ __forceinline__ void add_term(double dx, double dy, double dz, double nx, double ny, double nz, double s,
                                         double sigma, double& w, double* g) {
    const double r2 = dx * dx + dy * dy + dz * dz;
    const double dot = dx * nx + dy * ny + dz * nz;
    if (SCREENED) {
        if (!(r2 > 1e-20)) return;  // |p - q| <= 1e-10 is skipped
        const double r = sqrt(r2);
        const double rho = r > s ? r : s;
        const double e = exp(sigma * rho);
        const double r3 = rho * rho * rho;
        const double den = e * (kFourPiD * r3) + 1e-7;
        const double up = fabs(sigma * rho + 1.0);
        const double G = up / den;
        w += G * dot;
        if (GRAD) {
            const double dden = e * (sigma * kFourPiD * r3 + 3.0 * kFourPiD * rho * rho);
            const double Gp = (sigma * den - up * dden) / (den * den);
            const double k = r > s ? -dot * Gp / r : 0.0;
            g[0] += k * dx - G * nx;
            g[1] += k * dy - G * ny;
            g[2] += k * dz - G * nz;
        }
    } else {
        if (r2 == 0.0) return;  // a zero distance is a term of value 0
        const double r = sqrt(r2);
        const double den = kFourPiD * r * r2 + 1e-8;
        w += dot / den;
        if (GRAD) {
            const double k = dot * 3.0 * kFourPiD * r / (den * den);
            g[0] += k * dx - nx / den;
            g[1] += k * dy - ny / den;
            g[2] += k * dz - nz / den;
        }
    }
}

template <bool SCREENED, bool GRAD>
__device__ __forceinline__ void leaf_points_thread(const ThreadArgs& a, int st, int cnt, float qx, float qy, float qz,
                                                   double& w, double* g) {
    const double sig = (double)a.sigma;
    for (int j = st; j < st + cnt; ++j) {
        const float4 p = a.pa[j];
        const float4 n = a.nr[j];
        const double s = (double)(a.use_radii ? n.w : a.screen);
        add_term<SCREENED, GRAD>((double)p.x - qx, (double)p.y - qy, (double)p.z - qz, (double)p.w * n.x,
                                 (double)p.w * n.y, (double)p.w * n.z, s, sig, w, g);
    }
}

template <bool SCREENED, bool GRAD>
__global__ void __launch_bounds__(128) k_gwn_thread(ThreadArgs a) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < a.nq; j += stride) {
        const long long i = a.order ? a.order[j] : j;
        float qx, qy, qz;
        if (a.q) {
            qx = a.q[i * 3];
            qy = a.q[i * 3 + 1];
            qz = a.q[i * 3 + 2];
        } else {  // the grid sample of the warp kernels: origin + index * spacing, rounded per operation
            const long long x = i % a.rx, t = i / a.rx;
            const long long y = t % a.ry, z = t / a.ry;
            qx = __fadd_rn(a.ox, __fmul_rn((float)x, a.h));
            qy = __fadd_rn(a.oy, __fmul_rn((float)y, a.h));
            qz = __fadd_rn(a.oz, __fmul_rn((float)(z + a.zoff), a.h));
        }
        double w = 0, g[3] = {0, 0, 0};
        int first[kMaxDepth + 2], count[kMaxDepth + 2], next[kMaxDepth + 2];
        int lev = 0;
        {
            const unsigned rm = (unsigned)__float_as_int(a.node_b[0].w);
            if (rm & kMetaLeafBit) {
                const int st = (int)(rm & kMetaIndex), cnt = __float_as_int(a.node_a[0].w);
                if (cnt >= 0 && st + cnt <= a.num_points)
                    leaf_points_thread<SCREENED, GRAD>(a, st, cnt, qx, qy, qz, w, g);
                else
                    atomicOr(a.err, 4u);
            } else {
                first[0] = (int)(rm & kMetaIndex);
                count[0] = (int)((rm >> 28) & 7u) + 1;
                next[0] = 0;
                lev = 1;
            }
        }
        while (lev > 0) {
            const int L = lev - 1;
            if (next[L] == count[L]) {
                --lev;
                continue;
            }
            const int c = first[L] + next[L]++;
            if (c < 0 || c >= a.num_nodes) {
                atomicOr(a.err, 2u);
                --lev;
                continue;
            }
            const float4 na = a.node_a[c], nb = a.node_b[c];
            const unsigned meta = (unsigned)__float_as_int(nb.w);
            if (meta & kMetaLeafBit) {
                const int st = (int)(meta & kMetaIndex), cnt = __float_as_int(na.w);
                if (cnt < 0 || st + cnt > a.num_points) {
                    atomicOr(a.err, 4u);
                    continue;
                }
                leaf_points_thread<SCREENED, GRAD>(a, st, cnt, qx, qy, qz, w, g);
                continue;
            }
            const float dxf = __fsub_rn(na.x, qx), dyf = __fsub_rn(na.y, qy), dzf = __fsub_rn(na.z, qz);
            if (sq3_rn(dxf, dyf, dzf) > na.w) {  // far: the node's dipole term
                const int v = a.level_nodes[c];
                const double* cm = a.cm_d + (size_t)v * 3;
                const double* ec = a.ec_d + (size_t)c * 3;
                add_term<SCREENED, GRAD>(cm[0] - (double)qx, cm[1] - (double)qy, cm[2] - (double)qz, ec[0], ec[1],
                                         ec[2], a.screen, a.sigma, w, g);
                continue;
            }
            // opened: its children become the next level
            const int fc = (int)(meta & kMetaIndex), nch = (int)((meta >> 28) & 7u) + 1;
            if (fc <= c || fc + nch > a.num_nodes || lev >= kMaxDepth + 2) {
                atomicOr(a.err, 2u);
                continue;
            }
            first[lev] = fc;
            count[lev] = nch;
            next[lev] = 0;
            ++lev;
        }
        if (a.out_w) a.out_w[i] = w;
        if (GRAD && a.out_g) {
            a.out_g[i * 3] = g[0];
            a.out_g[i * 3 + 1] = g[1];
            a.out_g[i * 3 + 2] = g[2];
        }
    }
}

template <bool SCREENED, bool GRAD>
static int launch_thread(const ThreadArgs& a, cudaStream_t s) {
    const long long blocks = std::min<long long>((a.nq + 127) / 128, (long long)num_sms() * 16);
    k_gwn_thread<SCREENED, GRAD><<<(unsigned)(blocks > 0 ? blocks : 1), 128, 0, s>>>(a);
    DWG_CHECK_LAUNCH();
    return DWG_OK;
}

int gwn_eval_fp64(const Octree& t, const GwnQuery& q, const dwg_gwn_params& p, double* out_w, double* out_g,
                  cudaStream_t s) {
    DWG_REQUIRE(t.M > 0, "gwn: octree is empty");
    DWG_REQUIRE(out_w || out_g, "gwn: no output");
    DWG_REQUIRE(p.order == 0, "gwn: gradients and FP64 sums take the order-0 far field");
    DWG_REQUIRE(p.beta >= 0.f, "gwn: beta must be >= 0");
    DWG_TRY(octree_set_beta(const_cast<Octree&>(t), p.beta, s));
    DWG_TRY(t.work.reserve(2));
    ThreadArgs a;
    a.node_a = t.node_a.ptr;
    a.node_b = t.node_b.ptr;
    a.level_nodes = t.level_nodes.ptr;
    a.cm_d = t.cm_d.ptr;
    a.ec_d = t.ec_d.ptr;
    a.pa = t.pa.ptr;
    a.nr = t.nr.ptr;
    a.sigma = p.sigma;
    a.screen = p.screen;
    a.use_radii = p.use_radii;
    a.num_nodes = t.M;
    a.num_points = t.n;
    a.out_w = out_w;
    a.out_g = out_g;
    a.err = t.work.ptr + 1;
    a.order = nullptr;
    QueryOrder sorted;
    if (q.q) {
        a.q = q.q;
        a.nq = q.nq;
        // (few queries are done sooner than sorted: 1 query 74 us with, 61
        // without; 1,000 around 100,000 points 306 with, 340 without)
        if (!q.coherent && q.nq > 256) DWG_TRY(query_order(sorted, q.q, q.nq, t.root, s, &a.order));
        a.rx = a.ry = a.rz = a.zoff = 0;
        a.ox = a.oy = a.oz = a.h = 0.f;
    } else {
        DWG_REQUIRE(q.res[0] > 0 && q.res[1] > 0 && q.res[2] > 0, "gwn: bad grid resolution");
        a.q = nullptr;
        a.nq = (long long)q.res[0] * q.res[1] * q.res[2];
        a.rx = q.res[0];
        a.ry = q.res[1];
        a.rz = q.res[2];
        a.zoff = q.zoff;
        a.ox = q.origin[0];
        a.oy = q.origin[1];
        a.oz = q.origin[2];
        a.h = q.spacing;
    }
    if (a.nq == 0) return DWG_OK;
    const bool grad = out_g != nullptr;
    if (p.screened) return grad ? launch_thread<true, true>(a, s) : launch_thread<true, false>(a, s);
    return grad ? launch_thread<false, true>(a, s) : launch_thread<false, false>(a, s);
}

}  // namespace dwg
