// mlp.cu -- learned normal initialiser: covariance features and a small MLP
// trained and evaluated with this file's own kernels.
//
// Features (12 per point, from its 16 nearest points, self included):
// eigenvalues of the neighbourhood covariance divided by their sum (3), the
// eigenvectors of the smallest and of the largest eigenvalue, each turned to
// point away from the centre of the cloud's bounding box (3 + 3), and the
// offset from the point to the centroid of a wider neighbourhood (the 64
// nearest of every 4th point, ~256 points) divided by that neighbourhood's
// RMS spread (3): over 16 points the offset that tells convex from concave
// is buried in the sampling noise.  The network maps them to a 3-vector
// that is normalised into an initial normal.
//
// The products run on the tensor cores with mma.sync m16n8k16 (BF16 inputs,
// FP32 accumulation); activations are rounded to BF16 where they feed a
// product and kept in FP32 elsewhere.  Training is mean cosine loss with Adam.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <random>
#include <vector>

#include "mlp.cuh"
#include "octree.cuh"

namespace dwg {

// ---------------------------------------------------------------- features --
// eigen-decomposition of a symmetric 3x3 matrix: eigenvalues by the closed
// trigonometric form of the characteristic cubic (O. K. Smith, CACM 1961),
// eigenvectors as the largest cross product of two rows of (A - lambda I)
__device__ void eig_vec(const double a[6], double lam, double out[3], const double fallback[3]) {
    // a = (xx, yy, zz, xy, xz, yz)
    const double r0[3] = {a[0] - lam, a[3], a[4]};
    const double r1[3] = {a[3], a[1] - lam, a[5]};
    const double r2[3] = {a[4], a[5], a[2] - lam};
    double c[3][3] = {{r0[1] * r1[2] - r0[2] * r1[1], r0[2] * r1[0] - r0[0] * r1[2], r0[0] * r1[1] - r0[1] * r1[0]},
                      {r0[1] * r2[2] - r0[2] * r2[1], r0[2] * r2[0] - r0[0] * r2[2], r0[0] * r2[1] - r0[1] * r2[0]},
                      {r1[1] * r2[2] - r1[2] * r2[1], r1[2] * r2[0] - r1[0] * r2[2], r1[0] * r2[1] - r1[1] * r2[0]}};
    int best = 0;
    double bn = -1;
    for (int i = 0; i < 3; ++i) {
        double nn = c[i][0] * c[i][0] + c[i][1] * c[i][1] + c[i][2] * c[i][2];
        if (nn > bn) {
            bn = nn;
            best = i;
        }
    }
    if (bn < 1e-60) {
        for (int d = 0; d < 3; ++d) out[d] = fallback[d];
        return;
    }
    const double inv = 1.0 / sqrt(bn);
    for (int d = 0; d < 3; ++d) out[d] = c[best][d] * inv;
}

__global__ void k_features(const float* __restrict__ P, int n, const int* __restrict__ nb, int k,
                           const float* __restrict__ S, const int* __restrict__ nbw, int kw,
                           const float* __restrict__ bb, float* __restrict__ F) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double px = P[(size_t)i * 3], py = P[(size_t)i * 3 + 1], pz = P[(size_t)i * 3 + 2];
    double cx = 0, cy = 0, cz = 0;
    int cnt = 0;
    for (int j = 0; j < k; ++j) {
        const int q = nb[(size_t)i * k + j];
        if (q < 0) continue;
        cx += P[(size_t)q * 3];
        cy += P[(size_t)q * 3 + 1];
        cz += P[(size_t)q * 3 + 2];
        ++cnt;
    }
    cnt = cnt > 0 ? cnt : 1;
    cx /= cnt;
    cy /= cnt;
    cz /= cnt;
    double a[6] = {0, 0, 0, 0, 0, 0};
    for (int j = 0; j < k; ++j) {
        const int q = nb[(size_t)i * k + j];
        if (q < 0) continue;
        const double dx = P[(size_t)q * 3] - cx, dy = P[(size_t)q * 3 + 1] - cy, dz = P[(size_t)q * 3 + 2] - cz;
        a[0] += dx * dx;
        a[1] += dy * dy;
        a[2] += dz * dz;
        a[3] += dx * dy;
        a[4] += dx * dz;
        a[5] += dy * dz;
    }
    for (int t = 0; t < 6; ++t) a[t] /= cnt;
    // eigenvalues
    const double m = (a[0] + a[1] + a[2]) / 3.0;
    const double k0 = a[0] - m, k1 = a[1] - m, k2 = a[2] - m;
    const double p2 = (k0 * k0 + k1 * k1 + k2 * k2 + 2.0 * (a[3] * a[3] + a[4] * a[4] + a[5] * a[5])) / 6.0;
    double l1, l2, l3;
    if (p2 < 1e-60) {
        l1 = l2 = l3 = m;
    } else {
        const double pp = sqrt(p2);
        const double det = k0 * (k1 * k2 - a[5] * a[5]) - a[3] * (a[3] * k2 - a[5] * a[4]) + a[4] * (a[3] * a[5] - k1 * a[4]);
        double r = det / (2.0 * pp * pp * pp);
        r = r < -1.0 ? -1.0 : (r > 1.0 ? 1.0 : r);
        const double phi = acos(r) / 3.0;
        l1 = m + 2.0 * pp * cos(phi);
        l3 = m + 2.0 * pp * cos(phi + 2.0943951023931957);
        l2 = 3.0 * m - l1 - l3;
    }
    // direction from the bounding-box centre (orients the eigenvectors)
    const double gx = px - 0.5 * ((double)bb[0] + bb[3]), gy = py - 0.5 * ((double)bb[1] + bb[4]),
                 gz = pz - 0.5 * ((double)bb[2] + bb[5]);
    double gn = sqrt(gx * gx + gy * gy + gz * gz);
    const double g[3] = {gn > 0 ? gx / gn : 0.0, gn > 0 ? gy / gn : 0.0, gn > 0 ? gz / gn : 1.0};
    const double ex[3] = {1, 0, 0};
    double v3[3], v1[3];
    eig_vec(a, l3, v3, g);
    eig_vec(a, l1, v1, ex);
    if (v3[0] * g[0] + v3[1] * g[1] + v3[2] * g[2] < 0)
        for (int d = 0; d < 3; ++d) v3[d] = -v3[d];
    if (v1[0] * g[0] + v1[1] * g[1] + v1[2] * g[2] < 0)
        for (int d = 0; d < 3; ++d) v1[d] = -v1[d];
    const double sum = fmax(l1 + l2 + l3, 1e-30);
    float* f = F + (size_t)i * kMlpIn;
    f[0] = (float)(fmax(l1, 0.0) / sum);
    f[1] = (float)(fmax(l2, 0.0) / sum);
    f[2] = (float)(fmax(l3, 0.0) / sum);
    for (int d = 0; d < 3; ++d) f[3 + d] = (float)v3[d];
    for (int d = 0; d < 3; ++d) f[6 + d] = (float)v1[d];
    // centroid offset over the wide neighbourhood (kw nearest points of the
    // subsample S), over its RMS spread
    double wx = 0, wy = 0, wz = 0;
    int wc = 0;
    for (int j = 0; j < kw; ++j) {
        const int q = nbw[(size_t)i * kw + j];
        if (q < 0) continue;
        wx += S[(size_t)q * 3];
        wy += S[(size_t)q * 3 + 1];
        wz += S[(size_t)q * 3 + 2];
        ++wc;
    }
    wc = wc > 0 ? wc : 1;
    wx /= wc;
    wy /= wc;
    wz /= wc;
    double ws = 0;
    for (int j = 0; j < kw; ++j) {
        const int q = nbw[(size_t)i * kw + j];
        if (q < 0) continue;
        const double dx = S[(size_t)q * 3] - wx, dy = S[(size_t)q * 3 + 1] - wy, dz = S[(size_t)q * 3 + 2] - wz;
        ws += dx * dx + dy * dy + dz * dz;
    }
    const double wsc = 1.0 / sqrt(fmax(ws / wc, 1e-30));
    f[9] = (float)((wx - px) * wsc);
    f[10] = (float)((wy - py) * wsc);
    f[11] = (float)((wz - pz) * wsc);
}

__global__ void k_subsample(const float* __restrict__ P, int n, int stride, float* __restrict__ S) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int m = (n + stride - 1) / stride;
    if (j >= m) return;
    for (int d = 0; d < 3; ++d) S[(size_t)j * 3 + d] = P[(size_t)j * stride * 3 + d];
}

int mlp_features(const KnnIndex& ix, const float* P, int n, float* F, cudaStream_t s) {
    DWG_REQUIRE(P && F && n >= 1, "mlp_features: bad arguments");
    DWG_REQUIRE(ix.n >= 1, "mlp_features: empty index");
    const int k = ix.n < kMlpFeatureK ? ix.n : kMlpFeatureK;
    DevBuf<int> nb, nbw;
    DWG_TRY(nb.reserve((size_t)n * k));
    KnnQuery q;
    q.q = P;
    q.nq = n;
    DWG_TRY(knn_query(ix, q, k, nb.ptr, s));
    // wide neighbourhood: the kMlpWideK nearest of every kMlpWideStride-th point
    const int m = (n + kMlpWideStride - 1) / kMlpWideStride;
    DevBuf<float> S;
    DWG_TRY(S.reserve((size_t)m * 3));
    k_subsample<<<div_up(m, 256), 256, 0, s>>>(P, n, kMlpWideStride, S.ptr);
    DWG_CHECK_LAUNCH();
    KnnIndex iw;
    DWG_TRY(knn_build(iw, S.ptr, m, s));
    const int kw = m < kMlpWideK ? m : kMlpWideK;
    DWG_TRY(nbw.reserve((size_t)n * kw));
    DWG_TRY(knn_query(iw, q, kw, nbw.ptr, s));
    k_features<<<div_up(n, 128), 128, 0, s>>>(P, n, nb.ptr, k, S.ptr, nbw.ptr, kw, ix.bbox.ptr, F);
    DWG_CHECK_LAUNCH();
    DWG_CHECK_CUDA(cudaStreamSynchronize(s));
    return DWG_OK;
}

// ---------------------------------------------------------- the network --
// Two kernels.  k_mlp_rows takes a warp 16 rows through the whole network:
// the weights sit in shared memory, a layer's product stays in registers, and
// its activations are the next product's left operand as they stand (the
// accumulator layout of mma.m16n8k16 is that of its A operand), so a forward
// pass touches global memory for the features and the outputs only.  Training
// runs the backward products the same way; what the weight gradients need
// (activations and dZ in BF16) and gelu' (FP32, read back by the thread that
// wrote it) go to global memory in the fragments' own order, 512 bytes per
// warp and store.  k_mlp_weights forms H^T dZ per chunk of rows in shared
// memory.  Its partial sums, and the bias sums of k_mlp_rows, are added in a
// fixed order.  65,536 rows, forward and backward: 147 us and 78 us (1,030 us
// with a GEMM, an elementwise and a column-sum kernel per layer, each through
// global memory with 16-bit loads).  Two blocks of 8 warps share an SM, all that
// 128 registers a thread leave: the first kernel waits for its serial chain of
// products, error functions and exponentials, with 4 warps a scheduler to hide it.
__device__ __forceinline__ unsigned pack2(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const unsigned*>(&v);
}

__device__ __forceinline__ void mma16816(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// four 8x8 tiles; lane l gives the row l & 7 of tile l >> 3
template <bool TRANS>
__device__ __forceinline__ void ldmatrix4(unsigned (&r)[4], const __nv_bfloat16* row) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(row);
    if (TRANS)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(a)
                     : "memory");
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(a)
                     : "memory");
}

// gelu (erf form) and its derivative
__device__ __forceinline__ float gelu_both(float x, float& grad) {
    const float u = 1.0f + erff(x * 0.7071067811865476f);
    grad = 0.5f * u + x * 0.3989422804014327f * expf(-0.5f * x * x);
    return 0.5f * x * u;
}

constexpr int kRowWarps = 8;
constexpr int kWPad = kMlpHidden + 8;  // row stride of the weights in shared memory: conflict-free ldmatrix
constexpr int kW4Pad = 16;             // row stride of the last layer's
constexpr int kNT = kMlpHidden / 8;    // column tiles of a hidden layer
// offsets (BF16) of the layers' weights in shared memory
constexpr int kS1 = 0, kS2 = kS1 + kMlpInPad * kWPad, kS3 = kS2 + kMlpHidden * kWPad, kS4 = kS3 + kMlpHidden * kWPad;
constexpr int kSBias = kS4 + kMlpHidden * kW4Pad;  // then the biases (FP32): 3 x 128, 8
constexpr int kBias = 3 * kMlpHidden + kMlpOutPad;
constexpr int kRowSmem = kSBias * 2 + kBias * 4 + kRowWarps * kBias * 4;  // and the warps' bias sums

struct RowArgs {
    const float* F;
    const float* T;
    long long rows;
    const __nv_bfloat16* w[kMlpLayers];
    const float* b[kMlpLayers];
    float* out;            // forward: raw outputs, 3 per row
    float4* gp[3];         // training: gelu' of the hidden layers
    uint4* x;              // the inputs, hidden activations, dZ of the hidden layers and of the outputs
    uint2* h[3];
    uint2* dz[3];
    unsigned* dy;
    float* bias_part;      // per block: the bias gradients
    double* loss_part;     // per block
};

// acc[16 x N] += A[16 x 16 K] op(W): the weights of a layer as they are
// (TRANS false: B[k][n] = W[n][k], the backward products)
template <int K, int N, bool FORWARD>
__device__ __forceinline__ void row_product(float (&acc)[N][4], const unsigned (&A)[K][4], const __nv_bfloat16* w,
                                            int stride, int lane) {
    const int t = lane >> 3, r = lane & 7;
#pragma unroll
    for (int kk = 0; kk < K; ++kk)
#pragma unroll
        for (int n = 0; n < N; n += 2) {
            unsigned b[4];
            if (FORWARD) ldmatrix4<true>(b, w + (kk * 16 + (t & 1) * 8 + r) * stride + n * 8 + (t >> 1) * 8);
            else ldmatrix4<false>(b, w + (n * 8 + (t >> 1) * 8 + r) * stride + kk * 16 + (t & 1) * 8);
            mma16816(acc[n], A[kk], b[0], b[1]);
            mma16816(acc[n + 1], A[kk], b[2], b[3]);
        }
}

template <bool TRAIN>
__global__ void __launch_bounds__(kRowWarps * 32, 2) k_mlp_rows(RowArgs a) {
    extern __shared__ __align__(16) unsigned char row_smem[];
    __nv_bfloat16* const ws = reinterpret_cast<__nv_bfloat16*>(row_smem);
    float* const bs = reinterpret_cast<float*>(row_smem + kSBias * 2);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    float* const bsum = bs + kBias + w * kBias;
    // the weights, 8 at a time (the last layer's rows end in zeros)
    auto stage = [&](__nv_bfloat16* dst, int stride, const __nv_bfloat16* src, int chunks, int per_row) {
#pragma unroll 4
        for (int i = tid; i < chunks; i += kRowWarps * 32)
            *reinterpret_cast<uint4*>(dst + i / per_row * stride + i % per_row * 8) =
                reinterpret_cast<const uint4*>(src)[i];
    };
    constexpr int kRow = kMlpHidden / 8;
    stage(ws + kS1, kWPad, a.w[0], kMlpInPad * kRow, kRow);
    stage(ws + kS2, kWPad, a.w[1], kMlpHidden * kRow, kRow);
    stage(ws + kS3, kWPad, a.w[2], kMlpHidden * kRow, kRow);
    stage(ws + kS4, kW4Pad, a.w[3], kMlpHidden, 1);
    for (int i = tid; i < kMlpHidden; i += kRowWarps * 32) {
        *reinterpret_cast<uint4*>(ws + kS4 + i * kW4Pad + 8) = make_uint4(0u, 0u, 0u, 0u);
        for (int l = 0; l < 3; ++l) bs[l * kMlpHidden + i] = a.b[l][i];
        if (i < kMlpOutPad) bs[3 * kMlpHidden + i] = a.b[3][i];
    }
    for (int i = lane; i < kBias; i += 32) bsum[i] = 0.f;
    __syncthreads();
    double loss = 0.0;
    const long long tiles = (a.rows + 15) / 16, warps = (long long)gridDim.x * kRowWarps;
    for (long long tile = (long long)blockIdx.x * kRowWarps + w; tile < tiles; tile += warps) {
        const long long row[2] = {tile * 16 + g, tile * 16 + g + 8};
        const bool in[2] = {row[0] < a.rows, row[1] < a.rows};
        float acc[kNT][4];
        unsigned A[kMlpHidden / 16][4];
        {
            unsigned X[1][4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {  // rows g, g + 8; columns 2t, then 2t + 8
                const int c = 2 * t + (q >> 1) * 8;
                float2 v = make_float2(0.f, 0.f);
                if (in[q & 1] && c < kMlpIn) {
                    const float* f = a.F + row[q & 1] * kMlpIn + c;
                    v = make_float2(f[0], f[1]);
                }
                X[0][q] = pack2(v.x, v.y);
            }
            if (TRAIN) a.x[tile * 32 + lane] = make_uint4(X[0][0], X[0][1], X[0][2], X[0][3]);
#pragma unroll
            for (int n = 0; n < kNT; ++n)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[n][q] = 0.f;
            row_product<1, kNT, true>(acc, X, ws + kS1, kWPad, lane);
        }
#pragma unroll
        for (int l = 0; l < 3; ++l) {
            // activations: FP32 pre-activations, BF16 into the next product
#pragma unroll
            for (int n = 0; n < kNT; ++n) {
                const float2 b = *reinterpret_cast<const float2*>(bs + l * kMlpHidden + n * 8 + 2 * t);
                float4 d;
                const float h0 = gelu_both(acc[n][0] + b.x, d.x), h1 = gelu_both(acc[n][1] + b.y, d.y);
                const float h2 = gelu_both(acc[n][2] + b.x, d.z), h3 = gelu_both(acc[n][3] + b.y, d.w);
                const unsigned lo = pack2(h0, h1), hi = pack2(h2, h3);
                A[n / 2][(n & 1) * 2] = lo;
                A[n / 2][(n & 1) * 2 + 1] = hi;
                if (TRAIN) {
                    const long long o = (tile * kNT + n) * 32 + lane;
                    a.gp[l][o] = d;
                    a.h[l][o] = make_uint2(lo, hi);
                }
            }
            if (l == 2) break;
#pragma unroll
            for (int n = 0; n < kNT; ++n)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[n][q] = 0.f;
            row_product<kMlpHidden / 16, kNT, true>(acc, A, ws + (l == 0 ? kS2 : kS3), kWPad, lane);
        }
        // outputs: columns 2t, 2t + 1 of 8 (the second column tile is padding)
        float y[2][4] = {};
        row_product<kMlpHidden / 16, 2, true>(y, A, ws + kS4, kW4Pad, lane);
        const float* b4 = bs + 3 * kMlpHidden + 2 * t;
#pragma unroll
        for (int q = 0; q < 4; ++q) y[0][q] += b4[q & 1];
        if (!TRAIN) {
#pragma unroll
            for (int s = 0; s < 2; ++s)
                if (in[s]) {
                    if (t < 2) a.out[row[s] * 3 + 2 * t] = y[0][2 * s];
                    if (t == 0) a.out[row[s] * 3 + 1] = y[0][2 * s + 1];
                }
            continue;
        }
        // cosine loss and dY (BF16) of the two rows
        unsigned D[1][4] = {};
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const float y0 = __shfl_sync(0xffffffffu, y[0][2 * s], lane & ~3),
                        y1 = __shfl_sync(0xffffffffu, y[0][2 * s + 1], lane & ~3),
                        y2 = __shfl_sync(0xffffffffu, y[0][2 * s], (lane & ~3) + 1);
            float d[3] = {0.f, 0.f, 0.f};
            if (in[s]) {
                const float* tr = a.T + row[s] * 3;
                const float nn = sqrtf(y0 * y0 + y1 * y1 + y2 * y2) + 1e-12f;
                const float yh[3] = {y0 / nn, y1 / nn, y2 / nn};
                const float c = yh[0] * tr[0] + yh[1] * tr[1] + yh[2] * tr[2];
                if (t == 0) loss += (double)(1.0f - c);
#pragma unroll
                for (int q = 0; q < 3; ++q) d[q] = -(tr[q] - c * yh[q]) / nn / (float)a.rows;
            }
            D[0][s] = t == 0 ? pack2(d[0], d[1]) : t == 1 ? pack2(d[2], 0.f) : 0u;
        }
        a.dy[(tile * 32 + lane) * 2] = D[0][0];
        a.dy[(tile * 32 + lane) * 2 + 1] = D[0][1];
        // the output bias sums the BF16 dY
        {
            float s0 = __uint_as_float(D[0][0] << 16) + __uint_as_float(D[0][1] << 16);
            float s1 = __uint_as_float(D[0][0] & 0xffff0000u) + __uint_as_float(D[0][1] & 0xffff0000u);
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) {
                s0 += __shfl_xor_sync(0xffffffffu, s0, o);
                s1 += __shfl_xor_sync(0xffffffffu, s1, o);
            }
            if (g == 0) {
                bsum[3 * kMlpHidden + 2 * t] += s0;
                bsum[3 * kMlpHidden + 2 * t + 1] += s1;
            }
        }
#pragma unroll
        for (int l = 2; l >= 0; --l) {
            // dH of layer l's activations, then dZ = dH gelu'
#pragma unroll
            for (int n = 0; n < kNT; ++n)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[n][q] = 0.f;
            if (l == 2) row_product<1, kNT, false>(acc, D, ws + kS4, kW4Pad, lane);
            else row_product<kMlpHidden / 16, kNT, false>(acc, A, ws + (l == 1 ? kS3 : kS2), kWPad, lane);
            // (gelu' is loaded four column tiles ahead: it comes from L2)
            float4 ahead[4];
#pragma unroll
            for (int n = 0; n < 4; ++n) ahead[n] = a.gp[l][(tile * kNT + n) * 32 + lane];
#pragma unroll
            for (int n = 0; n < kNT; ++n) {
                const long long o = (tile * kNT + n) * 32 + lane;
                const float4 d = ahead[n & 3];
                if (n + 4 < kNT) ahead[n & 3] = a.gp[l][o + 4 * 32];
                acc[n][0] *= d.x;
                acc[n][1] *= d.y;
                acc[n][2] *= d.z;
                acc[n][3] *= d.w;
                const unsigned lo = pack2(acc[n][0], acc[n][1]), hi = pack2(acc[n][2], acc[n][3]);
                A[n / 2][(n & 1) * 2] = lo;
                A[n / 2][(n & 1) * 2 + 1] = hi;
                a.dz[l][o] = make_uint2(lo, hi);
                // the bias gradient sums the FP32 dZ over the 16 rows
                float s0 = acc[n][0] + acc[n][2], s1 = acc[n][1] + acc[n][3];
#pragma unroll
                for (int x = 4; x < 32; x <<= 1) {
                    s0 += __shfl_xor_sync(0xffffffffu, s0, x);
                    s1 += __shfl_xor_sync(0xffffffffu, s1, x);
                }
                if (g == 0) {
                    bsum[l * kMlpHidden + n * 8 + 2 * t] += s0;
                    bsum[l * kMlpHidden + n * 8 + 2 * t + 1] += s1;
                }
            }
        }
    }
    if (TRAIN) {
        // the block's warps in order
        for (int o = 16; o > 0; o >>= 1) loss += __shfl_down_sync(0xffffffffu, loss, o);
        __shared__ double losses[kRowWarps];
        if (lane == 0) losses[w] = loss;
        __syncthreads();
        for (int i = tid; i < kBias; i += kRowWarps * 32) {
            float s = 0.f;
            for (int k = 0; k < kRowWarps; ++k) s += bs[kBias + k * kBias + i];
            a.bias_part[(size_t)blockIdx.x * kBias + i] = s;
        }
        if (tid == 0) {
            double s = 0.0;
            for (int k = 0; k < kRowWarps; ++k) s += losses[k];
            a.loss_part[blockIdx.x] = s;
        }
    }
}

// Weight gradients of a chunk of row tiles (128 rows at a time): blockIdx.y 0
// and 1 the two hidden products (a warp 16 of the 128 rows of dW), 2 the first
// and the last layer's.
constexpr int kWRows = 128;
constexpr int kWSmem = (2 * kWRows * kWPad + kWRows * 24 + kWRows * 24) * 2;
struct WeightArgs {
    long long tiles;  // of 16 rows
    const uint4* x;
    const uint2* h[3];
    const uint2* dz[3];
    const unsigned* dy;
    float* part;  // per chunk: dW of the four layers (16 x 128, 128 x 128 twice, 128 x 8)
};
// places of the layers' dW in a part, and its size
constexpr int kPart1 = kMlpInPad * kMlpHidden, kPart2 = kPart1 + kMlpHidden * kMlpHidden,
              kPart3 = kPart2 + kMlpHidden * kMlpHidden, kParts = kPart3 + kMlpHidden * kMlpOutPad;

__global__ void __launch_bounds__(kRowWarps * 32) k_mlp_weights(WeightArgs a) {
    extern __shared__ __align__(16) unsigned char w_smem[];
    __nv_bfloat16* const hs = reinterpret_cast<__nv_bfloat16*>(w_smem);  // [row][column]
    __nv_bfloat16* const ds = hs + kWRows * kWPad;
    __nv_bfloat16* const xs = ds + kWRows * kWPad;  // stride 24: the inputs, and dY
    __nv_bfloat16* const ys = xs + kWRows * 24;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3, lt = lane >> 3, lr = lane & 7;
    const int kind = blockIdx.y;
    const uint2* H = kind == 2 ? a.h[2] : a.h[kind];
    const uint2* Z = kind == 2 ? a.dz[0] : a.dz[kind + 1];
    float acc[kNT][4];
#pragma unroll
    for (int n = 0; n < kNT; ++n)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[n][q] = 0.f;
    const long long sets = (a.tiles + 7) / 8;
    for (long long set = blockIdx.x; set < sets; set += gridDim.x) {
        // the warp's 16 rows, fragments back to rows
        const long long tile = set * 8 + w;
        const bool in = tile < a.tiles;
        __syncthreads();
#pragma unroll 4
        for (int n = 0; n < kNT; ++n) {
            const long long o = (tile * kNT + n) * 32 + lane;
            const uint2 h = in ? H[o] : make_uint2(0u, 0u), z = in ? Z[o] : make_uint2(0u, 0u);
            const int c = (w * 16 + g) * kWPad + n * 8 + 2 * t;
            *reinterpret_cast<unsigned*>(hs + c) = h.x;
            *reinterpret_cast<unsigned*>(hs + c + 8 * kWPad) = h.y;
            *reinterpret_cast<unsigned*>(ds + c) = z.x;
            *reinterpret_cast<unsigned*>(ds + c + 8 * kWPad) = z.y;
        }
        if (kind == 2) {
            const uint4 x = in ? a.x[tile * 32 + lane] : make_uint4(0u, 0u, 0u, 0u);
            const int c = (w * 16 + g) * 24 + 2 * t;
            *reinterpret_cast<unsigned*>(xs + c) = x.x;
            *reinterpret_cast<unsigned*>(xs + c + 8 * 24) = x.y;
            *reinterpret_cast<unsigned*>(xs + c + 8) = x.z;
            *reinterpret_cast<unsigned*>(xs + c + 8 * 24 + 8) = x.w;
            *reinterpret_cast<unsigned*>(ys + c) = in ? a.dy[(tile * 32 + lane) * 2] : 0u;
            *reinterpret_cast<unsigned*>(ys + c + 8 * 24) = in ? a.dy[(tile * 32 + lane) * 2 + 1] : 0u;
            *reinterpret_cast<unsigned*>(ys + c + 8) = 0u;
            *reinterpret_cast<unsigned*>(ys + c + 8 * 24 + 8) = 0u;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kWRows / 16; ++kk) {
            unsigned A[4], b[4];
            const int ra = kk * 16 + (lt >> 1) * 8 + lr, rb = kk * 16 + (lt & 1) * 8 + lr;
            if (kind < 2) {
                // rows 16 w .. of H^T, all columns of dZ
                ldmatrix4<true>(A, hs + ra * kWPad + w * 16 + (lt & 1) * 8);
#pragma unroll
                for (int n = 0; n < kNT; n += 2) {
                    ldmatrix4<true>(b, ds + rb * kWPad + n * 8 + (lt >> 1) * 8);
                    mma16816(acc[n], A, b[0], b[1]);
                    mma16816(acc[n + 1], A, b[2], b[3]);
                }
            } else {
                // X^T dZ1: the warp's 16 columns; H3^T dY: its 16 rows
                ldmatrix4<true>(A, xs + ra * 24 + (lt & 1) * 8);
                ldmatrix4<true>(b, ds + rb * kWPad + w * 16 + (lt >> 1) * 8);
                mma16816(acc[0], A, b[0], b[1]);
                mma16816(acc[1], A, b[2], b[3]);
                ldmatrix4<true>(A, hs + ra * kWPad + w * 16 + (lt & 1) * 8);
                ldmatrix4<true>(b, ys + rb * 24 + (lt >> 1) * 8);
                mma16816(acc[2], A, b[0], b[1]);
            }
        }
    }
    float* const part = a.part + (size_t)blockIdx.x * kParts;
    auto put = [&](float* o, int ld, int r, int c, const float (&v)[4]) {
        *reinterpret_cast<float2*>(o + (size_t)r * ld + c) = make_float2(v[0], v[1]);
        *reinterpret_cast<float2*>(o + (size_t)(r + 8) * ld + c) = make_float2(v[2], v[3]);
    };
    if (kind < 2) {
#pragma unroll
        for (int n = 0; n < kNT; ++n) put(part + (kind == 0 ? kPart1 : kPart2), kMlpHidden, w * 16 + g, n * 8 + 2 * t, acc[n]);
    } else {
        put(part, kMlpHidden, g, w * 16 + 2 * t, acc[0]);
        put(part, kMlpHidden, g, w * 16 + 8 + 2 * t, acc[1]);
        put(part + kPart3, kMlpOutPad, w * 16 + g, 2 * t, acc[2]);
    }
}

// the gradients from the chunks' and the blocks' parts, in a fixed order, and
// the loss
struct GradOut {
    float* gw[kMlpLayers];
    float* gb[kMlpLayers];
};
__global__ void __launch_bounds__(128) k_mlp_reduce(const float* __restrict__ part, int chunks,
                                                    const float* __restrict__ bias_part,
                                                    const double* __restrict__ loss_part, int blocks, long long rows,
                                                    GradOut o, float* __restrict__ loss) {
    static_assert(kParts % 128 == 0, "whole blocks of weights, then a warp per bias");
    const int i = blockIdx.x * 128 + threadIdx.x;
    if (i < kParts) {
        float s = 0.f;
#pragma unroll 8
        for (int c = 0; c < chunks; ++c) s += part[(size_t)c * kParts + i];
        const int l = i < kPart1 ? 0 : i < kPart2 ? 1 : i < kPart3 ? 2 : 3;
        o.gw[l][i - (l == 0 ? 0 : l == 1 ? kPart1 : l == 2 ? kPart2 : kPart3)] = s;
        return;
    }
    const int k = (i - kParts) >> 5, lane = threadIdx.x & 31;
    if (k < kBias) {
        float s = 0.f;
        for (int b = lane; b < blocks; b += 32) s += bias_part[(size_t)b * kBias + k];
        for (int d = 16; d > 0; d >>= 1) s += __shfl_down_sync(0xffffffffu, s, d);
        if (lane == 0) o.gb[k / kMlpHidden][k % kMlpHidden] = s;
    } else if (k == kBias) {
        double s = 0.0;
        for (int b = lane; b < blocks; b += 32) s += loss_part[b];
        for (int d = 16; d > 0; d >>= 1) s += __shfl_down_sync(0xffffffffu, s, d);
        if (lane == 0) *loss = (float)(s / (double)rows);
    }
}

__global__ void k_to_bf16(const float* __restrict__ x, long long n, __nv_bfloat16* __restrict__ y) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < n) y[i] = __float2bfloat16_rn(x[i]);
}

__global__ void k_adam(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
                       const float* __restrict__ g, long long n, float lr, float b1, float b2, float eps, float c1,
                       float c2) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// --------------------------------------------------------------- host side --
// blocks of a k_mlp_rows launch over `rows` rows (its shared memory opted into
// per device)
template <bool TRAIN>
static int row_blocks(long long rows, int* blocks) {
    static std::atomic<int> bps_of[64];
    int dev = 0;
    DWG_CHECK_CUDA(cudaGetDevice(&dev));
    DWG_REQUIRE(dev >= 0 && dev < 64, "mlp: device %d out of range", dev);
    if (!bps_of[dev]) {
        DWG_CHECK_CUDA(cudaFuncSetAttribute(k_mlp_rows<TRAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowSmem));
        DWG_CHECK_CUDA(cudaFuncSetAttribute(k_mlp_weights, cudaFuncAttributeMaxDynamicSharedMemorySize, kWSmem));
        int bps = 0;
        DWG_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_mlp_rows<TRAIN>, kRowWarps * 32, kRowSmem));
        bps_of[dev] = bps > 0 ? bps : 1;
    }
    const long long tiles = (rows + 15) / 16;
    *blocks = (int)std::min<long long>((tiles + kRowWarps - 1) / kRowWarps, (long long)num_sms() * bps_of[dev]);
    return DWG_OK;
}

static int ensure_cap(Mlp& m, long long B) {
    if (B <= m.cap) return DWG_OK;
    const size_t rows = (size_t)(B + 15) / 16 * 16;
    DWG_TRY(m.x.reserve(rows * kMlpInPad));
    for (int l = 0; l < 3; ++l) {
        DWG_TRY(m.gp[l].reserve(rows * kMlpHidden));
        DWG_TRY(m.h[l].reserve(rows * kMlpHidden));
        DWG_TRY(m.dz[l].reserve(rows * kMlpHidden));
    }
    DWG_TRY(m.dy.reserve(rows * kMlpOutPad));
    m.cap = B;
    return DWG_OK;
}

static int refresh_bf16(Mlp& m, cudaStream_t s) {
    for (int l = 0; l < kMlpLayers; ++l) {
        const long long nw = (long long)m.din[l] * m.dout[l];
        k_to_bf16<<<div_up(nw, 256), 256, 0, s>>>(m.w[l].ptr, nw, m.wb[l].ptr);
    }
    DWG_CHECK_LAUNCH();
    return DWG_OK;
}

int mlp_init(Mlp& m, unsigned long long seed, cudaStream_t s) {
    std::mt19937_64 gen(seed);
    const int real_in[kMlpLayers] = {kMlpIn, kMlpHidden, kMlpHidden, kMlpHidden};
    const int real_out[kMlpLayers] = {kMlpHidden, kMlpHidden, kMlpHidden, kMlpOut};
    for (int l = 0; l < kMlpLayers; ++l) {
        const int din = m.din[l], dout = m.dout[l];
        std::vector<float> w((size_t)din * dout, 0.f), b(dout, 0.f);
        const float lim = std::sqrt(6.0f / (float)real_in[l]);
        std::uniform_real_distribution<float> U(-lim, lim);
        for (int i = 0; i < real_in[l]; ++i)
            for (int o = 0; o < real_out[l]; ++o) w[(size_t)i * dout + o] = U(gen) * (l == kMlpLayers - 1 ? 0.3f : 1.f);
        DWG_TRY(m.w[l].reserve(w.size()));
        DWG_TRY(m.b[l].reserve(b.size()));
        DWG_TRY(m.wb[l].reserve(w.size()));
        for (auto* buf : {&m.mw[l], &m.vw[l]}) {
            DWG_TRY(buf->reserve(w.size()));
            DWG_CHECK_CUDA(cudaMemsetAsync(buf->ptr, 0, sizeof(float) * w.size(), s));
        }
        for (auto* buf : {&m.mb[l], &m.vb[l]}) {
            DWG_TRY(buf->reserve(b.size()));
            DWG_CHECK_CUDA(cudaMemsetAsync(buf->ptr, 0, sizeof(float) * b.size(), s));
        }
        DWG_CHECK_CUDA(cudaMemcpyAsync(m.w[l].ptr, w.data(), sizeof(float) * w.size(), cudaMemcpyHostToDevice, s));
        DWG_CHECK_CUDA(cudaMemcpyAsync(m.b[l].ptr, b.data(), sizeof(float) * b.size(), cudaMemcpyHostToDevice, s));
    }
    DWG_TRY(m.loss.reserve(1));
    DWG_TRY(m.grad.reserve((size_t)mlp_param_count()));
    float* g = m.grad.ptr;  // the gradients in the flat order
    for (int l = 0; l < kMlpLayers; ++l) {
        m.gw[l] = g;
        g += (size_t)m.din[l] * m.dout[l];
        m.gb[l] = g;
        g += m.dout[l];
    }
    m.step = 0;
    DWG_TRY(refresh_bf16(m, s));
    DWG_CHECK_CUDA(cudaStreamSynchronize(s));
    return DWG_OK;
}

long long mlp_param_count() {
    const Mlp m;
    long long c = 0;
    for (int l = 0; l < kMlpLayers; ++l) c += (long long)m.din[l] * m.dout[l] + m.dout[l];
    return c;
}

int mlp_set_flat(Mlp& m, const float* params_host, cudaStream_t s) {
    DWG_REQUIRE(params_host, "mlp_set_flat: null parameters");
    const float* src = params_host;
    for (int l = 0; l < kMlpLayers; ++l) {
        const size_t nw = (size_t)m.din[l] * m.dout[l];
        DWG_CHECK_CUDA(cudaMemcpyAsync(m.w[l].ptr, src, sizeof(float) * nw, cudaMemcpyHostToDevice, s));
        src += nw;
        DWG_CHECK_CUDA(cudaMemcpyAsync(m.b[l].ptr, src, sizeof(float) * m.dout[l], cudaMemcpyHostToDevice, s));
        src += m.dout[l];
    }
    DWG_TRY(refresh_bf16(m, s));
    DWG_CHECK_CUDA(cudaStreamSynchronize(s));
    return DWG_OK;
}

int mlp_get_flat(Mlp& m, float* params_host, cudaStream_t s) {
    DWG_REQUIRE(params_host, "mlp: null output");
    DWG_CHECK_CUDA(cudaStreamSynchronize(s));
    float* dst = params_host;
    for (int l = 0; l < kMlpLayers; ++l) {
        const size_t nw = (size_t)m.din[l] * m.dout[l];
        DWG_CHECK_CUDA(cudaMemcpy(dst, m.w[l].ptr, sizeof(float) * nw, cudaMemcpyDeviceToHost));
        dst += nw;
        DWG_CHECK_CUDA(cudaMemcpy(dst, m.b[l].ptr, sizeof(float) * m.dout[l], cudaMemcpyDeviceToHost));
        dst += m.dout[l];
    }
    return DWG_OK;
}

int mlp_get_grads_flat(Mlp& m, float* grads_host, cudaStream_t s) {
    DWG_REQUIRE(grads_host, "mlp: null output");
    DWG_CHECK_CUDA(cudaStreamSynchronize(s));
    DWG_CHECK_CUDA(cudaMemcpy(grads_host, m.grad.ptr, sizeof(float) * (size_t)mlp_param_count(), cudaMemcpyDeviceToHost));
    return DWG_OK;
}

static RowArgs row_args(const Mlp& m, const float* F, long long rows) {
    RowArgs a{};
    a.F = F;
    a.rows = rows;
    for (int l = 0; l < kMlpLayers; ++l) {
        a.w[l] = m.wb[l].ptr;
        a.b[l] = m.b[l].ptr;
    }
    return a;
}

int mlp_forward(Mlp& m, const float* F, long long n, float* out, cudaStream_t s) {
    DWG_REQUIRE(F && out && n >= 0, "mlp_forward: bad arguments");
    if (n == 0) return DWG_OK;
    RowArgs a = row_args(m, F, n);
    a.out = out;
    int blocks = 0;
    DWG_TRY(row_blocks<false>(n, &blocks));
    k_mlp_rows<false><<<blocks, kRowWarps * 32, kRowSmem, s>>>(a);
    DWG_CHECK_LAUNCH();
    return DWG_OK;
}

int mlp_backward(Mlp& m, const float* F, const float* T, long long B, float* loss_host, cudaStream_t s) {
    DWG_REQUIRE(F && T && B >= 1 && B < (1ll << 31), "mlp_backward: bad arguments");
    DWG_TRY(ensure_cap(m, B));
    int blocks = 0;
    DWG_TRY(row_blocks<true>(B, &blocks));
    const long long tiles = (B + 15) / 16, sets = (tiles + 7) / 8;
    // three blocks per chunk, about two per SM
    const int chunks = (int)std::min<long long>(sets, std::max(1, num_sms() * 2 / 3));
    DWG_TRY(m.bias_part.reserve((size_t)blocks * kBias));
    DWG_TRY(m.loss_part.reserve(blocks));
    DWG_TRY(m.part.reserve((size_t)chunks * kParts));
    RowArgs a = row_args(m, F, B);
    a.T = T;
    a.x = reinterpret_cast<uint4*>(m.x.ptr);
    a.dy = reinterpret_cast<unsigned*>(m.dy.ptr);
    a.bias_part = m.bias_part.ptr;
    a.loss_part = m.loss_part.ptr;
    WeightArgs wa{};
    wa.tiles = tiles;
    wa.x = a.x;
    wa.dy = a.dy;
    wa.part = m.part.ptr;
    GradOut o;
    for (int l = 0; l < 3; ++l) {
        a.gp[l] = reinterpret_cast<float4*>(m.gp[l].ptr);
        wa.h[l] = a.h[l] = reinterpret_cast<uint2*>(m.h[l].ptr);
        wa.dz[l] = a.dz[l] = reinterpret_cast<uint2*>(m.dz[l].ptr);
    }
    for (int l = 0; l < kMlpLayers; ++l) {
        o.gw[l] = m.gw[l];
        o.gb[l] = m.gb[l];
    }
    k_mlp_rows<true><<<blocks, kRowWarps * 32, kRowSmem, s>>>(a);
    DWG_CHECK_LAUNCH();
    k_mlp_weights<<<dim3(chunks, 3), kRowWarps * 32, kWSmem, s>>>(wa);
    DWG_CHECK_LAUNCH();
    k_mlp_reduce<<<div_up(kParts + (kBias + 1) * 32, 128), 128, 0, s>>>(m.part.ptr, chunks, m.bias_part.ptr,
                                                                        m.loss_part.ptr, blocks, B, o, m.loss.ptr);
    DWG_CHECK_LAUNCH();
    if (loss_host) {
        DWG_CHECK_CUDA(cudaMemcpyAsync(loss_host, m.loss.ptr, sizeof(float), cudaMemcpyDeviceToHost, s));
        DWG_CHECK_CUDA(cudaStreamSynchronize(s));
    }
    return DWG_OK;
}

int mlp_adam(Mlp& m, float lr, float b1, float b2, float eps, cudaStream_t s) {
    m.step += 1;
    const float c1 = 1.f - std::pow(b1, (float)m.step), c2 = 1.f - std::pow(b2, (float)m.step);
    for (int l = 0; l < kMlpLayers; ++l) {
        const long long nw = (long long)m.din[l] * m.dout[l];
        k_adam<<<div_up(nw, 256), 256, 0, s>>>(m.w[l].ptr, m.mw[l].ptr, m.vw[l].ptr, m.gw[l], nw, lr, b1, b2, eps,
                                               c1, c2);
        k_adam<<<div_up(m.dout[l], 256), 256, 0, s>>>(m.b[l].ptr, m.mb[l].ptr, m.vb[l].ptr, m.gb[l], m.dout[l], lr,
                                                      b1, b2, eps, c1, c2);
    }
    DWG_CHECK_LAUNCH();
    return refresh_bf16(m, s);
}

__global__ void k_unit_or_gauss(const float* __restrict__ y, const float* __restrict__ P, int n,
                                const float* __restrict__ bb, float* __restrict__ N) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float a = y[(size_t)i * 3], b = y[(size_t)i * 3 + 1], c = y[(size_t)i * 3 + 2];
    const float len = sqrtf(a * a + b * b + c * c);
    if (len > 1e-12f && isfinite(len)) {
        N[(size_t)i * 3] = a / len;
        N[(size_t)i * 3 + 1] = b / len;
        N[(size_t)i * 3 + 2] = c / len;
        return;
    }
    // Gauss map (src/TurboNormalInit.cu:3-44)
    float v[3];
    for (int d = 0; d < 3; ++d) v[d] = __fsub_rn(P[(size_t)i * 3 + d], __fdiv_rn(__fadd_rn(bb[d], bb[3 + d]), 2.0f));
    const float sc = inv_len_eps(__fsqrt_rn(sq3_rn(v[0], v[1], v[2])));
    for (int d = 0; d < 3; ++d) N[(size_t)i * 3 + d] = __fmul_rn(v[d], sc);
}

int mlp_init_normals(Mlp& m, const KnnIndex& ix, const float* P, int n, float* N, cudaStream_t s) {
    DWG_REQUIRE(P && N && n >= 1, "mlp_init_normals: bad arguments");
    DevBuf<float> F, y;
    DWG_TRY(F.reserve((size_t)n * kMlpIn));
    DWG_TRY(y.reserve((size_t)n * 3));
    DWG_TRY(mlp_features(ix, P, n, F.ptr, s));
    DWG_TRY(mlp_forward(m, F.ptr, n, y.ptr, s));
    k_unit_or_gauss<<<div_up(n, 256), 256, 0, s>>>(y.ptr, P, n, ix.bbox.ptr, N);
    DWG_CHECK_LAUNCH();
    DWG_CHECK_CUDA(cudaStreamSynchronize(s));  // F and y are released on return
    return DWG_OK;
}

}  // namespace dwg
