// Element-stratified feature maps summed per molecule, on the tensor cores.
//
// * Random Fourier features (the reference's elemental RFF,
//   src/rff_elemental.hpp:7-24, GPU version src/cuda_rff_features.cu):
//     z_mol = sum over atoms a of element e: sqrt(2/D) cos(x_a . W_e + b_e)
//   x_a . W_e runs as a split-fp16 tcgen05 GEMM (hi*hi + hi*lo + lo*hi, FP32
//   accumulation); the epilogue adds b_e, takes the cosine and sums the rows
//   of each molecule before one atomic add per (molecule run, feature).
// * The learned cos-MLP map (no reference counterpart), per element e:
//     phi_e(x) = sqrt(2/D) cos(W2_e h + b2_e),   h = cos(W1_e x + b1_e)
//   with BF16 weights and activations and FP32 accumulation; layer 1's
//   epilogue writes h, layer 2's sums phi per molecule like the RFF path.
// * Its training step on same-element atom pairs,
//     loss = mean_p (phi(x_i) . phi(x_j) - exp(-|x_i - x_j|^2 / (2 sigma^2)))^2,
//   forward GEMMs with activation epilogues, the pair loss kernel, the three
//   backward GEMMs (dW2 = dZ2^T H, dH = dZ2 W2 fused with the cos derivative,
//   dW1 = dZ1^T X) and an Adam update that refreshes the BF16 weight copies.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <mutex>
#include <vector>

#include "derivs.h"
#include "tc_gemm.h"

using bf16 = __nv_bfloat16;

struct kfb_cosmlp {
    int nelem = 0, rep = 0, hidden = 0, d = 0, max_pairs = 0, device = 0;
    // FP32 master parameters, element-major: w1 (nelem, H, rep), b1 (nelem, H),
    // w2 (nelem, D, H), b2 (nelem, D)
    kfb::DevBuf w1, b1, w2, b2;
    kfb::DevBuf w1b, w2b, w2tb;  // BF16 copies: w1, w2 and w2 transposed (nelem, H, D)
    kfb::DevBuf mom[4], var[4];  // Adam moments per parameter tensor
    kfb::DevBuf grad[4];         // gradients of the last step (one element)
    std::vector<int> steps;      // Adam step count per element
    // batch workspace (2 Bp rows, Bp = max_pairs rounded up to 8)
    kfb::DevBuf xb, xbt, z1, hb, hbt, z2, factor, dz2, dz2t, dz1t, loss, err;
};

namespace kfb {

namespace {

constexpr float ADAM_B1 = 0.9f, ADAM_B2 = 0.999f, ADAM_EPS = 1e-8f;

long long ru8(long long v) { return (v + 7) / 8 * 8; }
unsigned nblk(long long n, int b) { return (unsigned)std::max<long long>(1, (n + b - 1) / b); }

// out[r][c] = bf16(x[a][c]) for a = idx[r], or with idx2 (a pair batch of
// npairs) idx[r] for r < npairs, idx2[r - nrows / 2] for the first npairs rows
// of the second half, and no row between; a zero row for a < 0, a zero row and
// *bad raised for a >= nsrc; optionally also the transpose out_t[c * ld_t + r],
// through a 32 x 32 shared-memory tile.
template <class T>
__global__ void gather_rows_bf16_kernel(const T *__restrict__ x, long long nsrc,
                                        const int *__restrict__ idx,
                                        const int *__restrict__ idx2, int npairs, int nrows,
                                        int rep,
                                        bf16 *__restrict__ out, bf16 *__restrict__ out_t,
                                        long long ld_t, int *bad) {
    __shared__ float tile[32][33];
    const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
    for (int rr = threadIdx.y; rr < 32; rr += blockDim.y) {
        const int r = r0 + rr, c = c0 + threadIdx.x;
        float v = 0.f;
        if (r < nrows && c < rep) {
            int a;
            if (!idx2) {
                a = idx[r];
            } else {
                const int half = nrows / 2, p = r < half ? r : r - half;
                a = p < npairs ? (r < half ? idx[p] : idx2[p]) : -1;
            }
            if (a >= nsrc) {
                if (bad) atomicExch(bad, 1);  // index outside x: zero row, reported
            } else if (a >= 0) {
                v = (float)x[(size_t)a * rep + c];
            }
            out[(size_t)r * rep + c] = __float2bfloat16_rn(v);
        }
        tile[rr][threadIdx.x] = v;
    }
    if (!out_t) return;
    __syncthreads();
    for (int cc = threadIdx.y; cc < 32; cc += blockDim.y) {
        const int c = c0 + cc, r = r0 + threadIdx.x;
        if (c < rep && r < nrows)
            out_t[(size_t)c * ld_t + r] = __float2bfloat16_rn(tile[threadIdx.x][cc]);
    }
}

template <class T>
__global__ void gather_rows_f32_kernel(const T *__restrict__ x, const int *__restrict__ idx,
                                       int nrows, int rep, float *__restrict__ out) {
    const long long n = (long long)nrows * rep;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(i / rep), c = (int)(i % rep);
        const int a = idx[r];
        out[i] = a >= 0 ? (float)x[(size_t)a * rep + c] : 0.f;
    }
}

// dst[c * ld_dst + r] = src[r][c] for a BF16 (rows, cols) array.  64 x 64 tiles
// through shared memory; bf16x2 loads along c and bf16x2 stores along r when cols, ld_dst and
// the pointers allow it (128-byte accesses per warp), element-wise otherwise.
__global__ void transpose_bf16_kernel(const bf16 *__restrict__ src, int rows, int cols,
                                      bf16 *__restrict__ dst, long long ld_dst, int pairs) {
    __shared__ float tile[64][65];
    const int r0 = blockIdx.y * 64, c0 = blockIdx.x * 64;
    const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
    for (int rr = ty; rr < 64; rr += 8) {
        const int r = r0 + rr, c = c0 + 2 * tx;
        float v0 = 0.f, v1 = 0.f;
        if (r < rows) {
            if (pairs && c + 1 < cols) {
                const __nv_bfloat162 t =
                    *reinterpret_cast<const __nv_bfloat162 *>(src + (size_t)r * cols + c);
                v0 = __low2float(t);
                v1 = __high2float(t);
            } else {
                if (c < cols) v0 = __bfloat162float(src[(size_t)r * cols + c]);
                if (c + 1 < cols) v1 = __bfloat162float(src[(size_t)r * cols + c + 1]);
            }
        }
        tile[rr][2 * tx] = v0;
        tile[rr][2 * tx + 1] = v1;
    }
    __syncthreads();
    for (int cc = ty; cc < 64; cc += 8) {
        const int c = c0 + cc, r = r0 + 2 * tx;
        const float v0 = tile[2 * tx][cc], v1 = tile[2 * tx + 1][cc];
        if (c < cols) {
            bf16 *d = dst + (size_t)c * ld_dst + r;
            if (pairs && r + 1 < rows) {
                *reinterpret_cast<__nv_bfloat162 *>(d) = __floats2bfloat162_rn(v0, v1);
            } else {
                if (r < rows) d[0] = __float2bfloat16_rn(v0);
                if (r + 1 < rows) d[1] = __float2bfloat16_rn(v1);
            }
        }
    }
}

kfb_status transpose_bf16(const bf16 *src, int rows, int cols, bf16 *dst, long long ld_dst,
                          cudaStream_t s) {
    const bool pairs = cols % 2 == 0 && ld_dst % 2 == 0 &&
                       (reinterpret_cast<uintptr_t>(src) & 3u) == 0 &&
                       (reinterpret_cast<uintptr_t>(dst) & 3u) == 0;
    transpose_bf16_kernel<<<dim3(nblk(cols, 64), nblk(rows, 64)), dim3(32, 8), 0, s>>>(
        src, rows, cols, dst, ld_dst, pairs ? 1 : 0);
    KFB_CUDA_TRY(cudaGetLastError());
    return KFB_OK;
}

// out[r] = sum_c src[r][c] (BF16 rows, FP32 sums), one 256-thread block per
// row, 16-byte loads when the row allows them
__global__ void rowsum_bf16_kernel(const bf16 *__restrict__ src, int rows, int cols,
                                   float *__restrict__ out) {
    const int r = blockIdx.x;
    if (r >= rows) return;
    const bf16 *row = src + (size_t)r * cols;
    float t = 0.f;
    const bool vec = cols % 8 == 0 && (reinterpret_cast<uintptr_t>(row) & 15u) == 0;
    if (vec) {
        const uint4 *v = reinterpret_cast<const uint4 *>(row);
        for (int c = threadIdx.x; c < cols / 8; c += blockDim.x) {
            const uint4 u = v[c];
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const __nv_bfloat162 b2 = *reinterpret_cast<const __nv_bfloat162 *>(&w[q]);
                t += __low2float(b2) + __high2float(b2);
            }
        }
    } else {
        for (int c = threadIdx.x; c < cols; c += blockDim.x) t += __bfloat162float(row[c]);
    }
    __shared__ float red[32];
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        float s = 0.f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
        out[r] = s;
    }
}

// Exact pair-kernel values e_p = exp(-|x_i - x_j|^2 / (2 sigma^2)) (squared
// distance of the difference, FP64 accumulation), one warp per pair.
template <class T>
__global__ void pair_gaussian_kernel(const T *__restrict__ x, long long nsrc,
                                     const int *__restrict__ pi, const int *__restrict__ pj,
                                     int npairs, int rep, double c, float *__restrict__ out,
                                     int *bad) {
    const int p = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (p >= npairs) return;
    const int ia = pi[p], ib = pj[p];
    if (ia < 0 || ib < 0 || ia >= nsrc || ib >= nsrc) {
        if (lane == 0) {
            out[p] = 0.f;
            atomicExch(bad, 1);
        }
        return;
    }
    const T *a = x + (size_t)ia * rep;
    const T *b = x + (size_t)ib * rep;
    double t = 0.0;
    for (int k = lane; k < rep; k += 32) {
        const double d = (double)a[k] - (double)b[k];
        t += d * d;
    }
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) out[p] = (float)exp(c * t);
}

// sin and cos of x: reduce to r = x - 2 pi round(x / 2 pi) in [-pi, pi] (2 pi
// split into a float head and tail so the product is exact to ~1e-7 for the
// |x| < 1e3 the network produces), then the hardware approximation, whose
// absolute error on [-pi, pi] is about 1e-6.
__device__ __forceinline__ void sincos_reduced(float x, float &sn, float &cs) {
    const float TWO_PI_HI = 6.28318548202514648f;     // float(2 pi)
    const float TWO_PI_LO = -1.74845553e-07f;          // 2 pi - TWO_PI_HI
    const float k = rintf(x * 0.159154943091895336f);  // x / (2 pi)
    const float r = fmaf(-k, TWO_PI_LO, fmaf(-k, TWO_PI_HI, x));
    __sincosf(r, &sn, &cs);
}

// Pair loss and the gradient at layer 2's pre-activation.  Rows p and p + Bp
// of z2 are the two atoms of pair p.  With s2 = 2 / D:
//   k_p = s2 sum_d cos z_i[d] cos z_j[d],  r_p = k_p - t_p,  loss += r_p^2
//   dZ2_i[d] = -(2 r_p / npairs) s2 cos z_j[d] sin z_i[d]   (and i <-> j)
// Padded pairs (p >= npairs) get zero gradient rows.
//
// Two passes over z2: the dot products (a warp per pair; factor[p] = (2 r_p /
// npairs) s2), then the gradients by tiles of 64 pairs x 64 columns, written by
// rows and, through shared memory, transposed (dz2t, row length 2 Bp), with
// their column sums (db2, cleared by the caller).  Both are bound by HBM; a
// transpose pass that reads dZ2 back moves as much and more (50 + 48 us for
// 8,192 rows of 4,096), and 8- or 16-byte pieces of the transpose written
// straight from a block of few pairs took 110 us.
constexpr int PL_MAX_D = 4096;   // largest D a map is created with (what the tests cover)
__global__ void __launch_bounds__(256)
    pair_dot_kernel(const float *__restrict__ z2, int Bp, int npairs, int D,
                    const float *__restrict__ target, float s2, float gscale,
                    float *__restrict__ factor, double *__restrict__ loss) {
    const int p = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (p >= Bp) return;
    float t = 0.f;
    if (p < npairs) {
        const float4 *zi = reinterpret_cast<const float4 *>(z2 + (size_t)p * D);
        const float4 *zj = reinterpret_cast<const float4 *>(z2 + (size_t)(p + Bp) * D);
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int k = lane; k < D / 4; k += 32) {
            const float4 a = zi[k], b = zj[k];
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float sa, ca, sb, cb;
                sincos_reduced(av[c], sa, ca);
                sincos_reduced(bv[c], sb, cb);
                acc[c] = fmaf(ca, cb, acc[c]);
            }
        }
        t = (acc[0] + acc[1]) + (acc[2] + acc[3]);
    }
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) {
        float f = 0.f;
        if (p < npairs) {
            const float r = s2 * t - target[p];
            atomicAdd(loss, (double)r * (double)r);
            f = gscale * r * s2;
        }
        factor[p] = f;
    }
}

constexpr int PG_T = 64;   // pairs and columns of a tile
__global__ void __launch_bounds__(256)
    pair_grad_kernel(const float *__restrict__ z2, int Bp, int npairs, int D,
                     const float *__restrict__ factor, bf16 *__restrict__ dz2,
                     bf16 *__restrict__ dz2t, float *__restrict__ db2) {
    // [half][column][pair]; rows of 66 (33 words): columns go in and come out
    // without bank conflicts
    __shared__ __align__(4) bf16 tile[2][PG_T][PG_T + 2];
    const int p0 = blockIdx.y * PG_T, c0 = blockIdx.x * PG_T;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;   // 4 columns, pairs ty, ty + 16, ..
    const int c = c0 + 4 * tx;
#pragma unroll
    for (int h = 0; h < PG_T / 16; ++h) {
        const int q = ty + 16 * h, p = p0 + q;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        float f = 0.f;
        if (p < npairs && c < D) {   // D is a multiple of 8
            a = *reinterpret_cast<const float4 *>(z2 + (size_t)p * D + c);
            b = *reinterpret_cast<const float4 *>(z2 + (size_t)(p + Bp) * D + c);
            f = factor[p];
        }
        const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
        bf16 gi[4], gj[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            float sa, ca, sb, cb;
            sincos_reduced(av[u], sa, ca);
            sincos_reduced(bv[u], sb, cb);
            gi[u] = __float2bfloat16_rn(-f * cb * sa);
            gj[u] = __float2bfloat16_rn(-f * ca * sb);
            tile[0][4 * tx + u][q] = gi[u];
            tile[1][4 * tx + u][q] = gj[u];
        }
        if (p < Bp && c < D) {
            const __nv_bfloat162 w[4] = {{gi[0], gi[1]}, {gi[2], gi[3]}, {gj[0], gj[1]},
                                         {gj[2], gj[3]}};
            *reinterpret_cast<uint2 *>(dz2 + (size_t)p * D + c) =
                *reinterpret_cast<const uint2 *>(w);
            *reinterpret_cast<uint2 *>(dz2 + (size_t)(p + Bp) * D + c) =
                *reinterpret_cast<const uint2 *>(w + 2);
        }
    }
    __syncthreads();
    // a warp per column: 64 pairs of each half, two per lane (Bp is a multiple of 8)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int cc = warp; cc < PG_T && c0 + cc < D; cc += 8) {
        float t = 0.f;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const __nv_bfloat162 v =
                *reinterpret_cast<const __nv_bfloat162 *>(&tile[half][cc][2 * lane]);
            t += __low2float(v) + __high2float(v);
            if (p0 + 2 * lane < Bp)
                *reinterpret_cast<__nv_bfloat162 *>(dz2t + (size_t)(c0 + cc) * 2 * Bp +
                                                    (size_t)half * Bp + p0 + 2 * lane) = v;
        }
        for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) atomicAdd(db2 + c0 + cc, t);
    }
}

// Adam on the parameter tensors of an element in one launch, refreshing their
// BF16 copies (pb) where given; block b works on tensor k with first[k] <= b.
struct AdamSet {
    float *p[4], *m[4], *v[4];
    const float *g[4];
    bf16 *pb[4];
    long long n[4];
    int first[5];
};
__global__ void __launch_bounds__(256) adam_kernel(const __grid_constant__ AdamSet a, float lr,
                                                   float bc1, float bc2) {
    int k = 0;
    while (k < 3 && (int)blockIdx.x >= a.first[k + 1]) ++k;
    float *p = a.p[k], *m = a.m[k], *v = a.v[k];
    const float *g = a.g[k];
    bf16 *pb = a.pb[k];
    const long long n = a.n[k], step = (long long)(a.first[k + 1] - a.first[k]) * blockDim.x;
    for (long long i = (blockIdx.x - a.first[k]) * (long long)blockDim.x + threadIdx.x; i < n;
         i += step) {
        const float gi = g[i];
        const float mi = ADAM_B1 * m[i] + (1.f - ADAM_B1) * gi;
        const float vi = ADAM_B2 * v[i] + (1.f - ADAM_B2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float pi = p[i] - lr * (mi / bc1) / (sqrtf(vi / bc2) + ADAM_EPS);
        p[i] = pi;
        if (pb) pb[i] = __float2bfloat16_rn(pi);
    }
}

__global__ void to_bf16_kernel(const float *__restrict__ p, int rows, int cols,
                               bf16 *__restrict__ pb, bf16 *__restrict__ pbt) {
    const long long n = (long long)rows * cols;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const bf16 h = __float2bfloat16_rn(p[i]);
        if (pb) pb[i] = h;
        if (pbt) pbt[(i % cols) * rows + i / cols] = h;
    }
}

// Atoms of each element in molecule order: flat padded indices m * ma + j and
// the molecule of each row.
struct ElemRows {
    std::vector<std::vector<int>> idx, mol;
};

kfb_status elem_rows(const int *q, const int *n, int nm, int ma, int nelem, ElemRows &er) {
    er.idx.assign(nelem, {});
    er.mol.assign(nelem, {});
    for (int m = 0; m < nm; ++m) {
        const int na = std::min(std::max(n[m], 0), ma);
        for (int j = 0; j < na; ++j) {
            const int e = q[(size_t)m * ma + j];
            if (e < 0) continue;
            if (e >= nelem)
                return set_error(KFB_ERR_INVALID_ARG,
                                 "element index %d out of range [0, %d) (molecule %d, atom %d)", e,
                                 nelem, m, j);
            er.idx[e].push_back(m * ma + j);
            er.mol[e].push_back(m);
        }
    }
    return KFB_OK;
}

size_t feature_budget() {
    static size_t b = [] {
        const char *v = std::getenv("KFB_WORKSPACE_GB");
        double gb = v ? std::atof(v) : 4.0;
        if (!(gb > 0)) gb = 4.0;
        return (size_t)(gb * (1ull << 30));
    }();
    return b;
}

// ---------------------------------------------------------------- RFF
// Operands of the RFF products (x W_e and dX^T W_e): fp16 pairs with K along
// the descriptor columns that the atoms use (cols, n of them; W's rows that
// meet only zeros are left out), K padded with zeros to a multiple of 16, and
// a power-of-two scale for each element's W and for the x and dX of each chunk
// of an element's atoms: a pair resolves 2^-38 of its scale's largest value, so
// small elements need scales of their own.

// amax[e] = max |w_e|; a column with a value that is not finite counts as used
// (its products with zeros are not zero).  Rows of d values, row r is column
// r % rep of element r / rep.
__global__ void __launch_bounds__(256) rff_weight_scan_kernel(const float *__restrict__ w, int rep,
                                                              int d, float *__restrict__ amax,
                                                              int *__restrict__ used) {
    const float *row = w + (size_t)blockIdx.x * d;
    float m = 0.f;
    bool bad = false;
    for (int c = threadIdx.x; c < d; c += blockDim.x) {
        const float v = fabsf(row[c]);
        m = fmaxf(m, v);
        bad |= !(v <= 3.402823466e38f);
    }
    if (bad) used[blockIdx.x % rep] = 1;
    for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<int *>(amax) + blockIdx.x / rep, __float_as_int(m));
}

__device__ __forceinline__ void split_fp16(float v, __half &h, __half &l) {
    h = __float2half_rn(v);
    l = __float2half_rn(v - __half2float(h));
}

// out[r][p] = pair of scale x[idx[r]][cols[p]] (p < n), zero for n <= p < kpad
template <class T>
__global__ void rff_x_rows_kernel(const T *__restrict__ x, const int *__restrict__ idx, int nrows,
                                  int rep, const int *__restrict__ cols, int n, int kpad,
                                  float scale, __half *__restrict__ hi, __half *__restrict__ lo) {
    const long long total = (long long)nrows * kpad;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(i / kpad), p = (int)(i - (long long)r * kpad);
        const float v = p < n ? (float)x[(size_t)idx[r] * rep + cols[p]] * scale : 0.f;
        split_fp16(v, hi[i], lo[i]);
    }
}

// wt[c][p] = pair of scale w[cols[p]][c] (w: rep rows of d), zero for n <= p < kpad
__global__ void rff_w_rows_kernel(const float *__restrict__ w, int d, const int *__restrict__ cols,
                                  int n, int kpad, float scale, __half *__restrict__ hi,
                                  __half *__restrict__ lo) {
    __shared__ float tile[32][33];
    const int p0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int p = p0 + r, c = c0 + threadIdx.x;
        tile[r][threadIdx.x] = (p < n && c < d) ? w[(size_t)cols[p] * d + c] * scale : 0.f;
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int c = c0 + r, p = p0 + threadIdx.x;
        if (c < d && p < kpad) {
            const size_t o = (size_t)c * kpad + p;
            split_fp16(tile[threadIdx.x][r], hi[o], lo[o]);
        }
    }
}

// Jacobian rows of a chunk's atoms: row + c step = pair of scale
// dx[atom][cols[.]][c] for c < ncol; with them the destination row dst + c and
// the atom's number in the chunk (its row of sines).  Tiles of 64 columns x 32
// coordinates through shared memory: dX is read along its rows, the pairs are
// written 128 bytes a warp (a row per thread block read dX 4 bytes per 32-byte
// sector: 0.59 ms for 3,150 atoms of 21).
struct RffAtom {
    int atom, row, step, ncol, dst;
};
template <class T>
__global__ void __launch_bounds__(256) rff_jacobian_rows_kernel(
    const T *__restrict__ dx, const RffAtom *__restrict__ atoms, int rep, int ld,
    const int *__restrict__ cols, int n, int kpad, float scale, __half *__restrict__ hi,
    __half *__restrict__ lo, int *__restrict__ dst, int *__restrict__ aux) {
    __shared__ float tile[64][33];
    const RffAtom a = atoms[blockIdx.x];
    const int p0 = blockIdx.y * 64, c0 = blockIdx.z * 32;
    if (c0 >= a.ncol) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const T *base = dx + (size_t)a.atom * rep * ld;
    for (int r = warp; r < 64; r += 8) {
        const int p = p0 + r, c = c0 + lane;
        tile[r][lane] = (p < n && c < a.ncol) ? (float)base[(size_t)cols[p] * ld + c] * scale : 0.f;
    }
    __syncthreads();
    const int p = p0 + 2 * lane;
    for (int r = warp; r < 32; r += 8) {
        const int c = c0 + r;
        if (c >= a.ncol) break;
        const long long row = a.row + (long long)c * a.step;
        if (p < kpad) {   // kpad is a multiple of 16
            __half2 h, l;
            split_fp16(tile[2 * lane][r], h.x, l.x);
            split_fp16(tile[2 * lane + 1][r], h.y, l.y);
            *reinterpret_cast<__half2 *>(hi + row * kpad + p) = h;
            *reinterpret_cast<__half2 *>(lo + row * kpad + p) = l;
        }
        if (p0 == 0 && lane == 0) {
            dst[row] = a.dst + c;
            aux[row] = (int)blockIdx.x;
        }
    }
}

// What both RFF maps prepare: used columns, scales, element rows.  Chunk r0 /
// chunk of element e (atoms r0 .. of its list) has the slot first[e] + r0 / chunk.
struct RffPlan {
    ElemRows er;
    DevBuf cols, err, wh, wl, xh, xl;
    int n = 0, kpad = 0, chunk = 0;
    std::vector<int> first;
    std::vector<float> x_scale, dx_scale, w_scale;   // by slot, by slot, by element
    int slot(int e, int r0) const { return first[e] + r0 / chunk; }
};

template <class T>
kfb_status rff_plan(const T *x, const T *dx, const int *q, const int *n, int nm, int ma, int rep,
                    const float *w, int nelem, int d, int chunk, RffPlan &pl, cudaStream_t s) {
    KFB_TRY(elem_rows(q, n, nm, ma, nelem, pl.er));
    pl.chunk = chunk;
    // atom counts, then the slot of every atom (-1: of no element)
    std::vector<int> atoms((size_t)nm * (ma + 1), -1);
    std::copy(n, n + nm, atoms.begin());
    int nslot = 0;
    for (int e = 0; e < nelem; ++e) {
        const std::vector<int> &ai = pl.er.idx[e];
        pl.first.push_back(nslot);
        for (size_t t = 0; t < ai.size(); ++t)
            atoms[(size_t)nm + ai[t]] = nslot + (int)(t / (size_t)chunk);
        nslot += (int)((ai.size() + chunk - 1) / (size_t)chunk);
    }
    // used columns (rep ints), then max |w| by element, max |x|, |dx| by slot
    DevBuf scan, da;
    const size_t words = (size_t)rep + nelem + 2 * (size_t)nslot;
    KFB_TRY(scan.alloc(words * sizeof(int), s));
    KFB_TRY(zero(scan.ptr, words * sizeof(int), s));
    float *amax = reinterpret_cast<float *>(scan.as<int>() + rep);
    KFB_TRY(upload(da, atoms, s));
    DerivSet ds;
    ds.x = x;
    ds.dx = dx;
    ds.v.n = atoms.data();
    ds.v.nm = nm;
    ds.v.ma = ma;
    KFB_TRY(scan_columns<T>(ds, rep, da.as<int>(), scan.as<int>(), amax + nelem, s,
                            da.as<int>() + nm));
    rff_weight_scan_kernel<<<(unsigned)(nelem * rep), 256, 0, s>>>(w, rep, d, amax,
                                                                  scan.as<int>());
    KFB_CUDA_TRY(cudaGetLastError());
    std::vector<int> host(words), cols;
    KFB_CUDA_TRY(cudaMemcpyAsync(host.data(), scan.ptr, words * sizeof(int),
                                 cudaMemcpyDeviceToHost, s));
    KFB_CUDA_TRY(cudaStreamSynchronize(s));
    std::vector<float> mx(words - rep);
    std::memcpy(mx.data(), host.data() + rep, mx.size() * sizeof(float));
    for (int e = 0; e < nelem; ++e) pl.w_scale.push_back(pow2_for(mx[e]));
    for (int k = 0; k < nslot; ++k) {
        pl.x_scale.push_back(pow2_for(mx[nelem + 2 * k]));
        pl.dx_scale.push_back(pow2_for(mx[nelem + 2 * k + 1]));
    }
    for (int k = 0; k < rep; ++k)
        if (host[k]) cols.push_back(k);
    pl.n = (int)cols.size();
    pl.kpad = std::max(16, (pl.n + 15) / 16 * 16);
    cols.resize(std::max<size_t>(cols.size(), 1));
    KFB_TRY(upload(pl.cols, cols, s));
    KFB_TRY(pl.err.alloc(sizeof(int), s));
    KFB_TRY(zero(pl.err.ptr, sizeof(int), s));
    KFB_TRY(pl.wh.alloc((size_t)d * pl.kpad * sizeof(__half), s));
    KFB_TRY(pl.wl.alloc((size_t)d * pl.kpad * sizeof(__half), s));
    return KFB_OK;
}

// W_e as rows of features (B operand of the products)
kfb_status rff_weights(const RffPlan &pl, const float *w, int rep, int e, int d, TcOperand &B,
                       cudaStream_t s) {
    rff_w_rows_kernel<<<dim3(nblk(d, 32), nblk(pl.kpad, 32)), dim3(32, 8), 0, s>>>(
        w + (size_t)e * rep * d, d, pl.cols.as<int>(), pl.n, pl.kpad, pl.w_scale[e],
        pl.wh.as<__half>(), pl.wl.as<__half>());
    KFB_CUDA_TRY(cudaGetLastError());
    B.hi = pl.wh.ptr;
    B.lo = pl.wl.ptr;
    B.rows = d;
    B.cols = pl.kpad;
    return KFB_OK;
}

// Descriptor rows idx[0 .. nr) (device) of a slot as the A operand
template <class T>
kfb_status rff_rows(RffPlan &pl, const T *x, const int *idx, int nr, int rep, int slot,
                    TcOperand &A, cudaStream_t s) {
    rff_x_rows_kernel<T><<<nblk((long long)nr * pl.kpad, 256 * 8), 256, 0, s>>>(
        x, idx, nr, rep, pl.cols.as<int>(), pl.n, pl.kpad, pl.x_scale[slot],
        pl.xh.as<__half>(), pl.xl.as<__half>());
    KFB_CUDA_TRY(cudaGetLastError());
    A.hi = pl.xh.ptr;
    A.lo = pl.xl.ptr;
    A.rows = nr;
    A.cols = pl.kpad;
    return KFB_OK;
}

kfb_status rff_done(const RffPlan &pl, cudaStream_t s) {
    int herr = 0;
    KFB_CUDA_TRY(cudaMemcpyAsync(&herr, pl.err.ptr, sizeof(int), cudaMemcpyDeviceToHost, s));
    KFB_CUDA_TRY(cudaStreamSynchronize(s));
    if (herr) return set_error(KFB_ERR_TIMEOUT, "RFF features: a tensor-core pipeline wait timed out");
    return KFB_OK;
}

template <class T>
kfb_status rff_features_t(const T *x, const int *q, const int *n, int nm, int ma, int rep,
                          const float *w, const float *b, int nelem, int d, float *z,
                          cudaStream_t s) {
    KFB_TRY(zero(z, (size_t)nm * d * sizeof(float), s));
    RffPlan pl;
    // (before the used columns are known: full rows)
    const size_t row_bytes = (size_t)(rep + 15) / 16 * 16 * 4 * sizeof(__half);
    const int chunk = (int)std::min<size_t>(1 << 30, std::max<size_t>(128, feature_budget() / row_bytes));
    KFB_TRY(rff_plan<T>(x, nullptr, q, n, nm, ma, rep, w, nelem, d, chunk, pl, s));
    // rows and molecules of every element, one upload
    std::vector<int> rows;
    int most = 1;
    for (int e = 0; e < nelem; ++e) {
        rows.insert(rows.end(), pl.er.idx[e].begin(), pl.er.idx[e].end());
        rows.insert(rows.end(), pl.er.mol[e].begin(), pl.er.mol[e].end());
        most = std::max(most, std::min(chunk, (int)pl.er.idx[e].size()));
    }
    if (rows.empty()) return KFB_OK;
    DevBuf drows;
    KFB_TRY(upload(drows, rows, s));
    KFB_TRY(pl.xh.alloc((size_t)most * pl.kpad * sizeof(__half), s));
    KFB_TRY(pl.xl.alloc((size_t)most * pl.kpad * sizeof(__half), s));
    const float sc = std::sqrt(2.f / (float)d);
    const int *idx = drows.as<int>();
    for (int e = 0; e < nelem; ++e) {
        const int ne = (int)pl.er.idx[e].size();
        if (ne == 0) continue;
        TcOperand A, B;
        KFB_TRY(rff_weights(pl, w, rep, e, d, B, s));
        for (int r0 = 0; r0 < ne; r0 += chunk) {
            const int nr = std::min(chunk, ne - r0);
            const int slot = pl.slot(e, r0);
            KFB_TRY(rff_rows<T>(pl, x, idx + r0, nr, rep, slot, A, s));
            TcProb p{};
            p.M = nr;
            p.N = d;
            p.K = pl.kpad;
            p.alpha = 1.0 / ((double)pl.x_scale[slot] * (double)pl.w_scale[e]);
            TcEpi epi;
            epi.mode = EPI_COS_MOLSUM;
            epi.bias = b + (size_t)e * d;
            epi.mol = idx + ne + r0;
            epi.molsum = z;
            epi.ld = d;
            epi.scale = sc;
            KFB_TRY(tc_gemm_grouped(A, B, 3, false, {p}, ElemSink(), s, epi, pl.err.as<int>()));
        }
        idx += 2 * (size_t)ne;
    }
    return rff_done(pl, s);
}

// G (naq, d) += rows 3 off_m + c: sqrt(2/d) sum_j sin(z_j) (W_e^T dX[m, j, :, c]), z_j the
// pre-activation x_j W_e + b_e (src/rff_elemental.cpp:363-500 stores the transpose).
template <class T>
kfb_status rff_gradient_t(const T *x, const T *dx, const int *q, const int *n, int nm, int ma,
                          int rep, const float *w, const float *b, int nelem, int d, float *g,
                          cudaStream_t s) {
    std::vector<int> offs(nm + 1, 0);
    for (int m = 0; m < nm; ++m) offs[m + 1] = offs[m] + 3 * std::min(std::max(n[m], 0), ma);
    KFB_TRY(zero(g, (size_t)std::max(offs[nm], 1) * d * sizeof(float), s));
    RffPlan pl;
    const int ld = 3 * ma;
    // per atom: one row of d sines, one descriptor and up to 3 ma Jacobian rows
    // (full ones: the used columns are not known yet)
    const size_t atom_bytes = (size_t)d * sizeof(float) +
                              (size_t)(1 + ld) * ((rep + 15) / 16 * 16) * 4 * sizeof(__half);
    const int chunk = (int)std::min<size_t>((size_t)(1 << 30) / ld,
                                            std::max<size_t>(1, feature_budget() / atom_bytes));
    KFB_TRY(rff_plan<T>(x, dx, q, n, nm, ma, rep, w, nelem, d, chunk, pl, s));
    const int kpad = pl.kpad;
    // every element's atoms: descriptor row, then its Jacobian rows, ordered
    // (molecule, c, atom) inside a chunk so that one destination is one run
    std::vector<RffAtom> atoms;
    std::vector<int> idx;
    struct Chunk {
        int e, a0, na, nr, slot;
    };
    std::vector<Chunk> chunks;
    int most_a = 1, most_r = 1;
    for (int e = 0; e < nelem; ++e) {
        const std::vector<int> &ai = pl.er.idx[e], &am = pl.er.mol[e];
        for (int a0 = 0; a0 < (int)ai.size(); a0 += chunk) {
            const int na = std::min<int>(chunk, (int)ai.size() - a0);
            Chunk ck{e, (int)atoms.size(), na, 0, pl.slot(e, a0)};
            int row = 0;
            for (int t = 0; t < na;) {
                const int m = am[a0 + t];
                int t1 = t;
                while (t1 < na && am[a0 + t1] == m) ++t1;
                const int nc = offs[m + 1] - offs[m];
                for (int u = t; u < t1; ++u) {
                    atoms.push_back({ai[a0 + u], row + (u - t), t1 - t, nc, offs[m]});
                    idx.push_back(ai[a0 + u]);
                }
                row += nc * (t1 - t);
                t = t1;
            }
            ck.nr = row;
            chunks.push_back(ck);
            most_a = std::max(most_a, na);
            most_r = std::max(most_r, row);
        }
    }
    if (atoms.empty()) return KFB_OK;
    DevBuf datoms, didx, sines, jh, jl, ddst, daux;
    KFB_TRY(upload(datoms, atoms, s));
    KFB_TRY(upload(didx, idx, s));
    KFB_TRY(pl.xh.alloc((size_t)most_a * kpad * sizeof(__half), s));
    KFB_TRY(pl.xl.alloc((size_t)most_a * kpad * sizeof(__half), s));
    KFB_TRY(sines.alloc((size_t)most_a * d * sizeof(float), s));
    KFB_TRY(jh.alloc((size_t)most_r * kpad * sizeof(__half), s));
    KFB_TRY(jl.alloc((size_t)most_r * kpad * sizeof(__half), s));
    KFB_TRY(ddst.alloc((size_t)most_r * sizeof(int), s));
    KFB_TRY(daux.alloc((size_t)most_r * sizeof(int), s));
    const float sc = std::sqrt(2.f / (float)d);
    int elem = -1;
    TcOperand A, B;
    for (const Chunk &ck : chunks) {
        if (ck.e != elem) KFB_TRY(rff_weights(pl, w, rep, ck.e, d, B, s));
        elem = ck.e;
        // sqrt(2/d) sin(x W_e + b_e) of the chunk's atoms: once per atom and
        // feature, not once per Jacobian row (63 of a 21-atom molecule)
        KFB_TRY(rff_rows<T>(pl, x, didx.as<int>() + ck.a0, ck.na, rep, ck.slot, A, s));
        TcProb p{};
        p.M = ck.na;
        p.N = d;
        p.K = kpad;
        p.alpha = 1.0 / ((double)pl.x_scale[ck.slot] * (double)pl.w_scale[ck.e]);
        TcEpi epi;
        epi.mode = EPI_DENSE;
        epi.zf32 = sines.as<float>();
        epi.zsin = 1;
        epi.scale = sc;
        epi.bias = b + (size_t)ck.e * d;
        epi.ld = d;
        KFB_TRY(tc_gemm_grouped(A, B, 3, false, {p}, ElemSink(), s, epi, pl.err.as<int>()));
        // Jacobian rows times W_e, weighted by the sines and summed into G per
        // destination row
        rff_jacobian_rows_kernel<T><<<dim3(ck.na, nblk(kpad, 64), nblk(ld, 32)), 256, 0, s>>>(
            dx, datoms.as<RffAtom>() + ck.a0, rep, ld, pl.cols.as<int>(), pl.n, kpad,
            pl.dx_scale[ck.slot], jh.as<__half>(), jl.as<__half>(), ddst.as<int>(), daux.as<int>());
        KFB_CUDA_TRY(cudaGetLastError());
        A.hi = jh.ptr;
        A.lo = jl.ptr;
        A.rows = ck.nr;
        A.cols = kpad;
        TcProb pj{};
        pj.M = ck.nr;
        pj.N = d;
        pj.K = kpad;
        pj.alpha = 1.0 / ((double)pl.dx_scale[ck.slot] * (double)pl.w_scale[ck.e]);
        TcEpi ej;
        ej.mode = EPI_ROW_RUNSUM;
        ej.mol = ddst.as<int>();
        ej.atom = daux.as<int>();
        ej.aux = sines.as<float>();
        ej.ld_aux = d;
        ej.molsum = g;
        ej.ld = d;
        KFB_TRY(tc_gemm_grouped(A, B, 3, false, {pj}, ElemSink(), s, ej, pl.err.as<int>()));
    }
    return rff_done(pl, s);
}

kfb_status check_cosmlp(const kfb_cosmlp *h) {
    if (!h) return set_error(KFB_ERR_INVALID_ARG, "null cos-MLP handle");
    int dev = 0;
    KFB_CUDA_TRY(cudaGetDevice(&dev));
    if (dev != h->device)
        return set_error(KFB_ERR_INVALID_ARG, "cos-MLP handle belongs to device %d, current is %d",
                         h->device, dev);
    return KFB_OK;
}

template <class T>
kfb_status cosmlp_features_t(kfb_cosmlp *h, const T *x, const int *q, const int *n, int nm,
                             int ma, float *z, cudaStream_t s) {
    const int rep = h->rep, H = h->hidden, D = h->d;
    KFB_TRY(zero(z, (size_t)nm * D * sizeof(float), s));
    ElemRows er;
    KFB_TRY(elem_rows(q, n, nm, ma, h->nelem, er));
    const size_t row_bytes = (size_t)(rep + H) * sizeof(bf16);
    const int chunk = (int)std::max<size_t>(128, feature_budget() / row_bytes);
    DevBuf xb, hb, didx, dmol;
    const float sc = std::sqrt(2.f / (float)D);
    for (int e = 0; e < h->nelem; ++e) {
        const int ne = (int)er.idx[e].size();
        if (ne == 0) continue;
        KFB_TRY(upload(didx, er.idx[e], s));
        KFB_TRY(upload(dmol, er.mol[e], s));
        const int rows_max = std::min(ne, chunk);
        KFB_TRY(xb.alloc((size_t)rows_max * rep * sizeof(bf16), s));
        KFB_TRY(hb.alloc((size_t)rows_max * H * sizeof(bf16), s));
        for (int r0 = 0; r0 < ne; r0 += chunk) {
            const int nr = std::min(chunk, ne - r0);
            gather_rows_bf16_kernel<T><<<dim3(nblk(rep, 32), nblk(nr, 32)), dim3(32, 8), 0, s>>>(
                x, (long long)nm * ma, didx.as<int>() + r0, nullptr, 0, nr, rep, xb.as<bf16>(),
                nullptr, 0, nullptr);
            KFB_CUDA_TRY(cudaGetLastError());
            TcOperand A, B;
            A.hi = xb.ptr;
            A.rows = nr;
            A.cols = rep;
            B.hi = h->w1b.ptr;
            B.rows = (long long)h->nelem * H;
            B.cols = rep;
            TcProb p{};
            p.b_row0 = e * H;
            p.M = nr;
            p.N = H;
            p.K = rep;
            p.alpha = 1.0;
            TcEpi e1;
            e1.mode = EPI_DENSE;
            e1.bias = h->b1.as<float>() + (size_t)e * H;
            e1.act = hb.as<bf16>();
            e1.ld = H;
            KFB_TRY(tc_gemm_grouped(A, B, 1, true, {p}, ElemSink(), s, e1));
            TcOperand A2, B2;
            A2.hi = hb.ptr;
            A2.rows = nr;
            A2.cols = H;
            B2.hi = h->w2b.ptr;
            B2.rows = (long long)h->nelem * D;
            B2.cols = H;
            TcProb p2{};
            p2.b_row0 = e * D;
            p2.M = nr;
            p2.N = D;
            p2.K = H;
            p2.alpha = 1.0;
            TcEpi e2;
            e2.mode = EPI_COS_MOLSUM;
            e2.bias = h->b2.as<float>() + (size_t)e * D;
            e2.mol = dmol.as<int>() + r0;
            e2.molsum = z;
            e2.ld = D;
            e2.scale = sc;
            KFB_TRY(tc_gemm_grouped(A2, B2, 1, true, {p2}, ElemSink(), s, e2));
        }
    }
    return KFB_OK;
}

template <class T>
kfb_status cosmlp_step_t(kfb_cosmlp *h, int e, const T *x, long long nrows, const int *pi,
                         const int *pj, const float *target, int npairs, float lr, int update,
                         double *loss_out, cudaStream_t s) {
    const int rep = h->rep, H = h->hidden, D = h->d;
    const int Bp = (int)ru8(npairs);
    const int R = 2 * Bp;  // batch rows: i-atoms then j-atoms
    int *err = h->err.as<int>(), *bad = err + 1;
    KFB_TRY(zero(err, 2 * sizeof(int), s));
    KFB_TRY(zero(h->loss.ptr, sizeof(double), s));
    // batch rows: pi, padding, pj, padding
    gather_rows_bf16_kernel<T><<<dim3(nblk(rep, 32), nblk(R, 32)), dim3(32, 8), 0, s>>>(
        x, nrows, pi, pj, npairs, R, rep, h->xb.as<bf16>(), h->xbt.as<bf16>(), R, bad);
    KFB_CUDA_TRY(cudaGetLastError());
    // forward, layer 1: z1 = X W1^T + b1, h = cos z1 (rows and transposed)
    {
        TcOperand A, B;
        A.hi = h->xb.ptr;
        A.rows = R;
        A.cols = rep;
        B.hi = h->w1b.ptr;
        B.rows = (long long)h->nelem * H;
        B.cols = rep;
        TcProb p{};
        p.b_row0 = e * H;
        p.M = R;
        p.N = H;
        p.K = rep;
        p.alpha = 1.0;
        TcEpi ep;
        ep.mode = EPI_DENSE;
        ep.bias = h->b1.as<float>() + (size_t)e * H;
        ep.zf32 = h->z1.as<float>();
        ep.act = h->hb.as<bf16>();
        ep.act_t = h->hbt.as<bf16>();
        ep.ld = H;
        ep.ld_t = R;
        KFB_TRY(tc_gemm_grouped(A, B, 1, true, {p}, ElemSink(), s, ep, err));
    }
    // forward, layer 2: z2 = h W2^T + b2
    {
        TcOperand A, B;
        A.hi = h->hb.ptr;
        A.rows = R;
        A.cols = H;
        B.hi = h->w2b.ptr;
        B.rows = (long long)h->nelem * D;
        B.cols = H;
        TcProb p{};
        p.b_row0 = e * D;
        p.M = R;
        p.N = D;
        p.K = H;
        p.alpha = 1.0;
        TcEpi ep;
        ep.mode = EPI_DENSE;
        ep.bias = h->b2.as<float>() + (size_t)e * D;
        ep.zf32 = h->z2.as<float>();
        ep.ld = D;
        KFB_TRY(tc_gemm_grouped(A, B, 1, true, {p}, ElemSink(), s, ep, err));
    }
    float *gw1 = h->grad[0].as<float>(), *gb1 = h->grad[1].as<float>();
    float *gw2 = h->grad[2].as<float>(), *gb2 = h->grad[3].as<float>();
    KFB_TRY(zero(gb2, (size_t)D * sizeof(float), s));
    pair_dot_kernel<<<nblk(Bp, 8), 256, 0, s>>>(h->z2.as<float>(), Bp, npairs, D, target,
                                                2.f / (float)D, 2.f / (float)npairs,
                                                h->factor.as<float>(), h->loss.as<double>());
    pair_grad_kernel<<<dim3(nblk(D, PG_T), nblk(Bp, PG_T)), 256, 0, s>>>(
        h->z2.as<float>(), Bp, npairs, D, h->factor.as<float>(), h->dz2.as<bf16>(),
        h->dz2t.as<bf16>(), gb2);
    KFB_CUDA_TRY(cudaGetLastError());
    // dW2 = dZ2^T H  (D x H, contraction over the batch rows)
    {
        TcOperand A, B;
        A.hi = h->dz2t.ptr;
        A.rows = D;
        A.cols = R;
        B.hi = h->hbt.ptr;
        B.rows = H;
        B.cols = R;
        TcProb p{};
        p.M = D;
        p.N = H;
        p.K = R;
        p.alpha = 1.0;
        TcEpi ep;
        ep.mode = EPI_DENSE;
        ep.zf32 = gw2;
        ep.ld = H;
        KFB_TRY(tc_gemm_grouped(A, B, 1, true, {p}, ElemSink(), s, ep, err));
    }
    // dZ1 = (dZ2 W2) * -sin z1, written transposed (H x R)
    {
        TcOperand A, B;
        A.hi = h->dz2.ptr;
        A.rows = R;
        A.cols = D;
        B.hi = h->w2tb.ptr;
        B.rows = (long long)h->nelem * H;
        B.cols = D;
        TcProb p{};
        p.b_row0 = e * H;
        p.M = R;
        p.N = H;
        p.K = D;
        p.alpha = 1.0;
        TcEpi ep;
        ep.mode = EPI_DSIN_T;
        ep.aux = h->z1.as<float>();
        ep.ld = H;
        ep.act_t = h->dz1t.as<bf16>();
        ep.ld_t = R;
        KFB_TRY(tc_gemm_grouped(A, B, 1, true, {p}, ElemSink(), s, ep, err));
    }
    // dW1 = dZ1^T X  (H x rep): few output tiles, so the batch axis (K) is
    // split over problems that add into a zeroed gradient
    {
        TcOperand A, B;
        A.hi = h->dz1t.ptr;
        A.rows = H;
        A.cols = R;
        B.hi = h->xbt.ptr;
        B.rows = rep;
        B.cols = R;
        const int tiles = ((H + 127) / 128) * ((rep + 127) / 128);
        const int want = std::max(1, std::min(device_sm_count() / std::max(tiles, 1), R / 256));
        const int kc = (int)((R / want + 63) / 64 * 64);
        std::vector<TcProb> probs;
        for (int k0 = 0; k0 < R; k0 += kc) {
            TcProb p{};
            p.a_k0 = p.b_k0 = k0;
            p.M = H;
            p.N = rep;
            p.K = std::min(kc, R - k0);
            p.alpha = 1.0;
            probs.push_back(p);
        }
        TcEpi ep;
        ep.mode = EPI_DENSE;
        ep.zf32 = gw1;
        ep.ld = rep;
        ep.accumulate = probs.size() > 1 ? 1 : 0;
        if (ep.accumulate) KFB_TRY(zero(gw1, (size_t)H * rep * sizeof(float), s));
        KFB_TRY(tc_gemm_grouped(A, B, 1, true, probs, ElemSink(), s, ep, err));
    }
    rowsum_bf16_kernel<<<H, 256, 0, s>>>(h->dz1t.as<bf16>(), H, R, gb1);
    KFB_CUDA_TRY(cudaGetLastError());
    if (update) {
        const int t = ++h->steps[e];
        const float bc1 = 1.f - std::pow(ADAM_B1, (float)t);
        const float bc2 = 1.f - std::pow(ADAM_B2, (float)t);
        struct P {
            DevBuf *p;
            int k, rows, cols;
            bf16 *pb, *pbt;
        };
        const P ps[4] = {
            {&h->w1, 0, H, rep, h->w1b.as<bf16>() + (size_t)e * H * rep, nullptr},
            {&h->b1, 1, 1, H, nullptr, nullptr},
            {&h->w2, 2, D, H, h->w2b.as<bf16>() + (size_t)e * D * H,
             h->w2tb.as<bf16>() + (size_t)e * H * D},
            {&h->b2, 3, 1, D, nullptr, nullptr},
        };
        AdamSet as{};
        for (int k = 0; k < 4; ++k) {
            const P &q = ps[k];
            const size_t off = (size_t)e * q.rows * q.cols;
            as.n[k] = (long long)q.rows * q.cols;
            as.p[k] = q.p->as<float>() + off;
            as.g[k] = h->grad[q.k].as<float>();
            as.m[k] = h->mom[q.k].as<float>() + off;
            as.v[k] = h->var[q.k].as<float>() + off;
            as.pb[k] = q.pb;
            as.first[k + 1] = as.first[k] + (int)nblk(as.n[k], 256 * 4);
        }
        adam_kernel<<<as.first[4], 256, 0, s>>>(as, lr, bc1, bc2);
        KFB_CUDA_TRY(cudaGetLastError());
        for (const P &q : ps)
            if (q.pbt) KFB_TRY(transpose_bf16(q.pb, q.rows, q.cols, q.pbt, q.rows, s));
    }
    int herr[2] = {0, 0};
    double lsum = 0.0;
    KFB_CUDA_TRY(cudaMemcpyAsync(herr, err, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
    KFB_CUDA_TRY(cudaMemcpyAsync(&lsum, h->loss.ptr, sizeof(double), cudaMemcpyDeviceToHost, s));
    KFB_CUDA_TRY(cudaStreamSynchronize(s));
    if (herr[0]) return set_error(KFB_ERR_TIMEOUT, "cos-MLP step: a tensor-core pipeline wait timed out");
    if (herr[1])
        return set_error(KFB_ERR_INVALID_ARG,
                         "cos-MLP step: a pair index is outside the %lld rows of x (the step "
                         "used zero rows for it; parameters were %s)",
                         nrows, update ? "updated" : "not updated");
    if (loss_out) *loss_out = lsum / std::max(npairs, 1);
    return KFB_OK;
}

}  // namespace

}  // namespace kfb

using namespace kfb;

namespace {
// Host allocations (std::vector) may throw; no exception crosses the C ABI.
template <class F>
kfb_status guarded(F &&f) {
    try {
        return f();
    } catch (const std::exception &ex) {
        return set_error(KFB_ERR_ALLOC, "host exception: %s", ex.what());
    }
}
}  // namespace

extern "C" {

kfb_status kfb_rff_features_elemental(const void *x, const int *q, const int *n, int nm, int ma,
                                      int rep, const float *w, const float *b, int nelem, int d,
                                      kfb_dtype x_dtype, float *z, void *stream) {
    return guarded([&]() -> kfb_status {
        if (!x || !q || !n || !w || !b || !z)
            return set_error(KFB_ERR_INVALID_ARG, "null pointer argument");
        if (nm <= 0 || ma <= 0 || rep <= 0 || nelem <= 0 || d <= 0)
            return set_error(KFB_ERR_INVALID_ARG, "All dims must be positive.");
        if (d % 8 != 0)
            return set_error(KFB_ERR_UNSUPPORTED,
                             "rff_features_elemental: D must be a multiple of 8");
        if (!device_is_sm100())
            return set_error(KFB_ERR_UNSUPPORTED, "feature maps need an sm_100 (B200) device");
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        if (x_dtype == KFB_F64)
            return rff_features_t<double>(static_cast<const double *>(x), q, n, nm, ma, rep, w,
                                          b, nelem, d, z, s);
        return rff_features_t<float>(static_cast<const float *>(x), q, n, nm, ma, rep, w, b,
                                     nelem, d, z, s);
    });
}

kfb_status kfb_rff_gradient_elemental(const void *x, const void *dx, const int *q, const int *n,
                                      int nm, int ma, int rep, const float *w, const float *b,
                                      int nelem, int d, kfb_dtype x_dt, float *g, void *stream) {
    return guarded([&]() -> kfb_status {
        if (!x || !dx || !q || !n || !w || !b || !g)
            return set_error(KFB_ERR_INVALID_ARG, "null pointer");
        if (nm <= 0 || ma <= 0 || rep <= 0 || nelem <= 0 || d <= 0)
            return set_error(KFB_ERR_INVALID_ARG, "dimensions must be positive");
        if (d % 8 != 0) return set_error(KFB_ERR_INVALID_ARG, "D must be a multiple of 8");
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        if (x_dt == KFB_F64)
            return rff_gradient_t<double>(static_cast<const double *>(x),
                                          static_cast<const double *>(dx), q, n, nm, ma, rep, w,
                                          b, nelem, d, g, s);
        return rff_gradient_t<float>(static_cast<const float *>(x), static_cast<const float *>(dx),
                                     q, n, nm, ma, rep, w, b, nelem, d, g, s);
    });
}

kfb_status kfb_pair_gaussian(const void *x, long long nrows, const int *pi, const int *pj,
                             int npairs, int rep, double sigma, kfb_dtype x_dtype, float *out,
                             void *stream) {
    if (!x || !pi || !pj || !out) return set_error(KFB_ERR_INVALID_ARG, "null pointer argument");
    if (npairs < 0 || rep <= 0 || nrows <= 0)
        return set_error(KFB_ERR_INVALID_ARG, "All dims must be positive.");
    if (!(sigma > 0)) return set_error(KFB_ERR_INVALID_ARG, "sigma must be > 0");
    if (npairs == 0) return KFB_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    DevBuf bad;
    KFB_TRY(bad.alloc(sizeof(int), s));
    KFB_TRY(zero(bad.ptr, sizeof(int), s));
    const double c = -1.0 / (2.0 * sigma * sigma);
    if (x_dtype == KFB_F64)
        pair_gaussian_kernel<double><<<nblk(npairs, 8), 256, 0, s>>>(
            static_cast<const double *>(x), nrows, pi, pj, npairs, rep, c, out, bad.as<int>());
    else
        pair_gaussian_kernel<float><<<nblk(npairs, 8), 256, 0, s>>>(
            static_cast<const float *>(x), nrows, pi, pj, npairs, rep, c, out, bad.as<int>());
    KFB_CUDA_TRY(cudaGetLastError());
    int hb = 0;
    KFB_CUDA_TRY(cudaMemcpyAsync(&hb, bad.ptr, sizeof(int), cudaMemcpyDeviceToHost, s));
    KFB_CUDA_TRY(cudaStreamSynchronize(s));
    if (hb)
        return set_error(KFB_ERR_INVALID_ARG,
                         "pair_gaussian: a pair index is outside the %lld rows of x", nrows);
    return KFB_OK;
}

kfb_status kfb_cosmlp_create(int nelem, int rep, int hidden, int d, int max_pairs,
                             kfb_cosmlp **out) {
    return guarded([&]() -> kfb_status {
        if (!out) return set_error(KFB_ERR_INVALID_ARG, "null output handle pointer");
        *out = nullptr;
        if (nelem <= 0 || rep <= 0 || hidden <= 0 || d <= 0 || max_pairs <= 0)
            return set_error(KFB_ERR_INVALID_ARG, "All dims must be positive.");
        if (rep % 16 != 0 || hidden % 16 != 0 || d % 16 != 0)
            return set_error(KFB_ERR_UNSUPPORTED,
                             "cos-MLP: rep, hidden and D must be multiples of 16");
        if (d > PL_MAX_D)
            return set_error(KFB_ERR_UNSUPPORTED, "cos-MLP: D up to %d", PL_MAX_D);
        if (!device_is_sm100())
            return set_error(KFB_ERR_UNSUPPORTED, "cos-MLP needs an sm_100 (B200) device");
        auto *h = new kfb_cosmlp();
        h->nelem = nelem;
        h->rep = rep;
        h->hidden = hidden;
        h->d = d;
        h->max_pairs = max_pairs;
        h->steps.assign(nelem, 0);
        kfb_status st = KFB_OK;
        auto fail = [&](kfb_status v) {
            delete h;
            return v;
        };
        if ((st = [&]() -> kfb_status {
                 KFB_CUDA_TRY(cudaGetDevice(&h->device));
                 cudaStream_t s = nullptr;
                 const size_t n1 = (size_t)nelem * hidden * rep, nb1 = (size_t)nelem * hidden;
                 const size_t n2 = (size_t)nelem * d * hidden, nb2 = (size_t)nelem * d;
                 const size_t sizes[4] = {n1, nb1, n2, nb2};
                 DevBuf *ps[4] = {&h->w1, &h->b1, &h->w2, &h->b2};
                 for (int k = 0; k < 4; ++k) {
                     KFB_TRY(ps[k]->alloc(sizes[k] * sizeof(float), s));
                     KFB_TRY(zero(ps[k]->ptr, sizes[k] * sizeof(float), s));
                     KFB_TRY(h->mom[k].alloc(sizes[k] * sizeof(float), s));
                     KFB_TRY(h->var[k].alloc(sizes[k] * sizeof(float), s));
                     KFB_TRY(zero(h->mom[k].ptr, sizes[k] * sizeof(float), s));
                     KFB_TRY(zero(h->var[k].ptr, sizes[k] * sizeof(float), s));
                     KFB_TRY(h->grad[k].alloc(sizes[k] / nelem * sizeof(float), s));
                 }
                 KFB_TRY(h->w1b.alloc(n1 * sizeof(bf16), s));
                 KFB_TRY(h->w2b.alloc(n2 * sizeof(bf16), s));
                 KFB_TRY(h->w2tb.alloc(n2 * sizeof(bf16), s));
                 const long long R = 2 * ru8(max_pairs);
                 KFB_TRY(h->xb.alloc((size_t)R * rep * sizeof(bf16), s));
                 KFB_TRY(h->xbt.alloc((size_t)R * rep * sizeof(bf16), s));
                 KFB_TRY(h->z1.alloc((size_t)R * hidden * sizeof(float), s));
                 KFB_TRY(h->hb.alloc((size_t)R * hidden * sizeof(bf16), s));
                 KFB_TRY(h->hbt.alloc((size_t)R * hidden * sizeof(bf16), s));
                 KFB_TRY(h->z2.alloc((size_t)R * d * sizeof(float), s));
                 KFB_TRY(h->factor.alloc((size_t)R / 2 * sizeof(float), s));
                 KFB_TRY(h->dz2.alloc((size_t)R * d * sizeof(bf16), s));
                 KFB_TRY(h->dz2t.alloc((size_t)R * d * sizeof(bf16), s));
                 KFB_TRY(h->dz1t.alloc((size_t)R * hidden * sizeof(bf16), s));
                 KFB_TRY(h->loss.alloc(sizeof(double), s));
                 KFB_TRY(h->err.alloc(2 * sizeof(int), s));
                 KFB_CUDA_TRY(cudaStreamSynchronize(s));
                 return KFB_OK;
             }()) != KFB_OK)
            return fail(st);
        *out = h;
        return KFB_OK;
    });
}

void kfb_cosmlp_destroy(kfb_cosmlp *h) {
    if (!h) return;
    cudaDeviceSynchronize();
    delete h;
}

kfb_status kfb_cosmlp_params(kfb_cosmlp *h, float **w1, float **b1, float **w2, float **b2) {
    KFB_TRY(check_cosmlp(h));
    if (w1) *w1 = h->w1.as<float>();
    if (b1) *b1 = h->b1.as<float>();
    if (w2) *w2 = h->w2.as<float>();
    if (b2) *b2 = h->b2.as<float>();
    return KFB_OK;
}

kfb_status kfb_cosmlp_grads(kfb_cosmlp *h, float **w1, float **b1, float **w2, float **b2) {
    KFB_TRY(check_cosmlp(h));
    if (w1) *w1 = h->grad[0].as<float>();
    if (b1) *b1 = h->grad[1].as<float>();
    if (w2) *w2 = h->grad[2].as<float>();
    if (b2) *b2 = h->grad[3].as<float>();
    return KFB_OK;
}

kfb_status kfb_cosmlp_sync(kfb_cosmlp *h, int reset_optimizer, void *stream) {
    KFB_TRY(check_cosmlp(h));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int H = h->hidden, D = h->d, rep = h->rep;
    for (int e = 0; e < h->nelem; ++e) {
        to_bf16_kernel<<<nblk((long long)H * rep, 1024), 256, 0, s>>>(
            h->w1.as<float>() + (size_t)e * H * rep, H, rep, h->w1b.as<bf16>() + (size_t)e * H * rep,
            nullptr);
        to_bf16_kernel<<<nblk((long long)D * H, 1024), 256, 0, s>>>(
            h->w2.as<float>() + (size_t)e * D * H, D, H, h->w2b.as<bf16>() + (size_t)e * D * H,
            nullptr);
        KFB_CUDA_TRY(cudaGetLastError());
        KFB_TRY(transpose_bf16(h->w2b.as<bf16>() + (size_t)e * D * H, D, H,
                               h->w2tb.as<bf16>() + (size_t)e * H * D, D, s));
    }
    if (reset_optimizer) {
        const size_t sizes[4] = {(size_t)h->nelem * H * rep, (size_t)h->nelem * H,
                                 (size_t)h->nelem * D * H, (size_t)h->nelem * D};
        for (int k = 0; k < 4; ++k) {
            KFB_TRY(zero(h->mom[k].ptr, sizes[k] * sizeof(float), s));
            KFB_TRY(zero(h->var[k].ptr, sizes[k] * sizeof(float), s));
        }
        std::fill(h->steps.begin(), h->steps.end(), 0);
    }
    return KFB_OK;
}

kfb_status kfb_cosmlp_optimizer_state(kfb_cosmlp *h, float **m, float **v, int *steps) {
    KFB_TRY(check_cosmlp(h));
    for (int k = 0; k < 4; ++k) {
        if (m) m[k] = h->mom[k].as<float>();
        if (v) v[k] = h->var[k].as<float>();
    }
    if (steps)
        for (int e = 0; e < h->nelem; ++e) steps[e] = h->steps[e];
    return KFB_OK;
}

kfb_status kfb_cosmlp_set_steps(kfb_cosmlp *h, const int *steps) {
    KFB_TRY(check_cosmlp(h));
    if (!steps) return set_error(KFB_ERR_INVALID_ARG, "null pointer argument");
    for (int e = 0; e < h->nelem; ++e) h->steps[e] = steps[e];
    return KFB_OK;
}

kfb_status kfb_cosmlp_pair_step(kfb_cosmlp *h, int elem, const void *x, long long nrows,
                                kfb_dtype x_dtype, const int *pi, const int *pj,
                                const float *target, int npairs, float lr, int update,
                                double *loss, void *stream) {
    return guarded([&]() -> kfb_status {
        KFB_TRY(check_cosmlp(h));
        if (!x || !pi || !pj || !target)
            return set_error(KFB_ERR_INVALID_ARG, "null pointer argument");
        if (elem < 0 || elem >= h->nelem)
            return set_error(KFB_ERR_INVALID_ARG, "element %d out of range [0, %d)", elem,
                             h->nelem);
        if (nrows <= 0) return set_error(KFB_ERR_INVALID_ARG, "All dims must be positive.");
        if (npairs <= 0 || npairs > h->max_pairs)
            return set_error(KFB_ERR_INVALID_ARG, "npairs = %d outside [1, %d]", npairs,
                             h->max_pairs);
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        if (x_dtype == KFB_F64)
            return cosmlp_step_t<double>(h, elem, static_cast<const double *>(x), nrows, pi, pj,
                                         target, npairs, lr, update, loss, s);
        return cosmlp_step_t<float>(h, elem, static_cast<const float *>(x), nrows, pi, pj, target,
                                    npairs, lr, update, loss, s);
    });
}

kfb_status kfb_cosmlp_features_elemental(kfb_cosmlp *h, const void *x, const int *q,
                                         const int *n, int nm, int ma, int rep, kfb_dtype x_dtype,
                                         float *z, void *stream) {
    return guarded([&]() -> kfb_status {
        KFB_TRY(check_cosmlp(h));
        if (!x || !q || !n || !z) return set_error(KFB_ERR_INVALID_ARG, "null pointer argument");
        if (nm <= 0 || ma <= 0) return set_error(KFB_ERR_INVALID_ARG, "All dims must be positive.");
        if (rep != h->rep)
            return set_error(KFB_ERR_INVALID_ARG, "rep = %d but the network takes %d", rep, h->rep);
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        if (x_dtype == KFB_F64)
            return cosmlp_features_t<double>(h, static_cast<const double *>(x), q, n, nm, ma, z, s);
        return cosmlp_features_t<float>(h, static_cast<const float *>(x), q, n, nm, ma, z, s);
    });
}

}  // extern "C"
