// Contracted energy / force prediction with the local FCHL19 kernels (the
// "J^T alpha" form of src/local_kernels.cpp:2821-3425: compute_alpha_desc
// :2821-2894, hessian_matvec :2895-3154, jacobian_t_matvec :3155-3262,
// full_matvec :3263-3425): predictions of a model
// trained on energies and forces without forming the (query x training) E+F
// kernel matrix.
//
// With d = x_i - x_j, e = exp(-|d|^2 / 2 sigma^2), w = e / sigma^2,
// w2 = e / sigma^4 over same-label pairs (i query, j training atom) and
// Ad_j = J_j alpha_F,b (compute_alpha_desc):
//   E_a     = sum_{i in a, j} alpha_E[b] e + w (d . Ad_j)
//   F_(a,c) = sum_{i in a} J_i[:, c] . g_i,
//   g_i     = sum_j w Ad_j + sum_j v_ij d,  v_ij = -w alpha_E[b] - w2 (d . Ad_j)
//           = W Ad + rowsum(V) x_i - V X2     (W_ij = w, V_ij = v_ij)
// Per label bucket: G = X1 X2^T and P = X1 Ad^T as FP64-class products on the
// int8 tensor cores (ozaki.h: 7 digit planes per operand, exact int32 level
// sums combined in FP64), one fused kernel for e, w, v, the energy sums and
// W, V (written over G, P), two more such products for g (contracting over the
// label's training atoms, in chunks of 65,536), and a contraction of g with
// each query atom's Jacobian.  Every product is oriented so that the rows of
// its first operand run along the output's contiguous dimension (coalesced
// epilogue stores).  Query rows are processed in chunks that keep the two
// (rows x training atoms) matrices within the workspace budget.

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <vector>

#include "kernels_common.cuh"
#include "ozaki.h"

namespace kfb {

namespace {

unsigned nblk(long long n, int t) { return (unsigned)std::max<long long>(1, (n + t - 1) / t); }

// Ad[b, j, :] = dX2[b, j] (rep x 3 n_b) . alpha[off_b : off_b + 3 n_b]; zero
// for padded atoms.  Block per (b, j), threads over k.
template <class Tin>
__global__ void alpha_desc_kernel(const Tin *__restrict__ dx2, const int *__restrict__ n2,
                                  const int *__restrict__ off2, int ma2, int rep,
                                  const double *__restrict__ alpha, double *__restrict__ ad) {
    const int b = blockIdx.y, j = blockIdx.x;
    const int nb = min(max(n2[b], 0), ma2);
    const int ld = 3 * ma2, nc = 3 * nb;
    const double *al = alpha + off2[b];
    double *out = ad + ((size_t)b * ma2 + j) * rep;
    const Tin *J = dx2 + ((size_t)b * ma2 + j) * rep * (size_t)ld;
    for (int k = threadIdx.x; k < rep; k += blockDim.x) {
        double acc = 0.0;
        if (j < nb)
            for (int c = 0; c < nc; ++c) acc = fma((double)J[(size_t)k * ld + c], al[c], acc);
        out[k] = acc;
    }
}

// out[r, :] = (double) src[idx[r], :] (rows of rep values), and |row|^2
template <class Tin>
__global__ void gather_f64_kernel(const Tin *__restrict__ src, const int *__restrict__ idx,
                                  int nrows, int rep, double *__restrict__ out,
                                  double *__restrict__ norm2) {
    const int r = blockIdx.x;
    if (r >= nrows) return;
    const Tin *row = src + (size_t)idx[r] * rep;
    double s = 0.0;
    for (int k = threadIdx.x; k < rep; k += blockDim.x) {
        const double v = (double)row[k];
        out[(size_t)r * rep + k] = v;
        s = fma(v, v, s);
    }
    __shared__ double red[32];
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0 && norm2) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
        norm2[r] = t;
    }
}

// sc[r] = x_r . Ad_r and aE[r] = alpha_E of atom idx[r]'s molecule (0 without
// alpha_E)
__global__ void train_scalars_kernel(const double *__restrict__ X, const double *__restrict__ Ad,
                                     const int *__restrict__ idx, int ma,
                                     const double *__restrict__ alpha_e, int nrows, int rep, double *__restrict__ sc,
                                     double *__restrict__ ae) {
    const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (r >= nrows) return;
    double s = 0.0;
    if (Ad)
        for (int k = lane; k < rep; k += 32) s = fma(X[(size_t)r * rep + k], Ad[(size_t)r * rep + k], s);
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
        sc[r] = s;
        ae[r] = alpha_e ? alpha_e[idx[r] / ma] : 0.0;
    }
}

// One block per query row i of the chunk: the Gaussian weights of all
// training atoms j of the label, the energy sum of row i (added to its
// molecule), and with forces W[i, j] = w, V[i, j] = v_ij (over G, P) and
// rowsum(V)[i].
__global__ void pair_weights_kernel(double *__restrict__ G, double *__restrict__ P, int r2,
                                    const double *__restrict__ n1, const double *__restrict__ n2,
                                    const double *__restrict__ sc, const double *__restrict__ ae,
                                    const int *__restrict__ idx1, int ma1, int with_ad,
                                    int with_f, double c, double is2, double is4, double *__restrict__ E,
                                    double *__restrict__ rowv) {
    const int i = blockIdx.x;
    double *Gi = G + (size_t)i * r2;
    double *Pi = P + (size_t)i * r2;
    const double ni = n1[i];
    double esum = 0.0, vsum = 0.0;
    for (int j = threadIdx.x; j < r2; j += blockDim.x) {
        const double d2 = fmax(ni + n2[j] - 2.0 * Gi[j], 0.0);
        const double e = exp(c * d2);
        const double w = e * is2;
        const double dad = with_ad ? Pi[j] - sc[j] : 0.0;
        esum += ae[j] * e + w * dad;
        if (with_f) {
            const double v = -w * ae[j] - e * is4 * dad;
            Gi[j] = w;
            Pi[j] = v;
            vsum += v;
        }
    }
    __shared__ double red[2][32];
    for (int o = 16; o; o >>= 1) {
        esum += __shfl_xor_sync(0xffffffffu, esum, o);
        vsum += __shfl_xor_sync(0xffffffffu, vsum, o);
    }
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = esum;
        red[1][threadIdx.x >> 5] = vsum;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double te = 0.0, tv = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            te += red[0][w];
            tv += red[1][w];
        }
        if (E) atomicAdd(E + idx1[i] / ma1, te);
        if (rowv) rowv[i] = tv;
    }
}

// g[i, :] += rowv[i] x1[i, :]
__global__ void add_row_scaled_kernel(const double *__restrict__ X1, const double *__restrict__ rowv,
                                      int rows, int rep, double *__restrict__ g) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e < (long long)rows * rep) g[e] += rowv[e / rep] * X1[e];
}

// F[off_a + c] += sum_k dX1[a, i, k, c] (g[r, k] + rowv[r] x1[a, i, k]) for the
// query rows r (molecule a, atom i) and the columns k of this block's slice
// (blockIdx.y); rowv null: g alone.  Lanes over c (64 at a time, coalesced
// along the Jacobian's rows), 4 columns k at once; the slices of a row fill
// the SMs that one block per row left idle for a few molecules.
constexpr int FC_K = 80;

template <class Tin>
__global__ void __launch_bounds__(256) force_contract_kernel(
    const Tin *__restrict__ x1, const Tin *__restrict__ dx1, const int *__restrict__ idx1,
    const int *__restrict__ n1, const int *__restrict__ off1, int ma1, int rep,
    const double *__restrict__ g, const double *__restrict__ rowv,
    double *__restrict__ F) {
    __shared__ double gs[FC_K], part[4][64];
    const int r = blockIdx.x, k0 = blockIdx.y * FC_K, nk = min(FC_K, rep - k0);
    const int flat = idx1[r], a = flat / ma1;
    const int na = min(max(n1[a], 0), ma1);
    const int ld = 3 * ma1, nc = 3 * na;
    const double rv = rowv ? rowv[r] : 0.0;
    for (int k = threadIdx.x; k < nk; k += 256) {
        const double gk = g[(size_t)r * rep + k0 + k];
        gs[k] = rowv ? fma(rv, (double)x1[(size_t)flat * rep + k0 + k], gk) : gk;
    }
    __syncthreads();
    const Tin *J = dx1 + ((size_t)flat * rep + k0) * (size_t)ld;
    const int cl = threadIdx.x & 63, kq = threadIdx.x >> 6;
    for (int c0 = 0; c0 < nc; c0 += 64) {
        const int cc = c0 + cl;
        double acc = 0.0;
        if (cc < nc) {
#pragma unroll 10
            for (int k = kq; k < nk; k += 4) acc = fma((double)J[(size_t)k * ld + cc], gs[k], acc);
        }
        part[kq][cl] = acc;
        __syncthreads();
        if (kq == 0 && cc < nc)
            atomicAdd(F + off1[a] + cc, part[0][cl] + part[1][cl] + part[2][cl] + part[3][cl]);
        __syncthreads();
    }
}

// ----------------------------------------------------- direct FP64 products
// Few (query, training) atom pairs: the digit planes of the training rows and
// of their transposes cost more than the products themselves, and a launch per
// label and product leaves most SMs idle.  Three kernels take every label at
// once: row sums, weights, gradient rows; the products are FP64 mma.sync.
// Columns are taken in groups of 8, and groups in which the training rows and
// their coefficients are all zero (the sulphur channels of molecules without
// sulphur: 28 of 90) add nothing to any product and are skipped.
//
// Label l: query rows [sa, sa + ra), training rows [sb, sb + rb), W and V of
// ra rows of ldw doubles from woff; blocks [tile1, next label's tile1) of the
// weights kernel and [tile2, ...) of the gradient kernel.
struct MvLabel {
    int sa, ra, sb, rb;
    int tile1, tile2, ldw, pad;
    long long woff;
};
constexpr int MD_M = 32, MD_N = 64, MD_K = 32;
constexpr int MD_LDK = MD_K + 4;   // row strides (elements): the fragment loads of a warp
                                   // (floats) or half warp (doubles) hit different banks
template <class Tin> constexpr int md_ldn() { return MD_N + (sizeof(Tin) == 4 ? 8 : 4); }

__device__ __forceinline__ void md_cp16(void *dst, const void *src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                     static_cast<unsigned>(__cvta_generic_to_shared(dst))),
                 "l"(src), "r"(ok ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void md_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void md_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// dst[0 .. 16 / sizeof(T)) = src[0 ..] (with vec 16-byte aligned, and an address of the array
// where !ok too), zeros where !ok and for columns from `left` on.
template <class T>
__device__ __forceinline__ void md_piece(T *dst, const T *src, bool ok, int left, bool vec) {
    if (vec) {
        md_cp16(dst, src, ok);
    } else {
#pragma unroll
        for (int u = 0; u < 16 / (int)sizeof(T); ++u) dst[u] = ok && u < left ? src[u] : T(0);
    }
}

// Warp per row.  Query rows r < R1: n1[r] = |x|^2 (-infinity for a row that holds an
// infinity, unlike one whose finite values have too large a sum).  Training rows: n2 = |x|^2,
// sc = x . Ad, and used[g] = 1 for the column groups with a value that is not
// zero.  Four columns a lane (vec: 16-byte loads, 128 columns of the warp in
// flight per step), so a group of 8 is two neighbouring lanes.
template <class Tin>
__global__ void __launch_bounds__(256) mv_rows_kernel(
    const Tin *__restrict__ x1, const int *__restrict__ idx1, int R1, const Tin *__restrict__ x2,
    const int *__restrict__ idx2, int R2, const double *__restrict__ ad, int rep, int vec,
    double *__restrict__ n1, double *__restrict__ n2, double *__restrict__ sc,
    int *__restrict__ used) {
    const int r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (r >= R1 + R2) return;
    const bool train = r >= R1;
    const size_t at = (size_t)(train ? idx2[r - R1] : idx1[r]) * rep;
    const Tin *x = (train ? x2 : x1) + at;
    const double *a = train && ad ? ad + at : nullptr;
    double n = 0.0, s = 0.0;
#pragma unroll 3
    for (int k0 = 0; k0 < rep; k0 += 128) {
        const int k = k0 + 4 * lane;
        double v[4] = {0.0, 0.0, 0.0, 0.0}, w[4] = {0.0, 0.0, 0.0, 0.0};
        if (vec && k < rep) {
            if constexpr (sizeof(Tin) == 4) {
                const float4 f = *reinterpret_cast<const float4 *>(x + k);
                v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
            } else {
                const double2 f = *reinterpret_cast<const double2 *>(x + k);
                const double2 h = *reinterpret_cast<const double2 *>(x + k + 2);
                v[0] = f.x; v[1] = f.y; v[2] = h.x; v[3] = h.y;
            }
            if (a) {
                const double2 f = *reinterpret_cast<const double2 *>(a + k);
                const double2 h = *reinterpret_cast<const double2 *>(a + k + 2);
                w[0] = f.x; w[1] = f.y; w[2] = h.x; w[3] = h.y;
            }
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (k + u < rep) {
                    v[u] = (double)x[k + u];
                    if (a) w[u] = a[k + u];
                }
        }
        bool on = false;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            n = fma(v[u], v[u], n);
            s = fma(v[u], w[u], s);
            on |= !(v[u] == 0.0) || !(w[u] == 0.0);
        }
        if (train && on && !used[k >> 3]) used[k >> 3] = 1;
    }
    for (int o = 16; o; o >>= 1) {
        n += __shfl_xor_sync(0xffffffffu, n, o);
        s += __shfl_xor_sync(0xffffffffu, s, o);
    }
    bool inf = false;
    if (!train && isinf(n)) {   // (warp-uniform; its values' sum or one of them)
        for (int k = lane; k < rep; k += 32) inf |= isinf((double)x[k]);
        inf = __any_sync(0xffffffffu, inf);
    }
    if (lane == 0) {
        if (train) {
            n2[r - R1] = n;
            sc[r - R1] = s;
        } else {
            n1[r] = inf ? -n : n;
        }
    }
}

// list = the used groups in order; returns their number (whole block; warp 0 works).
__device__ __forceinline__ int md_groups(const int *__restrict__ used, int ng, int *list,
                                         int *count) {
    if (threadIdx.x < 32) {
        int n = 0;
        for (int g0 = 0; g0 < ng; g0 += 32) {
            const int g = g0 + threadIdx.x;
            const bool on = g < ng && used[g] != 0;
            const unsigned m = __ballot_sync(0xffffffffu, on);
            if (on) list[n + __popc(m & ((1u << threadIdx.x) - 1u))] = g;
            n += __popc(m);
        }
        if (threadIdx.x == 0) *count = n;
    }
    __syncthreads();
    return *count;
}

// Stages of the weights kernel: x1 (MD_M rows), x2 (MD_N) and Ad (MD_N) of MD_K columns.
template <class Tin> struct MvW {
    static constexpr int NST = sizeof(Tin) == 4 ? 3 : 2;
    static constexpr int A = 0, X = MD_M * MD_LDK * (int)sizeof(Tin);
    static constexpr int D = X + MD_N * MD_LDK * (int)sizeof(Tin);
    static constexpr int STAGE = D + MD_N * MD_LDK * (int)sizeof(double);
};

// Tile of MD_M query rows x MD_N training rows of a label: G = x1 . x2 and
// P = x1 . Ad over the used columns, then e, w, v of every pair, the energy
// sums (E of the query row's molecule), and with forces W = w, V = -v and
// rowsum(V).  Warp (wm, wn) holds 16 x 16 of both products.
template <class Tin>
__global__ void __launch_bounds__(256, 2) mv_weights_kernel(
    const Tin *__restrict__ x1, const int *__restrict__ idx1, int ma1,
    const Tin *__restrict__ x2, const int *__restrict__ idx2, int ma2,
    const double *__restrict__ ad, const double *__restrict__ alpha_e,
    const MvLabel *__restrict__ labels, int nlab, int rep, int vec, int with_f, double c,
    double is2, double is4, const double *__restrict__ n1, const double *__restrict__ n2,
    const double *__restrict__ sc, const int *__restrict__ used, double *__restrict__ W,
    double *__restrict__ V, double *__restrict__ E, double *__restrict__ rowv) {
    using S = MvW<Tin>;
    extern __shared__ __align__(16) unsigned char md_raw[];
    int *list = reinterpret_cast<int *>(md_raw + S::NST * S::STAGE);   // [ng], then the count
    const int ng = (rep + 7) / 8;
    const int nused = md_groups(used, ng, list, list + ng);
    int l = 0;
    while (l + 1 < nlab && (int)blockIdx.x >= labels[l + 1].tile1) ++l;
    const MvLabel lb = labels[l];
    const int mt = (lb.ra + MD_M - 1) / MD_M;
    const int local = blockIdx.x - lb.tile1;
    const int i0 = (local % mt) * MD_M, j0 = (local / mt) * MD_N;
    const int na = min(MD_M, lb.ra - i0), nb = min(MD_N, lb.rb - j0);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    // staging, in 16-byte pieces: PT of a row of Tin, PD of a row of Ad
    constexpr int ET = 16 / sizeof(Tin), PT = MD_K / ET, PD = MD_K / 2;
    auto stage = [&](int s, int chunk) {
        unsigned char *base = md_raw + s * S::STAGE;
        Tin *As = reinterpret_cast<Tin *>(base + S::A), *Xs = reinterpret_cast<Tin *>(base + S::X);
        double *Ds = reinterpret_cast<double *>(base + S::D);
        auto column = [&](int at, bool &ok) {   // of column `at` of the chunk
            const int g = chunk * (MD_K / 8) + at / 8;
            ok = ok && g < nused;
            return g < nused ? list[g] * 8 + at % 8 : 0;
        };
        for (int e = t; e < MD_M * PT; e += 256) {
            const int r = e / PT, at = (e - r * PT) * ET;
            bool ok = r < na;
            const int k = column(at, ok);
            const Tin *row = x1 + (size_t)(r < na ? idx1[lb.sa + i0 + r] : 0) * rep;
            md_piece<Tin>(As + r * MD_LDK + at, row + k, ok, rep - k, vec);
        }
#pragma unroll
        for (int e = t; e < MD_N * PT; e += 256) {
            const int r = e / PT, at = (e - r * PT) * ET;
            bool ok = r < nb;
            const int k = column(at, ok);
            const Tin *row = x2 + (size_t)(r < nb ? idx2[lb.sb + j0 + r] : 0) * rep;
            md_piece<Tin>(Xs + r * MD_LDK + at, row + k, ok, rep - k, vec);
        }
        if (ad) {
#pragma unroll
            for (int e = t; e < MD_N * PD; e += 256) {
                const int r = e / PD, at = (e - r * PD) * 2;
                bool ok = r < nb;
                const int k = column(at, ok);
                const double *row = ad + (size_t)(r < nb ? idx2[lb.sb + j0 + r] : 0) * rep;
                md_piece<double>(Ds + r * MD_LDK + at, row + k, ok, rep - k, vec);
            }
        }
        md_commit();
    };
    const int wm = warp & 1, wn = warp >> 1;
    const bool active = 16 * wm < na;
    double g[2][2][2] = {}, p[2][2][2] = {};
    const int nch = (nused + MD_K / 8 - 1) / (MD_K / 8);
    for (int s = 0; s < S::NST - 1; ++s) {
        if (s < nch) stage(s, s);
        else md_commit();
    }
    for (int ch = 0; ch < nch; ++ch) {
        md_wait<S::NST - 2>();
        __syncthreads();   // the slice has landed, and the one before is read
        if (ch + S::NST - 1 < nch) stage((ch + S::NST - 1) % S::NST, ch + S::NST - 1);
        else md_commit();
        if (!active) continue;
        const unsigned char *base = md_raw + (ch % S::NST) * S::STAGE;
        const Tin *As = reinterpret_cast<const Tin *>(base + S::A);
        const Tin *Xs = reinterpret_cast<const Tin *>(base + S::X);
        const double *Ds = reinterpret_cast<const double *>(base + S::D);
        const int r = lane >> 2, kl = lane & 3;
#pragma unroll
        for (int kk = 0; kk < MD_K; kk += 4) {
            const int k = kk + kl;
            const double a0 = (double)As[(16 * wm + r) * MD_LDK + k];
            const double a1 = (double)As[(16 * wm + 8 + r) * MD_LDK + k];
#pragma unroll
            for (int nj = 0; nj < 2; ++nj) {
                const int row = (16 * wn + 8 * nj + r) * MD_LDK + k;
                const double x = (double)Xs[row];
                dmma(g[0][nj], a0, x);
                dmma(g[1][nj], a1, x);
                if (ad) {
                    const double d = Ds[row];
                    dmma(p[0][nj], a0, d);
                    dmma(p[1][nj], a1, d);
                }
            }
        }
    }
    md_wait<0>();
    __syncthreads();   // every warp is past its fragment loads
    double *es = reinterpret_cast<double *>(md_raw), *vs = es + 4 * MD_M;   // [wn][row] sums
    if (active) {
#pragma unroll
        for (int mi = 0; mi < 2; ++mi) {
            const int i = 16 * wm + 8 * mi + (lane >> 2);
            const double ni = i < na ? n1[lb.sa + i0 + i] : 0.0;
            const double bad = ni >= 0.0 ? 0.0 : ni - ni;   // NaN for a row that is not finite
            double esum = 0.0, vsum = 0.0;
#pragma unroll
            for (int nj = 0; nj < 2; ++nj) {
                const int j = 16 * wn + 8 * nj + 2 * (lane & 3);
                double w[2] = {0.0, 0.0}, v[2] = {0.0, 0.0};
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    if (i >= na || j + u >= nb) continue;
                    const int jr = lb.sb + j0 + j + u;
                    // (with a norm that is not finite the product need not be either)
                    const double nn = fabs(ni) + n2[jr];
                    const double e =
                        exp(c * (isfinite(nn) ? fmax(nn - 2.0 * g[mi][nj][u], 0.0) : nn));
                    const double dad = ad ? p[mi][nj][u] - sc[jr] + bad : 0.0;
                    const double ae = alpha_e ? alpha_e[idx2[jr] / ma2] : 0.0;
                    w[u] = e * is2;
                    v[u] = w[u] * ae + e * is4 * dad;
                    esum += ae * e + w[u] * dad;
                    vsum += v[u];
                }
                if (with_f && i < na && j < nb) {
                    // ldw is even and j too: 16-byte stores, the second value in the row's padding
                    const long long at = lb.woff + (long long)(i0 + i) * lb.ldw + j0 + j;
                    *reinterpret_cast<double2 *>(W + at) = make_double2(w[0], w[1]);
                    *reinterpret_cast<double2 *>(V + at) = make_double2(v[0], v[1]);
                }
            }
            for (int o = 2; o; o >>= 1) {
                esum += __shfl_xor_sync(0xffffffffu, esum, o);
                vsum += __shfl_xor_sync(0xffffffffu, vsum, o);
            }
            if ((lane & 3) == 0) {
                es[wn * MD_M + i] = esum;
                vs[wn * MD_M + i] = vsum;
            }
        }
    }
    __syncthreads();
    if (t < na) {
        double te = 0.0, tv = 0.0;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            te += es[w * MD_M + t];
            tv += vs[w * MD_M + t];
        }
        if (E) atomicAdd(E + idx1[lb.sa + i0 + t] / ma1, te);
        if (with_f) atomicAdd(rowv + lb.sa + i0 + t, -tv);
    }
}

// Stages of the gradient kernel: W and V (MD_M rows of MD_K partners), x2 and
// Ad (MD_K rows of MD_N columns).
template <class Tin> struct MvG {
    static constexpr int NST = 2, LDN = md_ldn<Tin>(), LDD = md_ldn<double>();
    static constexpr int W = 0, V = MD_M * MD_LDK * (int)sizeof(double);
    static constexpr int X = 2 * V, D = X + MD_K * LDN * (int)sizeof(Tin);
    static constexpr int STAGE = D + MD_K * LDD * (int)sizeof(double);
};

// g[i, k] += sum_j W_ij Ad_jk + (-v)_ij x2_jk over the training rows
// [split jlen, ...) of a label: MD_M query rows x MD_N used columns per block,
// the split-K sums combined by atomics.
template <class Tin>
__global__ void __launch_bounds__(256, 2) mv_grad_kernel(
    const Tin *__restrict__ x2, const int *__restrict__ idx2, const double *__restrict__ ad,
    const MvLabel *__restrict__ labels, int nlab, int rep, int jlen, int vec,
    const int *__restrict__ used, const double *__restrict__ W, const double *__restrict__ V,
    double *__restrict__ g) {
    using S = MvG<Tin>;
    extern __shared__ __align__(16) unsigned char md_raw[];
    int *list = reinterpret_cast<int *>(md_raw + S::NST * S::STAGE);
    const int ng = (rep + 7) / 8;
    const int nused = md_groups(used, ng, list, list + ng);
    int l = 0;
    while (l + 1 < nlab && (int)blockIdx.x >= labels[l + 1].tile2) ++l;
    const MvLabel lb = labels[l];
    const int mt = (lb.ra + MD_M - 1) / MD_M, nt = (rep + MD_N - 1) / MD_N;
    const int local = blockIdx.x - lb.tile2;
    const int i0 = (local % mt) * MD_M, g0 = (local / mt % nt) * (MD_N / 8);
    if (g0 >= nused) return;   // block-uniform
    const int jb = local / (mt * nt) * jlen, je = min(lb.rb, jb + jlen);
    const int na = min(MD_M, lb.ra - i0);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    constexpr int ET = 16 / sizeof(Tin), PT = MD_N / ET, PD = MD_N / 2, PW = MD_K / 2;
    auto stage = [&](int s, int j0) {
        unsigned char *base = md_raw + s * S::STAGE;
        double *Ws = reinterpret_cast<double *>(base + S::W);
        double *Vs = reinterpret_cast<double *>(base + S::V);
        Tin *Xs = reinterpret_cast<Tin *>(base + S::X);
        double *Ds = reinterpret_cast<double *>(base + S::D);
        // W, V rows: an odd last partner has a zero in the row's padding
#pragma unroll
        for (int e = t; e < MD_M * PW; e += 256) {
            const int r = e / PW, at = (e - r * PW) * 2;
            const bool ok = r < na && j0 + at < je;
            const long long row = lb.woff + (long long)(i0 + (r < na ? r : 0)) * lb.ldw;
            md_cp16(Ws + r * MD_LDK + at, ok ? W + row + j0 + at : W, ok);
            md_cp16(Vs + r * MD_LDK + at, ok ? V + row + j0 + at : V, ok);
        }
        auto column = [&](int at, bool &ok) {
            const int gi = g0 + at / 8;
            ok = ok && gi < nused;
            return gi < nused ? list[gi] * 8 + at % 8 : 0;
        };
#pragma unroll
        for (int e = t; e < MD_K * PT; e += 256) {
            const int r = e / PT, at = (e - r * PT) * ET, j = j0 + r;
            bool ok = j < je;
            const int k = column(at, ok);
            const Tin *row = x2 + (size_t)(j < je ? idx2[lb.sb + j] : 0) * rep;
            md_piece<Tin>(Xs + r * S::LDN + at, row + k, ok, rep - k, vec);
        }
        if (ad) {
#pragma unroll
            for (int e = t; e < MD_K * PD; e += 256) {
                const int r = e / PD, at = (e - r * PD) * 2, j = j0 + r;
                bool ok = j < je;
                const int k = column(at, ok);
                const double *row = ad + (size_t)(j < je ? idx2[lb.sb + j] : 0) * rep;
                md_piece<double>(Ds + r * S::LDD + at, row + k, ok, rep - k, vec);
            }
        }
        md_commit();
    };
    const int wm = warp & 1, wn = warp >> 1;
    const bool active = 16 * wm < na;
    double acc[2][2][2] = {};
    stage(0, jb);
    int s = 0;
    for (int j0 = jb; j0 < je; j0 += MD_K, s ^= 1) {
        md_wait<0>();
        __syncthreads();   // the slice has landed, and the other buffer is read
        if (j0 + MD_K < je) stage(s ^ 1, j0 + MD_K);
        if (!active) continue;
        const unsigned char *base = md_raw + s * S::STAGE;
        const double *Ws = reinterpret_cast<const double *>(base + S::W);
        const double *Vs = reinterpret_cast<const double *>(base + S::V);
        const Tin *Xs = reinterpret_cast<const Tin *>(base + S::X);
        const double *Ds = reinterpret_cast<const double *>(base + S::D);
        const int r = lane >> 2, kl = lane & 3;
#pragma unroll
        for (int kk = 0; kk < MD_K; kk += 4) {
            const int k = kk + kl, r0 = (16 * wm + r) * MD_LDK + k, r1 = r0 + 8 * MD_LDK;
            const double v0 = Vs[r0], v1 = Vs[r1], w0 = Ws[r0], w1 = Ws[r1];
#pragma unroll
            for (int nj = 0; nj < 2; ++nj) {
                const int col = 16 * wn + 8 * nj + r;
                const double x = (double)Xs[k * S::LDN + col];
                dmma(acc[0][nj], v0, x);
                dmma(acc[1][nj], v1, x);
                if (ad) {
                    const double d = Ds[k * S::LDD + col];
                    dmma(acc[0][nj], w0, d);
                    dmma(acc[1][nj], w1, d);
                }
            }
        }
    }
    if (!active) return;
#pragma unroll
    for (int mi = 0; mi < 2; ++mi) {
        const int i = 16 * wm + 8 * mi + (lane >> 2);
        if (i >= na) continue;
        double *row = g + (size_t)(lb.sa + i0 + i) * rep;
#pragma unroll
        for (int nj = 0; nj < 2; ++nj) {
            const int gi = g0 + 2 * wn + nj;
            if (gi >= nused) continue;
            const int k = list[gi] * 8 + 2 * (lane & 3);
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (k + u < rep) atomicAdd(row + k + u, acc[mi][nj][u]);
        }
    }
}

size_t workspace_budget() {
    const char *v = std::getenv("KFB_WORKSPACE_GB");
    double gb = v ? std::atof(v) : 4.0;
    if (!(gb > 0)) gb = 4.0;
    return (size_t)(gb * (1ull << 30));
}

// FP64-class products on the int8 tensor cores (ozaki.h): 7 digit planes per
// operand (about 48 significant bits), exact int32 level sums combined in FP64.
constexpr int MV_S = 7;
constexpr int MV_KMAX = 65536;   // K of one product (int32 level sums stay exact)

// Digit planes of one operand, the buffers grown on demand.
struct MvOperand {
    DevBuf d, e;
    OzSlices sl;
    kfb_status reserve(long long rows, int K, cudaStream_t s) {
        const int kp = oz_kp(std::max(K, 1));
        const size_t nd = (size_t)MV_S * (size_t)std::max<long long>(rows, 1) * kp;
        const size_t ne = (size_t)std::max<long long>(rows, 1) * sizeof(int);
        if (d.bytes < nd) {
            d.release();
            KFB_TRY(d.alloc(nd, s));
        }
        if (e.bytes < ne) {
            e.release();
            KFB_TRY(e.alloc(ne, s));
        }
        sl.d = d.as<int8_t>();
        sl.e = e.as<int>();
        sl.S = MV_S;
        sl.rows = rows;
        sl.kp = kp;
        return KFB_OK;
    }
    // rows of a row-major source (ld between rows)
    kfb_status rows_of(const double *src, long long rows, int K, long long ld, cudaStream_t s) {
        KFB_TRY(reserve(rows, K, s));
        return oz_slice_rows<double>(src, rows, K, ld, sl, s);
    }
    // rows of the transpose of a row-major source: row i = column i
    kfb_status cols_of(const double *src, long long rows, int K, long long ld, DevBuf &mx,
                       cudaStream_t s) {
        KFB_TRY(reserve(rows, K, s));
        if (mx.bytes < (size_t)rows * 8) {
            mx.release();
            KFB_TRY(mx.alloc((size_t)rows * 8, s));
        }
        return oz_slice_colmajor(src, rows, K, ld, sl, mx.as<unsigned long long>(), s);
    }
};

// C[j * ldc + i] (or +=) alpha sum_k A[i][k] B[j][k] for i < M (rows of A),
// j < N (rows of B): A's rows run along C's contiguous dimension, so the
// epilogue's stores are coalesced.
kfb_status mv_gemm(const OzSlices &A, const OzSlices &B, int M, int N, double *C, long long ldc,
                   double alpha, bool add, int *err, cudaStream_t s) {
    OzGen g;
    g.mode = OZ_GEN_RECT;
    g.M = M;
    g.N = N;
    OzEpi epi;
    epi.c = C;
    epi.ldr = 1;
    epi.ldc = ldc;
    epi.mode = add ? OZ_ADD : OZ_STORE;
    epi.alpha = alpha;
    return oz_gemm_gen(A, B, g, epi, err, s);
}

// Same-label (query atom, training atom) pairs up to which the direct FP64
// kernels are used: they take 1.1, 1.9, 3.5 and 6.6 ms for 4, 8, 17 and 33
// million pairs, the label products on the int8 tensor cores (with their
// launches and host work per label) 1.7, 2.1, 3.1 and 4.6 ms.
constexpr long long MD_MAX_PAIRS = 10LL << 20;
constexpr int MD_MAX_REP = 1 << 16;   // (a list of column groups in shared memory)

template <class Tin>
kfb_status matvec_direct(const Tin *x1, const Tin *dx1, const Tin *x2, const double *ad,
                         const double *alpha_e, const SetView &s1, const std::vector<int> &off1,
                         int s2_ma, const Buckets &b1, const Buckets &b2, int rep, double sigma,
                         double *E, double *F, cudaStream_t s) {
    const int L = (int)b1.labels.size();
    std::vector<MvLabel> labs;
    std::vector<int> src1, src2;   // rows of the labels that both sets have
    long long words = 0, blocks = 0;
    int tiles1 = 0;
    const int nt = (rep + MD_N - 1) / MD_N;
    for (int l = 0; l < L; ++l) {
        const int a0 = b1.lab_start[l], a1 = b1.lab_start[l + 1];
        const int c0 = b2.lab_start[l], c1 = b2.lab_start[l + 1];
        if (a1 == a0 || c1 == c0) continue;
        MvLabel m{};
        m.sa = (int)src1.size();
        m.ra = a1 - a0;
        m.sb = (int)src2.size();
        m.rb = c1 - c0;
        src1.insert(src1.end(), b1.src.begin() + a0, b1.src.begin() + a1);
        src2.insert(src2.end(), b2.src.begin() + c0, b2.src.begin() + c1);
        m.tile1 = tiles1;
        tiles1 += (m.ra + MD_M - 1) / MD_M * ((m.rb + MD_N - 1) / MD_N);
        m.ldw = (m.rb + 1) / 2 * 2;
        m.woff = words;
        words += (long long)m.ra * m.ldw;
        blocks += (long long)((m.ra + MD_M - 1) / MD_M) * nt * ((m.rb + MD_K - 1) / MD_K);
        labs.push_back(m);
    }
    if (labs.empty()) return KFB_OK;
    // training rows per gradient block: enough blocks for four per SM, but not
    // so few rows that the atomics of the split outweigh them
    const long long per = std::max<long long>(4, blocks / (4LL * device_sm_count()));
    const int jlen = (int)std::min<long long>(per, 1 << 20) * MD_K;
    int tiles2 = 0;
    for (MvLabel &m : labs) {
        m.tile2 = tiles2;
        tiles2 += (m.ra + MD_M - 1) / MD_M * nt * ((m.rb + jlen - 1) / jlen);
    }
    // one upload: label table, then the rows of both sets, offsets, atom counts
    std::vector<int> blob(labs.size() * sizeof(MvLabel) / sizeof(int));
    std::memcpy(blob.data(), labs.data(), labs.size() * sizeof(MvLabel));
    auto append = [&](const std::vector<int> &v) {
        const size_t at = blob.size();
        blob.insert(blob.end(), v.begin(), v.end());
        return at;
    };
    const int R1 = (int)src1.size();
    const size_t o_src1 = append(src1), o_src2 = append(src2), o_off1 = append(off1);
    const size_t o_n1 = blob.size();
    for (int m = 0; m < s1.nm; ++m) blob.push_back(s1.natoms(m));
    const int R2 = (int)src2.size(), ng = (rep + 7) / 8;
    DevBuf plan, wv, gr;
    KFB_TRY(upload(plan, blob, s));
    const int *dp = plan.as<int>();
    const bool with_f = F != nullptr;
    // cleared: gradient rows and rowsum(V) (with forces), then the group flags; then the row sums
    const size_t gwords = with_f ? (size_t)R1 * (rep + 1) : 0;
    const size_t clear = gwords * sizeof(double) + (size_t)(ng + 1) / 2 * sizeof(double);
    if (with_f) KFB_TRY(wv.alloc((size_t)words * 2 * sizeof(double), s));
    KFB_TRY(gr.alloc(clear + ((size_t)R1 + 2 * (size_t)R2) * sizeof(double), s));
    KFB_TRY(zero(gr.ptr, clear, s));
    double *W = wv.as<double>(), *V = W + words;
    double *g = gr.as<double>(), *rowv = g + (size_t)R1 * rep;
    int *used = reinterpret_cast<int *>(g + gwords);
    double *n1 = reinterpret_cast<double *>(gr.as<char>() + clear), *n2 = n1 + R1, *sc = n2 + R2;
    auto aligned = [](const void *p) { return (reinterpret_cast<size_t>(p) & 15) == 0; };
    const int vec = rep % 8 == 0 && aligned(x1) && aligned(x2) && aligned(ad);
    const double c = -1.0 / (2.0 * sigma * sigma), is2 = 1.0 / (sigma * sigma), is4 = is2 * is2;
    const int nlab = (int)labs.size();
    const MvLabel *dl = reinterpret_cast<const MvLabel *>(dp);
    // the kernels' limit is that of the longest list, the same in every call: another
    // thread's call may come between this one's setting and its launch
    constexpr size_t st_w = (size_t)MvW<Tin>::NST * MvW<Tin>::STAGE;
    constexpr size_t st_g = (size_t)MvG<Tin>::NST * MvG<Tin>::STAGE;
    constexpr size_t lmax = (size_t)(MD_MAX_REP / 8 + 1) * sizeof(int);
    static_assert(st_w + lmax <= 227 * 1024 && st_g + lmax <= 227 * 1024, "shared memory");
    const size_t lbytes = (size_t)(ng + 1) * sizeof(int);
    const size_t sm_w = st_w + lbytes, sm_g = st_g + lbytes;
    KFB_CUDA_TRY(cudaFuncSetAttribute(mv_weights_kernel<Tin>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(st_w + lmax)));
    KFB_CUDA_TRY(cudaFuncSetAttribute(mv_grad_kernel<Tin>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(st_g + lmax)));
    mv_rows_kernel<Tin><<<nblk((long long)R1 + R2, 8), 256, 0, s>>>(
        x1, dp + o_src1, R1, x2, dp + o_src2, R2, ad, rep, vec, n1, n2, sc, used);
    mv_weights_kernel<Tin><<<tiles1, 256, sm_w, s>>>(
        x1, dp + o_src1, s1.ma, x2, dp + o_src2, s2_ma, ad, alpha_e, dl, nlab, rep, vec,
        with_f ? 1 : 0, c, is2, is4, n1, n2, sc, used, W, V, E, rowv);
    KFB_CUDA_TRY(cudaGetLastError());
    if (!with_f) return KFB_OK;
    mv_grad_kernel<Tin><<<tiles2, 256, sm_g, s>>>(x2, dp + o_src2, ad, dl, nlab, rep, jlen, vec,
                                                  used, W, V, g);
    KFB_CUDA_TRY(cudaGetLastError());
    force_contract_kernel<Tin><<<dim3(R1, (rep + FC_K - 1) / FC_K), 256, 0, s>>>(
        x1, dx1, dp + o_src1, dp + o_n1, dp + o_off1, s1.ma, rep, g, rowv, F);
    KFB_CUDA_TRY(cudaGetLastError());
    return KFB_OK;
}

template <class Tin>
kfb_status matvec_t(const Tin *x1, const Tin *dx1, const Tin *x2, const double *ad,
                    const double *alpha_e, const SetView &s1, const SetView &s2, int rep,
                    double sigma, double *E, double *F, cudaStream_t s) {
    if (E) KFB_TRY(zero(E, (size_t)s1.nm * sizeof(double), s));
    std::vector<int> off1;
    const long long naq1 = deriv_offsets(s1, off1);
    if (F) KFB_TRY(zero(F, (size_t)std::max<long long>(naq1, 1) * sizeof(double), s));
    Buckets b1, b2;
    plan_buckets(s1, &s2, b1, &b2);
    const std::vector<int> &labels = b1.labels;
    if (labels.empty()) return KFB_OK;
    if (!device_is_sm100())
        return set_error(KFB_ERR_UNSUPPORTED, "the contracted prediction needs an sm_100 (B200) device");
    long long pairs = 0;
    for (size_t l = 0; l < labels.size(); ++l)
        pairs += (long long)(b1.lab_start[l + 1] - b1.lab_start[l]) *
                 (b2.lab_start[l + 1] - b2.lab_start[l]);
    if (pairs <= MD_MAX_PAIRS && rep <= MD_MAX_REP &&
        (size_t)pairs * 2 * sizeof(double) <= workspace_budget())
        return matvec_direct<Tin>(x1, dx1, x2, ad, alpha_e, s1, off1, s2.ma, b1, b2, rep, sigma, E, F,
                                  s);
    std::vector<int> n1v(s1.nm);
    for (int m = 0; m < s1.nm; ++m) n1v[m] = s1.natoms(m);
    DevBuf dn1, doff1, didx1, didx2, derr, mx;
    KFB_TRY(upload(dn1, n1v, s));
    KFB_TRY(upload(doff1, off1, s));
    KFB_TRY(upload(didx1, b1.src, s));
    KFB_TRY(upload(didx2, b2.src, s));
    // one pipeline-timeout flag for every tensor-core product of the call
    KFB_TRY(derr.alloc(sizeof(int), s));
    KFB_TRY(zero(derr.ptr, sizeof(int), s));
    int *err = derr.as<int>();
    const double c = -1.0 / (2.0 * sigma * sigma), is2 = 1.0 / (sigma * sigma), is4 = is2 * is2;
    const bool with_ad = ad != nullptr, with_f = F != nullptr;
    MvOperand X2s, Ads, X1s, Ms;
    for (int l = 0; l < (int)labels.size(); ++l) {
        const int sa = b1.lab_start[l], r1 = b1.lab_start[l + 1] - sa;
        const int sb = b2.lab_start[l], r2 = b2.lab_start[l + 1] - sb;
        if (r1 == 0 || r2 == 0) continue;
        // training side of the label: X2, |x|^2, Ad, x.Ad, alpha_E of its molecule
        DevBuf X2l, n2l, Adl, scl, ael;
        KFB_TRY(X2l.alloc((size_t)r2 * rep * sizeof(double), s));
        KFB_TRY(n2l.alloc((size_t)r2 * sizeof(double), s));
        KFB_TRY(scl.alloc((size_t)r2 * sizeof(double), s));
        KFB_TRY(ael.alloc((size_t)r2 * sizeof(double), s));
        gather_f64_kernel<Tin><<<r2, 128, 0, s>>>(x2, didx2.as<int>() + sb, r2, rep,
                                                  X2l.as<double>(), n2l.as<double>());
        if (with_ad) {
            KFB_TRY(Adl.alloc((size_t)r2 * rep * sizeof(double), s));
            gather_f64_kernel<double><<<r2, 128, 0, s>>>(ad, didx2.as<int>() + sb, r2, rep,
                                                         Adl.as<double>(), nullptr);
        }
        train_scalars_kernel<<<nblk(r2, 8), 256, 0, s>>>(
            X2l.as<double>(), with_ad ? Adl.as<double>() : nullptr, didx2.as<int>() + sb,
            s2.ma, alpha_e, r2, rep, scl.as<double>(), ael.as<double>());
        KFB_CUDA_TRY(cudaGetLastError());
        // digit planes of the training rows (K = rep) and, for the force
        // products g = W Ad - V X2 (K = r2, in chunks of MV_KMAX), of their
        // transposes
        KFB_TRY(X2s.rows_of(X2l.as<double>(), r2, rep, rep, s));
        if (with_ad) KFB_TRY(Ads.rows_of(Adl.as<double>(), r2, rep, rep, s));
        const int nkc = (r2 + MV_KMAX - 1) / MV_KMAX;
        std::vector<std::unique_ptr<MvOperand>> X2t, Adt;
        if (with_f)
            for (int kc = 0; kc < nkc; ++kc) {
                const int k0 = kc * MV_KMAX, kn = std::min(MV_KMAX, r2 - k0);
                X2t.emplace_back(new MvOperand);
                KFB_TRY(X2t.back()->cols_of(X2l.as<double>() + (size_t)k0 * rep, rep, kn, rep,
                                            mx, s));
                if (with_ad) {
                    Adt.emplace_back(new MvOperand);
                    KFB_TRY(Adt.back()->cols_of(Adl.as<double>() + (size_t)k0 * rep, rep, kn,
                                                rep, mx, s));
                }
            }
        // query rows in chunks: G and P (r1c x r2 each), X1 and g (r1c x rep)
        const size_t per_row = ((size_t)2 * r2 + 2 * rep + 2) * sizeof(double) +
                               (size_t)MV_S * (std::min(r2, MV_KMAX) + rep + 64);
        const int chunk = (int)std::max<size_t>(1, std::min<size_t>(r1, workspace_budget() / per_row));
        DevBuf X1c, n1c, Gm, Pm, gm, rowv;
        KFB_TRY(X1c.alloc((size_t)chunk * rep * sizeof(double), s));
        KFB_TRY(n1c.alloc((size_t)chunk * sizeof(double), s));
        KFB_TRY(Gm.alloc((size_t)chunk * r2 * sizeof(double), s));
        KFB_TRY(Pm.alloc((size_t)chunk * r2 * sizeof(double), s));
        if (with_f) {
            KFB_TRY(gm.alloc((size_t)chunk * rep * sizeof(double), s));
            KFB_TRY(rowv.alloc((size_t)chunk * sizeof(double), s));
        }
        for (int q0 = 0; q0 < r1; q0 += chunk) {
            const int rc = std::min(chunk, r1 - q0);
            gather_f64_kernel<Tin><<<rc, 128, 0, s>>>(x1, didx1.as<int>() + sa + q0, rc, rep,
                                                      X1c.as<double>(), n1c.as<double>());
            KFB_CUDA_TRY(cudaGetLastError());
            KFB_TRY(X1s.rows_of(X1c.as<double>(), rc, rep, rep, s));
            // G (rc x r2 row-major) = X1 X2^T, P = X1 Ad^T
            KFB_TRY(mv_gemm(X2s.sl, X1s.sl, r2, rc, Gm.as<double>(), r2, 1.0, false, err, s));
            if (with_ad)
                KFB_TRY(mv_gemm(Ads.sl, X1s.sl, r2, rc, Pm.as<double>(), r2, 1.0, false, err, s));
            pair_weights_kernel<<<rc, 256, 0, s>>>(
                Gm.as<double>(), Pm.as<double>(), r2, n1c.as<double>(), n2l.as<double>(),
                scl.as<double>(), ael.as<double>(), didx1.as<int>() + sa + q0, s1.ma, with_ad ? 1 : 0,
                with_f ? 1 : 0, c, is2, is4, E, with_f ? rowv.as<double>() : nullptr);
            KFB_CUDA_TRY(cudaGetLastError());
            if (!with_f) continue;
            // g = W Ad + rowsum(V) x1 - V X2 (rc x rep row-major), W over G and V over P
            if (with_ad) {
                for (int kc = 0; kc < nkc; ++kc) {
                    const int k0 = kc * MV_KMAX, kn = std::min(MV_KMAX, r2 - k0);
                    KFB_TRY(Ms.rows_of(Gm.as<double>() + k0, rc, kn, r2, s));
                    KFB_TRY(mv_gemm(Adt[kc]->sl, Ms.sl, rep, rc, gm.as<double>(), rep, 1.0,
                                    kc > 0, err, s));
                }
            } else {
                KFB_TRY(zero(gm.ptr, (size_t)rc * rep * sizeof(double), s));
            }
            add_row_scaled_kernel<<<nblk((long long)rc * rep, 256), 256, 0, s>>>(
                X1c.as<double>(), rowv.as<double>(), rc, rep, gm.as<double>());
            KFB_CUDA_TRY(cudaGetLastError());
            for (int kc = 0; kc < nkc; ++kc) {
                const int k0 = kc * MV_KMAX, kn = std::min(MV_KMAX, r2 - k0);
                KFB_TRY(Ms.rows_of(Pm.as<double>() + k0, rc, kn, r2, s));
                KFB_TRY(mv_gemm(X2t[kc]->sl, Ms.sl, rep, rc, gm.as<double>(), rep, -1.0, true,
                                err, s));
            }
            force_contract_kernel<Tin><<<dim3(rc, (rep + FC_K - 1) / FC_K), 256, 0, s>>>(
                x1, dx1, didx1.as<int>() + sa + q0, dn1.as<int>(), doff1.as<int>(), s1.ma, rep, gm.as<double>(), nullptr, F);
            KFB_CUDA_TRY(cudaGetLastError());
        }
    }
    int herr = 0;
    KFB_CUDA_TRY(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s));
    KFB_CUDA_TRY(cudaStreamSynchronize(s));
    if (herr)
        return set_error(KFB_ERR_TIMEOUT, "contracted prediction: a tensor-core pipeline wait timed out");
    return KFB_OK;
}

template <class Tin>
kfb_status alpha_desc_t(const Tin *dx2, const SetView &s2, int rep, const double *alpha,
                        double *ad, cudaStream_t s) {
    std::vector<int> off2;
    deriv_offsets(s2, off2);
    std::vector<int> n2v(s2.nm);
    for (int m = 0; m < s2.nm; ++m) n2v[m] = s2.natoms(m);
    DevBuf dn2, doff2;
    KFB_TRY(upload(dn2, n2v, s));
    KFB_TRY(upload(doff2, off2, s));
    alpha_desc_kernel<Tin><<<dim3(s2.ma, s2.nm), 256, 0, s>>>(dx2, dn2.as<int>(), doff2.as<int>(),
                                                             s2.ma, rep, alpha, ad);
    KFB_CUDA_TRY(cudaGetLastError());
    return KFB_OK;
}

}  // namespace

}  // namespace kfb

using namespace kfb;

extern "C" {

kfb_status kfb_local_alpha_desc(const void *dx2, const int32_t *q2, const int32_t *n2, int nm2,
                                int ma2, int rep, kfb_dtype x_dt, const double *alpha,
                                double *alpha_desc, void *stream) {
    (void)q2;  // the contraction does not depend on the labels
    if (!dx2 || !n2 || !alpha || !alpha_desc)
        return set_error(KFB_ERR_INVALID_ARG, "null pointer");
    if (nm2 <= 0 || ma2 <= 0 || rep <= 0)
        return set_error(KFB_ERR_INVALID_ARG, "dimensions must be positive");
    SetView v;
    v.n = n2;
    v.nm = nm2;
    v.ma = ma2;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (x_dt == KFB_F64)
        return alpha_desc_t<double>(static_cast<const double *>(dx2), v, rep, alpha, alpha_desc, s);
    return alpha_desc_t<float>(static_cast<const float *>(dx2), v, rep, alpha, alpha_desc, s);
}

kfb_status kfb_local_matvec(const void *x1, const void *dx1, const void *x2,
                            const double *alpha_desc, const double *alpha_e, const int32_t *q1,
                            const int32_t *q2, const int32_t *n1, const int32_t *n2, int nm1,
                            int nm2, int ma1, int ma2, int rep, double sigma, kfb_dtype x_dt,
                            double *e_out, double *f_out, void *stream) {
    if (!x1 || !x2 || !q1 || !q2 || !n1 || !n2)
        return set_error(KFB_ERR_INVALID_ARG, "null pointer");
    if (nm1 <= 0 || nm2 <= 0 || ma1 <= 0 || ma2 <= 0 || rep <= 0)
        return set_error(KFB_ERR_INVALID_ARG, "dimensions must be positive");
    if (!(sigma > 0.0)) return set_error(KFB_ERR_INVALID_ARG, "sigma must be > 0");
    if (f_out && !dx1) return set_error(KFB_ERR_INVALID_ARG, "forces need dX1");
    if (!e_out && !f_out) return KFB_OK;
    SetView v1, v2;
    v1.q = q1;
    v1.n = n1;
    v1.nm = nm1;
    v1.ma = ma1;
    v2.q = q2;
    v2.n = n2;
    v2.nm = nm2;
    v2.ma = ma2;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (x_dt == KFB_F64)
        return matvec_t<double>(static_cast<const double *>(x1), static_cast<const double *>(dx1),
                                static_cast<const double *>(x2), alpha_desc, alpha_e, v1, v2, rep,
                                sigma, e_out, f_out, s);
    return matvec_t<float>(static_cast<const float *>(x1), static_cast<const float *>(dx1),
                           static_cast<const float *>(x2), alpha_desc, alpha_e, v1, v2, rep,
                           sigma, e_out, f_out, s);
}

}  // extern "C"
