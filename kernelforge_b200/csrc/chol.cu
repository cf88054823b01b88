// Blocked right-looking Cholesky factorisation: the diagonal blocks, the rows
// below them and the updates within an outer panel on FP64 mma.sync, the
// trailing updates on the int8 tensor cores (digit-sliced FP64 products,
// ozaki.h).  Column-major storage, lower triangle.
//
// Outer panels of 512 columns.  Per panel (o0, rows R = o0 + 512 .. n - 1 below):
//   1. its 512 x 512 diagonal block, per 128-column block:
//      chol_block64_kernel (FP32-class factor: chol_block_kernel): one CTA
//        factors the w x w diagonal block in shared memory and forms W =
//        L_jj^{-1}; the first non-positive pivot is recorded (LAPACK potrf's
//        info);
//      chol_panel_kernel: L_21 = A_21 W^T for the rows of the outer panel;
//      chol_update_kernel: the rest of the diagonal block -= L_21 L_21^T, the
//        next 128 columns on the critical stream, the rest beside that block's
//        factorisation;
//   2. chol_far_kernel: the rows below, all 512 columns of a row tile in one
//      CTA, with their digit planes; the 512 rows of the next diagonal block on
//      the critical stream, the others on the far stream;
//   3. trailing products with K = 512 on the tensor cores: the next diagonal
//      block on the critical stream, the columns below it on the far stream, the
//      rest on the bulk stream, the columns of the panel after the next first.
// So the critical path holds what the next diagonal block needs and no more:
// per panel four diagonal blocks and seven launches of few CTAs.  The other
// streams' work, which fills the GPU, has a panel's time to finish (look-ahead;
// digit planes and inverted blocks of consecutive panels alternate between two
// buffers).  With every row of a 128-column panel on the critical path, and its
// digit planes sliced per 128 and again per 512 columns, n = 10,000 took 10.6
// ms; now 5.9 ms.
// The block order is that of LAPACK's right-looking dpotrf with the panel's
// triangular solve replaced by a product with the inverted diagonal block
// (the inverse-based form used by GPU Cholesky codes).  A failed pivot raises
// a device flag that makes every later kernel of the factorisation return at
// once; the host reads the pivot index once, at the end.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "chol.h"
#include "kernels_common.cuh"
#include "ozaki.h"

namespace kfb {

namespace {

constexpr int NB = CHOL_NB;       // 128
constexpr int SB = 32;            // sub-block of the diagonal factorisation
constexpr int LDT = NB + 2;       // shared column stride of the block (doubles; even)
constexpr int LDW = SB + 1;       // shared column stride of a 32 x 32 inverse block
constexpr int NWB = 10;           // lower 32 x 32 blocks of a 128 x 128 triangle
constexpr int BLK_THREADS = 512;
constexpr int BLK_WARPS = BLK_THREADS / 32;
constexpr int NB2 = 4 * NB;       // outer panel (two-level blocking)
constexpr int PR = 16;            // panel rows per CTA
constexpr int UT = 32;            // tile of the near update
constexpr int PANEL_THREADS = 256;
constexpr int FAR_THREADS = 256;
// tiles per CTA of a bulk update: 2 .. 8 are equal within 1%, with persistent CTAs the other
// streams wait (n = 10,000: 12.2 against 11.1 ms a solve)
constexpr int BULK_TILES = 4;

static_assert(NB == 4 * SB, "the block kernel assumes four sub-blocks");

__host__ __device__ constexpr int wblk(int i, int j) { return i * (i + 1) / 2 + j; }

using F = float;   // arithmetic of the FP32-class diagonal block
constexpr size_t BLK_SMEM = ((size_t)NB * LDT + (size_t)NWB * SB * LDW + SB) * sizeof(F) + 16;
constexpr int LDP = NB + 4, LDX = PR + 4;   // panel kernel: strides of W and of the rows (4 mod 16)
constexpr int LDU = UT + 4;
constexpr size_t UPD_SMEM = (size_t)2 * NB * LDU * sizeof(double);
constexpr size_t PANEL_SMEM = (size_t)NB * (LDP + LDX) * sizeof(double);

// Asynchronous global -> shared copies (cp.async): `bytes` of 8 or 16, with
// the shared destination zero-filled instead when `valid` is false (the
// source pointer must still be a valid address).
__device__ __forceinline__ void cp_async(void *sdst, const void *gsrc, int bytes, bool valid) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(sdst));
    if (bytes == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(gsrc),
                     "r"(valid ? 16 : 0)
                     : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(gsrc),
                     "r"(valid ? 8 : 0)
                     : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.wait_all;" ::: "memory");
}

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ float pivot_rsqrt(float d) { return rsqrtf(d); }

// Factor the w x w block at (c0, c0) of the column-major matrix A in place
// (lower triangle) and write W = L^{-1} column-major into Wout (NB x NB, zero
// above the diagonal and beyond w), with FP32 arithmetic (an FP32-class
// factor; chol_block64_kernel is the FP64 one).
//
// Shared memory: T[k * LDT + r] = A[c0 + r][c0 + k] (zero outside the lower
// w x w triangle); WB holds the lower 32 x 32 blocks of W, block (i, j) at
// WB + wblk(i, j) * SB * LDW, element (r, c) at [c * LDW + r]; rd[r] = 1 /
// L[o + r][o + r] of the current sub-block.
__global__ void __launch_bounds__(BLK_THREADS, 1)
    chol_block_kernel(double *__restrict__ A, long long ld, int c0, int w,
                      double *__restrict__ Wout, int *info, int *skip) {
    using F2 = float2;
    if (*(volatile int *)skip) return;
    extern __shared__ __align__(16) unsigned char sm_raw[];
    F *T = reinterpret_cast<F *>(sm_raw);
    F *WB = T + NB * LDT;
    F *rd = WB + NWB * SB * LDW;   // 1 / L[o + r][o + r] of the current sub-block
    int *flag = reinterpret_cast<int *>(rd + SB);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double *blk = A + (long long)c0 * ld + c0;
    {
        // eight independent loads in flight per thread, then the conversions
        constexpr int PER = NB * NB / BLK_THREADS;
        static_assert(PER % 8 == 0, "load batches");
        for (int b = 0; b < PER; b += 8) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int idx = tid + (b + u) * BLK_THREADS, k = idx / NB, r = idx - k * NB;
                v[u] = (r < w && k < w && r >= k) ? blk[(long long)k * ld + r] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int idx = tid + (b + u) * BLK_THREADS, k = idx / NB, r = idx - k * NB;
                T[k * LDT + r] = (F)v[u];
            }
        }
    }
    if (tid == 0) *flag = 0;
    __syncthreads();
    const int P = (w + SB - 1) / SB;
    for (int p = 0; p < P; ++p) {
        const int o = p * SB, wp = min(SB, w - o);
        if (warp == 0) {
            // (a) right-looking factorisation of the wp x wp diagonal
            // sub-block in registers: lane = row, a[k] = L[lane][k] (k <= lane)
            F a[SB];
#pragma unroll
            for (int k = 0; k < SB; ++k) a[k] = (k <= lane) ? T[(o + k) * LDT + o + lane] : F(0);
            F rinv = F(0);   // 1 / L[lane][lane]
            int bad = SB;        // first column with a non-positive pivot
#pragma unroll
            for (int c = 0; c < SB; ++c) {
                if (c < wp) {
                    const F d = __shfl_sync(FULL, a[c], c);
                    if (!(d > F(0)) || !isfinite(d)) bad = min(bad, c);   // warp-uniform
                    const F rs = pivot_rsqrt(d);
                    const F l = (lane == c) ? d * rs : a[c] * rs;
                    if (lane == c) rinv = rs;
                    a[c] = l;
                    // the scaled column is final: write it, then read it back as
                    // a broadcast (faster than 31 shuffles on the pivot chain:
                    // 164 vs 247 cycles per column)
                    if (lane >= c && lane < wp) T[(o + c) * LDT + o + lane] = l;
                    __syncwarp();
#pragma unroll
                    for (int k = c + 1; k < SB; ++k) {
                        const F lk = T[(o + c) * LDT + o + k];   // L[k][c] (0 beyond wp)
                        // a select and an unconditional FMA (no divergent
                        // branch per k: 71 -> 60 us per block)
                        const F m = (k <= lane) ? l : F(0);
                        a[k] = fma(-m, lk, a[k]);
                    }
                }
            }
            if (bad < wp) {
                if (lane == 0) {
                    *info = c0 + o + bad + 1;
                    atomicExch(skip, 1);
                    *flag = 1;
                }
            } else {
                rd[lane] = rinv;
            }
        }
        __syncthreads();
        if (*flag) return;   // block-uniform after the barrier
        if (warp == 0) {
            // (b) W_pp = L_pp^{-1}, lane = column l, forward substitution in
            // right-looking order: W[r][l] = s[r] / L[r][r], then
            // s[r'] -= L[r'][r] W[r][l] for r' > r (column r of L read as a
            // broadcast), so each row adds one FMA and one multiply to the
            // dependent chain instead of a dot product
            F sacc[SB];
#pragma unroll
            for (int r = 0; r < SB; ++r) sacc[r] = (r == lane) ? F(1) : F(0);
            F *Wp = WB + wblk(p, p) * SB * LDW + lane * LDW;
#pragma unroll
            for (int r = 0; r < SB; ++r) {
                const F xr = (r < wp && lane < wp) ? sacc[r] * rd[r] : F(0);
                Wp[r] = xr;
#pragma unroll
                for (int r2 = r + 1; r2 < SB; ++r2)
                    sacc[r2] = fma(-T[(o + r) * LDT + o + r2], xr, sacc[r2]);
            }
        }
        __syncthreads();
        const int rb = o + wp, mr = w - rb;
        if (mr <= 0) continue;
        const int ns = (mr + 31) / 32;
        // (c) rows below the sub-block: X[r][c] = sum_{k <= c} A[r][o + k] W_pp[c][k]
        //     (unit = 32 rows x 8 columns; lane = row)
        {
            const F *Wp = WB + wblk(p, p) * SB * LDW;
            const int u = warp, s = u >> 2, g = u & 3;
            const int r = rb + 32 * s + lane;
            const bool act = s < ns && r < w;
            F x[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = F(0);
            if (s < ns) {
                const int rr = min(r, NB - 1);
#pragma unroll
                for (int k = 0; k < SB; ++k) {
                    const F a = T[(o + k) * LDT + rr];
#pragma unroll
                    for (int j = 0; j < 8; ++j) x[j] = fma(a, Wp[k * LDW + 8 * g + j], x[j]);
                }
            }
            __syncthreads();
            if (act)
#pragma unroll
                for (int j = 0; j < 8; ++j) T[(o + 8 * g + j) * LDT + r] = x[j];
            __syncthreads();
        }
        // (d) the rest of the block: T[k][r] -= sum_c X[r][c] X[k][c], rb <= k <= r < w
        //     (unit = 32 rows of strip s x 8 columns; strip s has 4 (s + 1) groups)
        {
            const int nunits = 2 * ns * (ns + 1);
            for (int u = warp; u < nunits; u += BLK_WARPS) {
                int s = 0;
                while (2 * (s + 1) * (s + 2) <= u) ++s;
                const int g = u - 2 * s * (s + 1);
                const int r = rb + 32 * s + lane, k0 = rb + 8 * g;
                const int rr = min(r, NB - 1);
                F acc[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j] = F(0);
#pragma unroll
                for (int c = 0; c < SB; ++c) {
                    const F *col = T + (o + c) * LDT;
                    const F a = col[rr];
                    const F2 *kv = reinterpret_cast<const F2 *>(col + k0);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const F2 b = kv[j];
                        acc[2 * j] = fma(a, b.x, acc[2 * j]);
                        acc[2 * j + 1] = fma(a, b.y, acc[2 * j + 1]);
                    }
                }
                if (r < w)
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (k0 + j <= r) T[(k0 + j) * LDT + r] -= acc[j];
            }
            __syncthreads();
        }
    }
    // W = L^{-1} off the diagonal, by block substitution along block diagonals
    // d = i - j:  M = sum_{j <= k < i} L_ik W_kj,  W_ij = -W_ii M
    // (unit = one 8-column group of one block pair; lane = row)
    for (int d = 1; d < P; ++d) {
        const int nunits = 4 * (P - d);
        for (int u = warp; u < nunits; u += BLK_WARPS) {
            const int j = u >> 2, g = u & 3, i = j + d;
            F m[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) m[q] = F(0);
            for (int k = j; k < i; ++k) {
                const F *Wkj = WB + wblk(k, j) * SB * LDW;
#pragma unroll
                for (int t = 0; t < SB; ++t) {
                    const F l = T[(SB * k + t) * LDT + SB * i + lane];
#pragma unroll
                    for (int q = 0; q < 8; ++q) m[q] = fma(l, Wkj[(8 * g + q) * LDW + t], m[q]);
                }
            }
            F *Wij = WB + wblk(i, j) * SB * LDW;
#pragma unroll
            for (int q = 0; q < 8; ++q) Wij[(8 * g + q) * LDW + lane] = m[q];
        }
        __syncthreads();
        for (int u = warp; u < nunits; u += BLK_WARPS) {
            const int j = u >> 2, g = u & 3, i = j + d;
            const F *Wii = WB + wblk(i, i) * SB * LDW;
            F *Wij = WB + wblk(i, j) * SB * LDW;
            F o[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) o[q] = F(0);
#pragma unroll
            for (int t = 0; t < SB; ++t) {
                const F wv = Wii[t * LDW + lane];
#pragma unroll
                for (int q = 0; q < 8; ++q) o[q] = fma(wv, Wij[(8 * g + q) * LDW + t], o[q]);
            }
            // only this warp reads its columns of M: overwrite them in place
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 8; ++q) Wij[(8 * g + q) * LDW + lane] = -o[q];
        }
        __syncthreads();
    }
    double *ablk = A + (long long)c0 * ld + c0;
    for (int idx = tid; idx < w * NB; idx += BLK_THREADS) {
        const int k = idx / NB, r = idx - k * NB;
        if (r < w && r >= k) ablk[(long long)k * ld + r] = (double)T[k * LDT + r];
    }
    // W column-major, two rows per 16-byte store
    for (int idx = tid; idx < NB * NB / 2; idx += BLK_THREADS) {
        const int c = idx / (NB / 2), r = 2 * (idx - c * (NB / 2));
        double v[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int rr = r + u;
            v[u] = (rr < w && c < w && rr >= c)
                       ? (double)WB[wblk(rr / SB, c / SB) * SB * LDW + (c % SB) * LDW + (rr % SB)]
                       : 0.0;
        }
        reinterpret_cast<double2 *>(Wout)[idx] = make_double2(v[0], v[1]);
    }
}

// FP64 diagonal block on mma.sync: the w x w block at (c0, c0) factored in
// place and W = L^{-1} written to Wout, as chol_block_kernel does in FP32.
//
// 16 micro-panels of 8 columns over the whole block, one barrier each:
//   A  warp 0 factors the 8 x 8 diagonal block of panel p in registers (every
//      lane the same: no exchange on the pivot chain), and after the barrier
//      solves the next 8 rows with it, updates the next diagonal block and goes
//      on with that one's A;
//   B  four warps solve the other rows below, a thread per row; another one
//      inverts the 8 x 8 block;
//   C  when the rows are there, twelve warps update the rest of the trailing
//      triangle (8 x 8 tiles, K = 8) and form row block p of W, -W_pp sum_{k<p}
//      L_pk W_kj, block by block.  A tile lives in its warp's registers until
//      its column is next (its diagonal tile one panel sooner): read and
//      written in shared memory at every panel, the tiles alone took 2,500
//      cycles of an early panel.  They are dealt out from the last column
//      backwards, so that the warps have equal shares at every panel.
// What bounds it is warp 0's chain over the panels; the rest hides behind it.
// Warps 4, 8 and 12 only copy: warp 0 has its scheduler's FP64 unit for itself
// (with their products on it A took 2,450 cycles).
// (32-column sub-blocks factored by one warp with a lane per row, then
// inverted and applied in phases of their own, took 75-83 us a block; this one
// takes 33 us.)
//
// Shared memory: T[k * DLT + r] holds the lower triangle in column k, row r;
// its strict upper triangle takes W's blocks off the diagonal transposed into
// the same index pattern, W[r][c] at T[r * DLT + c] (c < r); Wp[p] is W_pp by
// rows.  Row strides of 4 and 12 mod 16 doubles keep the fragment loads of a
// half warp on different banks.  Beyond w the block is the identity.
constexpr int DB = 8, DP = NB / DB;      // micro-panel width, their number
constexpr int DLT = NB + 4;              // shared column stride (4 mod 16)
constexpr int DLW = DB + 4;              // row stride of an inverted 8 x 8 block
constexpr size_t DBLK_SMEM =
    ((size_t)NB * DLT + (size_t)DP * (DB * DLW + DB * DB + DB)) * sizeof(double) + 16;
constexpr int BLK_WORK = BLK_WARPS * 3 / 4;   // warps of B and C

// a (lower triangle) -> its Cholesky factor, rinv = 1 / diagonal.  1 /
// sqrt(pivot) is PTX's approximation instruction (about 2^-20) refined by one step
// of Chebyshev's third-order iteration (Traub, Iterative Methods for the Solution
// of Equations, 1964) for f(r) = r^-2 - d: with e = 1 - d r^2, the
// first terms of the binomial series (1 - e)^(-1/2) = 1 + e/2 + 3 e^2/8 + ...; the
// rest is 5/16 e^3.  False (a, rinv void) unless every pivot is positive and far from
// the ends of the range: an integer test of the exponents, off the pivot chain.
__device__ __forceinline__ bool chol8(double (&a)[DB][DB], double (&rinv)[DB]) {
    bool ok = true;
#pragma unroll
    for (int c = 0; c < DB; ++c) {
        const double d = a[c][c];
        // exponents -900 .. 900 (a negative number or a NaN is above them)
        ok &= (unsigned)(__double2hiint(d) - ((1023 - 900) << 20)) <= (1800u << 20);
        double r;
        asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
        const double e = fma(-(d * r), r, 1.0);
        r = fma(r * e, fma(0.375, e, 0.5), r);
        rinv[c] = r;
        a[c][c] = d * r;
#pragma unroll
        for (int k = c + 1; k < DB; ++k) a[k][c] *= r;
#pragma unroll
        for (int k = c + 1; k < DB; ++k)
#pragma unroll
            for (int q = k; q < DB; ++q) a[q][k] = fma(-a[q][c], a[k][c], a[q][k]);
    }
    return ok;
}

// The same by one thread in shared memory, for any pivots: t (column stride DLT)
// -> Ls, rd.  Returns the first column whose pivot is not positive and finite
// (DB: none).
__device__ __noinline__ int chol8_any(const double *t, double *Ls, double *rd) {
    int bad = DB;
    for (int c = 0; c < DB; ++c) {
        for (int r = c; r < DB; ++r) {
            double v = t[c * DLT + r];
            for (int k = 0; k < c; ++k) v = fma(-Ls[r * DB + k], Ls[c * DB + k], v);
            if (r == c) {
                if (!(v > 0.0) || !isfinite(v)) bad = min(bad, c);
                rd[c] = rsqrt(v);
            }
            Ls[r * DB + c] = v * rd[c];
        }
    }
    return bad;
}

// d (a tile's accumulator lanes) -= X_rb X_kb^T for panel columns o .. o + 7 and
// the tile (kb, rb): D's rows are the tile's columns, so that a lane's two
// values are neighbours in T.
__device__ __forceinline__ void chol_tile(double (&d)[2], const double *T, int o, int kb, int rb,
                                          int lane) {
    const int i = lane >> 2, j = lane & 3;
    const double *x0 = T + (o + j) * DLT, *x1 = x0 + 4 * DLT;
    const double a0 = -x0[DB * kb + i], a1 = -x1[DB * kb + i];
    const double b0 = x0[DB * rb + i], b1 = x1[DB * rb + i];
    dmma(d, a0, b0);
    dmma(d, a1, b1);
}

__global__ void __launch_bounds__(BLK_THREADS, 1)
    chol_block64_kernel(double *__restrict__ A, long long ld, int c0, int w,
                        double *__restrict__ Wout, int *info, int *skip) {
    if (*(volatile int *)skip) return;
    extern __shared__ __align__(16) unsigned char sm_raw[];
    double *T = reinterpret_cast<double *>(sm_raw);
    double *Wp = T + NB * DLT;            // [DP][DB][DLW]
    // of each panel: [DB][DB] factor of its 8 x 8 block by rows, [DB] 1 / its diagonal
    double *L8 = Wp + DP * DB * DLW;
    int *flag = reinterpret_cast<int *>(L8 + DP * (DB * DB + DB));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double *blk = A + (long long)c0 * ld + c0;
    if (w == NB && (ld & 1) == 0 && (c0 & 1) == 0) {
        // 16-byte copies (the strict upper triangle comes along and is overwritten before it
        // is read)
#pragma unroll 4
        for (int idx = tid; idx < NB * NB / 2; idx += BLK_THREADS) {
            const int k = idx / (NB / 2), r = 2 * (idx - k * (NB / 2));
            cp_async(T + k * DLT + r, blk + (long long)k * ld + r, 16, true);
        }
        cp_async_wait_all();
    } else {
#pragma unroll 4
        for (int idx = tid; idx < NB * NB; idx += BLK_THREADS) {
            const int k = idx / NB, r = idx - k * NB;
            const bool v = r < w && k < w && r >= k;
            cp_async(T + k * DLT + r, v ? blk + (long long)k * ld + r : blk, 8, v);
        }
        cp_async_wait_all();
        __syncthreads();
        for (int k = w + tid; k < NB; k += BLK_THREADS) T[k * DLT + k] = 1.0;
    }
    if (tid == 0) *flag = DP;   // the panel whose factor failed
    __syncthreads();

    // phase A of panel p (warp 0)
    double a[DB][DB], rinv[DB];
    auto factor = [&](int p) {
        const int o = DB * p;
        double *Ls = L8 + p * (DB * DB + DB), *rd = Ls + DB * DB;
#pragma unroll
        for (int c = 0; c < DB; ++c)
#pragma unroll
            for (int r = c & ~1; r < DB; r += 2) {
                const double2 v = *reinterpret_cast<const double2 *>(T + (o + c) * DLT + o + r);
                if (r >= c) a[r][c] = v.x;
                a[r + 1][c] = v.y;
            }
        if (chol8(a, rinv)) {   // (the same in every lane)
            if (lane == 0) {
#pragma unroll
                for (int r = 0; r < DB; ++r)
#pragma unroll
                    for (int c = 0; c <= r; c += 2)
                        *reinterpret_cast<double2 *>(Ls + r * DB + c) =
                            make_double2(a[r][c], c + 1 <= r ? a[r][c + 1] : 0.0);
#pragma unroll
                for (int c = 0; c < DB; c += 2)
                    *reinterpret_cast<double2 *>(rd + c) = make_double2(rinv[c], rinv[c + 1]);
            }
            return;
        }
        if (lane == 0) {
            const int bad = chol8_any(T + o * DLT + o, Ls, rd);
            if (o + bad < w && bad < DB) {
                *info = c0 + o + bad + 1;
                atomicExch(skip, 1);
                *flag = p;
            }
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < DB; ++r) {
            rinv[r] = rd[r];
#pragma unroll
            for (int c = 0; c <= r; ++c) a[r][c] = Ls[r * DB + c];
        }
    };
    // the panels' barrier; false, in every thread, when panel p's factor failed
    // (warp 0 may be at p + 1 already)
    auto next_panel = [&](int p) {
        asm volatile("bar.sync 0;" ::: "memory");
        return *(volatile int *)flag > p;
    };
    if (warp == 0) {
        factor(0);
        for (int p = 0; p < DP; ++p) {
            const int o = DB * p;
            if (!next_panel(p)) return;
            if (p == DP - 1) {
                asm volatile("bar.arrive 1, %0;" ::"n"(32 * (BLK_WORK + 1)) : "memory");
                break;
            }
            // the next 8 rows (lanes 8 .. 31 repeat lanes 0 .. 7)
            double *x = T + o * DLT + o + DB + (lane & 7), v[DB];
#pragma unroll
            for (int c = 0; c < DB; ++c) v[c] = x[c * DLT];
#pragma unroll
            for (int c = 0; c < DB; ++c) {
                v[c] *= rinv[c];
#pragma unroll
                for (int k = c + 1; k < DB; ++k) v[k] = fma(-v[c], a[k][c], v[k]);
            }
            __syncwarp();
            if (lane < DB)
#pragma unroll
                for (int c = 0; c < DB; ++c) x[c * DLT] = v[c];
            __syncwarp();
            asm volatile("bar.arrive 1, %0;" ::"n"(32 * (BLK_WORK + 1)) : "memory");
            double2 *t = reinterpret_cast<double2 *>(T + (o + DB + (lane >> 2)) * DLT + o + DB +
                                                     2 * (lane & 3));
            double d[2] = {t->x, t->y};
            chol_tile(d, T, o, p + 1, p + 1, lane);
            *t = make_double2(d[0], d[1]);
            __syncwarp();
            factor(p + 1);
        }
    } else if ((warp & 3) == 0) {
        for (int p = 0; p < DP; ++p)
            if (!next_panel(p)) return;
    } else {
        const int wk = warp - 1 - (warp >> 2);   // worker 0 .. BLK_WORK - 1
        // tile number BLK_WORK s + wk from the last column backwards (1 + 2 + ..
        // tiles of columns DP - 1, DP - 2, ..)
        constexpr int NS = (DP * (DP + 1) / 2 + BLK_WORK - 1) / BLK_WORK;
        double acc[NS][2];
        int kr[NS];   // DP column + row of the tile; -1: none
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            int u = 0, t = BLK_WORK * s + wk;
            while (t > u) t -= ++u;
            kr[s] = u < DP ? (DP - 1 - u) * DP + DP - 1 - u + t : -1;
            if (kr[s] >= 0) {
                const double2 v = *reinterpret_cast<const double2 *>(
                    T + (DB * (kr[s] / DP) + (lane >> 2)) * DLT + DB * (kr[s] % DP) +
                    2 * (lane & 3));
                acc[s][0] = v.x;
                acc[s][1] = v.y;
            }
        }
        for (int p = 0; p < DP; ++p) {
            const int o = DB * p, below = NB - o - DB;
            if (!next_panel(p)) return;
            const double *Ls = L8 + p * (DB * DB + DB), *rd = Ls + DB * DB;
            // ---- B: the other rows below, and the inverse of the diagonal block
            const int row = 32 * wk + lane;
            if (row < below - DB) {
                double *x = T + o * DLT + o + DB + DB + row;
                double v[DB];
#pragma unroll
                for (int c = 0; c < DB; ++c) v[c] = x[c * DLT];
#pragma unroll
                for (int c = 0; c < DB; ++c) {
                    v[c] *= rd[c];
#pragma unroll
                    for (int k = c + 1; k < DB; ++k) v[k] = fma(-v[c], Ls[k * DB + c], v[k]);
                }
#pragma unroll
                for (int c = 0; c < DB; ++c) x[c * DLT] = v[c];
            } else if (wk == BLK_WORK - 1 && lane < DB) {
                // column `lane` of W_pp
                double s[DB];
#pragma unroll
                for (int r = 0; r < DB; ++r) s[r] = r == lane ? 1.0 : 0.0;
#pragma unroll
                for (int r = 0; r < DB; ++r) {
                    s[r] *= rd[r];
#pragma unroll
                    for (int k = r + 1; k < DB; ++k) s[k] = fma(-Ls[k * DB + r], s[r], s[k]);
                }
#pragma unroll
                for (int r = 0; r < DB; ++r) Wp[(p * DB + r) * DLW + lane] = s[r];
            }
            asm volatile("bar.sync 1, %0;" ::"n"(32 * (BLK_WORK + 1)) : "memory");
            // ---- C: the tiles of later columns (the next diagonal one is warp 0's)
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                const int kb = kr[s] / DP, rb = kr[s] % DP;
                if (kr[s] >= 0 && kb > p && (kb > p + 1 || rb > kb)) {
                    chol_tile(acc[s], T, o, kb, rb, lane);
                    if (kb == (rb == kb ? p + 2 : p + 1))
                        *reinterpret_cast<double2 *>(T + (DB * kb + (lane >> 2)) * DLT + DB * rb +
                                                     2 * (lane & 3)) =
                            make_double2(acc[s][0], acc[s][1]);
                }
            }
            // W row block p first (the longer chains): block column j to worker j,
            // those beyond the workers to the ones with the shortest chains
            for (int j = wk; j < p; j = 2 * BLK_WORK - 1 - j, j = j < BLK_WORK ? p : j) {
                const int i4 = lane >> 2, k4 = lane & 3;
                double m0[2] = {0.0, 0.0}, m1[2] = {0.0, 0.0};
#pragma unroll 4
                for (int k = j; k < p; ++k) {
                    // A = L_pk, B = W_kj, K = 8 in two steps
                    const double *l = T + (DB * k + k4) * DLT + o + i4;
                    const double *wkj = k == j ? Wp + (DB * j + k4) * DLW + i4
                                               : T + (DB * k + k4) * DLT + DB * j + i4;
                    const int ws = k == j ? DLW : DLT;
                    dmma(m0, l[0], wkj[0]);
                    dmma(m1, l[4 * DLT], wkj[4 * ws]);
                }
                m0[0] += m1[0];
                m0[1] += m1[1];
                // W_pj = -W_pp M: M from its accumulator lanes into B fragments
                double d[2] = {0.0, 0.0};
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int src = (k4 + 4 * h) * 4 + (i4 >> 1);
                    const double e0 = __shfl_sync(FULL, m0[0], src), e1 = __shfl_sync(FULL, m0[1], src);
                    dmma(d, -Wp[(o + i4) * DLW + k4 + 4 * h], (i4 & 1) ? e1 : e0);
                }
                *reinterpret_cast<double2 *>(T + (o + i4) * DLT + DB * j + 2 * k4) =
                    make_double2(d[0], d[1]);
            }
        }
    }
    __syncthreads();
    double *ablk = A + (long long)c0 * ld + c0;
    for (int idx = tid; idx < w * NB; idx += BLK_THREADS) {
        const int k = idx / NB, r = idx - k * NB;
        if (r < w && r >= k)
            ablk[(long long)k * ld + r] =
                r / DB == k / DB ? L8[(r / DB) * (DB * DB + DB) + (r % DB) * DB + k % DB]
                                 : T[k * DLT + r];
    }
    // W column-major, two rows per 16-byte store
    for (int idx = tid; idx < NB * NB / 2; idx += BLK_THREADS) {
        const int c = idx / (NB / 2), r = 2 * (idx - c * (NB / 2));
        double v[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int rr = r + u;
            v[u] = 0.0;
            if (rr < w && c < w && rr >= c)
                v[u] = rr / DB == c / DB ? Wp[rr * DLW + c % DB] : T[rr * DLT + c];
        }
        reinterpret_cast<double2 *>(Wout)[idx] = make_double2(v[0], v[1]);
    }
}

// L_21 = A_21 W^T for rows r0 + 16 blockIdx.x ... of the outer panel (columns
// c0 .. c0 + 127), written over A_21.  Products by FP64 mma.sync: warp v holds
// columns 8 v .. and 8 (15 - v) .., so that every warp walks 17 blocks of W's
// triangle.  At most 384 rows and on the critical path: few rows per CTA, so
// that loading W is what is left of its time.
//
// Shared memory: Ws[k * LDP + c] = W[c][k] (= Wout, column-major W); Xs[k *
// LDX + r] = A[row r][c0 + k], then the rows of L_21.
__global__ void __launch_bounds__(PANEL_THREADS)
    chol_panel_kernel(double *__restrict__ A, long long ld, int c0, int r0, int m,
                      const double *__restrict__ Wout, const int *skip) {
    if (*(volatile const int *)skip) return;
    extern __shared__ __align__(16) double sm[];
    double *Ws = sm;
    double *Xs = sm + NB * LDP;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rbase = blockIdx.x * PR;
#pragma unroll 8
    for (int idx = tid; idx < NB * NB / 2; idx += PANEL_THREADS) {
        const int k = idx / (NB / 2), c = 2 * (idx - k * (NB / 2));
        if (c + 1 >= k) cp_async(Ws + k * LDP + c, Wout + 2 * idx, 16, true);
        else Ws[k * LDP + c] = Ws[k * LDP + c + 1] = 0.0;
    }
    const double *arows = A + (long long)c0 * ld + r0 + rbase;
#pragma unroll
    for (int idx = tid; idx < NB * PR; idx += PANEL_THREADS) {
        const int k = idx / PR, r = idx - k * PR;
        const bool v = rbase + r < m;
        cp_async(Xs + k * LDX + r, v ? arows + (long long)k * ld + r : arows, 8, v);
    }
    cp_async_wait_all();
    __syncthreads();
    static_assert(PANEL_THREADS / 32 == NB / 16, "two column tiles a warp");
    const int t0 = warp, t1 = NB / 8 - 1 - warp;   // column tiles, t0 < t1
    const int i4 = lane >> 2, k4 = lane & 3;
    double acc[2][PR / 8][2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < PR / 8; ++i) acc[h][i][0] = acc[h][i][1] = 0.0;
    {
        const double *xk = Xs + k4 * LDX + i4, *wk = Ws + k4 * LDP + i4;
        // W[c][k] = 0 for k > c
        for (int k = 0; k < 8 * (t1 + 1); k += 4, xk += 4 * LDX, wk += 4 * LDP) {
            const double b1 = wk[8 * t1];
            double x[PR / 8];
#pragma unroll
            for (int i = 0; i < PR / 8; ++i) x[i] = xk[8 * i];
#pragma unroll
            for (int i = 0; i < PR / 8; ++i) dmma(acc[1][i], x[i], b1);
            if (k < 8 * (t0 + 1)) {
                const double b0 = wk[8 * t0];
#pragma unroll
                for (int i = 0; i < PR / 8; ++i) dmma(acc[0][i], x[i], b0);
            }
        }
    }
    __syncthreads();   // every warp is past its loads of the rows
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < PR / 8; ++i)
#pragma unroll
            for (int u = 0; u < 2; ++u)
                Xs[(8 * (h ? t1 : t0) + 2 * k4 + u) * LDX + 8 * i + i4] = acc[h][i][u];
    __syncthreads();
    for (int idx = tid; idx < NB * PR; idx += PANEL_THREADS) {
        const int c = idx / PR, r = idx - c * PR;
        if (rbase + r < m) A[(long long)(c0 + c) * ld + r0 + rbase + r] = Xs[c * LDX + r];
    }
}

// The rest of the outer panel's diagonal block -= L_21 L_21^T (rows and columns
// r0 .. r0 + m - 1, lower triangle, K = 128) by FP64 mma.sync: one 32 x 32 tile
// per CTA, tile first + blockIdx.x of the triangle by rows (the first ten are
// the next 128-column block).
__global__ void __launch_bounds__(PANEL_THREADS)
    chol_update_kernel(double *__restrict__ A, long long ld, int c0, int r0, int m, int first,
                       const int *skip) {
    if (*(volatile const int *)skip) return;
    extern __shared__ __align__(16) double sm[];
    double *Xi = sm, *Xj = sm + NB * LDU;   // [k][row] of the tile's rows and columns
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int ti = 0, tj = first + blockIdx.x;
    while (tj > ti) tj -= ++ti;
    const int ri = UT * ti, rj = UT * tj;
    const double *src = A + (long long)c0 * ld + r0;
#pragma unroll
    for (int idx = tid; idx < NB * UT; idx += PANEL_THREADS) {
        const int k = idx / UT, r = idx - k * UT;
        const bool vi = ri + r < m, vj = rj + r < m;
        cp_async(Xi + k * LDU + r, vi ? src + (long long)k * ld + ri + r : src, 8, vi);
        cp_async(Xj + k * LDU + r, vj ? src + (long long)k * ld + rj + r : src, 8, vj);
    }
    // D's rows are columns of the tile: a lane's two values are neighbours in memory
    const int i4 = lane >> 2, k4 = lane & 3;
    const int col = 8 * (warp & 3) + i4, row = 16 * (warp >> 2) + 2 * k4;
    double *out = A + (long long)(r0 + rj + col) * ld + r0 + ri + row;
    double old[2][2];
    bool ok[2][2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int r = ri + row + 8 * h + u;
            ok[h][u] = r < m && r >= rj + col;
            old[h][u] = ok[h][u] ? out[8 * h + u] : 0.0;
        }
    cp_async_wait_all();
    __syncthreads();
    double acc[2][2][2] = {};
    const double *xj = Xj + k4 * LDU + col, *xi = Xi + k4 * LDU + 16 * (warp >> 2) + i4;
#pragma unroll 4
    for (int k = 0; k < NB; k += 8) {
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const double a = xj[(k + 4 * v) * LDU];
#pragma unroll
            for (int h = 0; h < 2; ++h) dmma(acc[v][h], a, xi[(k + 4 * v) * LDU + 8 * h]);
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int u = 0; u < 2; ++u)
            if (ok[h][u]) out[8 * h + u] = old[h][u] - (acc[0][h][u] + acc[1][h][u]);
}

// Rows below an outer panel's diagonal block: X L_D^T = A for RT rows of all
// 512 columns per CTA, written over A, with the digit planes and row exponents
// for the trailing updates.  Block column j: X_j = (A_j - sum_{k<j} X_k
// L_jk^T) W_j^T, FP64 mma.sync, the rows resident in shared memory and L_jk,
// W_j streamed through it 16 columns at a time.
//
// Bound by the FP64 rate (RT x 147,456 multiply-adds).  One pass replaces four
// panel solves, three tensor-core updates of the panel's other columns and a
// slicing pass, which had to run one behind the other beside the bulk update.
//
// Xs[k * LDF + r] = A[row r][o0 + k], then X; stage: Bs[k * LDP + c].  Stages
// of 32 columns and fragments one step ahead: with 16 columns, or every
// fragment of a stage loaded before its products, shared-memory loads and
// addressing added 1,000 cycles to the 1,024 of a stage's products (RT = 32).
template <int RT>
struct FarCfg {
    static constexpr int LDF = RT + 4;   // 4 mod 16
    static constexpr int BKF = 32, NST = RT > 16 ? 2 : 4;
    static constexpr size_t SMEM =
        ((size_t)NB2 * LDF + (size_t)NST * BKF * LDP) * sizeof(double);
};

template <int S, int RT>
__global__ void __launch_bounds__(FAR_THREADS)
    chol_far_kernel(double *__restrict__ A, long long ld, int o0, int first, int last, int m,
                    const double *__restrict__ W, int8_t *__restrict__ dpl,
                    int *__restrict__ dex, const int *skip) {
    using C = FarCfg<RT>;
    constexpr int LDF = C::LDF, BKF = C::BKF, NST = C::NST, NC = NB / BKF;
    if (*(volatile const int *)skip) return;
    extern __shared__ __align__(16) double sm[];
    double *Xs = sm, *Bs = sm + NB2 * LDF;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rbase = first + blockIdx.x * RT;
    double *arows = A + (long long)o0 * ld + o0 + NB2 + rbase;
    for (int idx = tid; idx < NB2 * RT; idx += FAR_THREADS) {
        const int k = idx / RT, r = idx - k * RT;
        const bool v = rbase + r < last;
        cp_async(Xs + k * LDF + r, v ? arows + (long long)k * ld + r : arows, 8, v);
    }
    // the stream of chunks: for each j, those of columns 0 .. 128 j - 1 of L's
    // block row j, then those of W_j
    const bool vec = (ld & 1) == 0;
    constexpr int KT = 2 * FAR_THREADS / NB;   // columns a pass of the block's threads (vec)
    const int lk = tid / (NB / 2), lc = 2 * (tid % (NB / 2));
    const double *src_l = A + (long long)(o0 + lk) * ld + o0 + lc, *src_w = W + 2 * tid;
    int lj = 0, lt = 0, ls = 0;
    auto load = [&] {
        if (lj < NB2 / NB) {
            const bool w = lt >= NC * lj;
            const double *src = w ? src_w : src_l + (long long)(lt * BKF) * ld + NB * lj;
            const long long sld = w ? NB : ld;
            double *dst = Bs + ls * BKF * LDP;
            if (vec || w) {
#pragma unroll
                for (int k = 0; k < BKF; k += KT)
                    cp_async(dst + (lk + k) * LDP + lc, src + k * sld, 16, true);
            } else {
                for (int k = 0; k < BKF; k += KT)
                    for (int u = 0; u < 2; ++u)
                        cp_async(dst + (lk + k) * LDP + lc + u, src + k * sld + u, 8, true);
            }
            if (w) src_w += BKF * NB;
            if (++lt == NC * (lj + 1)) {
                lt = 0;
                ++lj;
            }
            ls = ls + 1 == NST ? 0 : ls + 1;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int q = 0; q < NST - 1; ++q) load();
    // warp v: all rows, column tiles v and 15 - v (the same share of a triangle)
    constexpr int RW = RT / 8;
    static_assert(FAR_THREADS / 32 == NB / 16, "two column tiles a warp");
    const int t0 = warp, t1 = NB / 8 - 1 - warp;
    const int i4 = lane >> 2, k4 = lane & 3;
    double acc[2][RW][2];
    auto clear = [&] {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < RW; ++i) acc[h][i][0] = acc[h][i][1] = 0.0;
    };
    // own elements of block column j: Xs = sub ? Xs - acc : acc
    auto put = [&](int j, bool sub) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < RW; ++i)
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    double *x = Xs + (NB * j + 8 * (h ? t1 : t0) + 2 * k4 + u) * LDF + 8 * i + i4;
                    *x = sub ? *x - acc[h][i][u] : acc[h][i][u];
                }
    };
    auto multiply = [&](const double *xk, const double *bk, auto both) {
        constexpr bool BOTH = decltype(both)::value;
        double x[2][RW], b[2][2];
        auto fetch = [&](int k) {
            b[k & 1][1] = bk[4 * k * LDP + 8 * t1];
            if constexpr (BOTH) b[k & 1][0] = bk[4 * k * LDP + 8 * t0];
#pragma unroll
            for (int i = 0; i < RW; ++i) x[k & 1][i] = xk[4 * k * LDF + 8 * i];
        };
        fetch(0);
#pragma unroll
        for (int k = 0; k < BKF / 4; ++k) {
            if (k + 1 < BKF / 4) fetch(k + 1);
#pragma unroll
            for (int i = 0; i < RW; ++i) {
                dmma(acc[1][i], x[k & 1][i], b[k & 1][1]);
                if constexpr (BOTH) dmma(acc[0][i], x[k & 1][i], b[k & 1][0]);
            }
        }
    };
    int st = 0;
    for (int j = 0; j < NB2 / NB; ++j) {
        clear();
        for (int t = 0; t < NC * (j + 1); ++t) {
            const bool w = t >= NC * j;
            if (t == NC * j && j > 0) {
                put(j, true);
                clear();
            }
            asm volatile("cp.async.wait_group %0;" ::"n"(NST - 2) : "memory");
            __syncthreads();   // the chunk has landed, the one before is read, the rows are written
            load();
            // k of the chunk within the block column whose rows it multiplies;
            // W[c][k] = 0 for k > c
            const int k0 = w ? (t - NC * j) * BKF : 0;
            const double *xk = Xs + (t * BKF + k4) * LDF + i4;
            const double *bk = Bs + (st * BKF + k4) * LDP + i4;
            st = st + 1 == NST ? 0 : st + 1;
            if (k0 < 8 * (t0 + 1)) multiply(xk, bk, std::true_type{});
            else if (k0 < 8 * (t1 + 1)) multiply(xk, bk, std::false_type{});
        }
        __syncthreads();   // every warp is past its loads of block column j
        put(j, false);
    }
    __syncthreads();
    for (int idx = tid; idx < NB2 * RT; idx += FAR_THREADS) {
        const int k = idx / RT, r = idx - k * RT;
        if (rbase + r < last) arows[(long long)k * ld + r] = Xs[k * LDF + r];
    }
    // digit planes: a warp per row, lane l holds columns l, l + 32, ...
    const long long plane = (long long)m * NB2;
    for (int rl = warp; rl < RT; rl += FAR_THREADS / 32) {
        const int row = rbase + rl;
        if (row >= last) break;
        double mx = 0.0;
#pragma unroll
        for (int c = 0; c < NB2 / 32; ++c) mx = fmax(mx, fabs(Xs[(lane + 32 * c) * LDF + rl]));
#pragma unroll
        for (int o = 16; o; o >>= 1) mx = fmax(mx, __shfl_xor_sync(FULL, mx, o));
        const int ex = oz_row_exponent(mx);
        if (lane == 0) dex[row] = ex;
        int8_t *d = dpl + (long long)row * NB2 + lane;
#pragma unroll 4
        for (int c = 0; c < NB2 / 32; ++c) {
            int8_t dg[S];
            oz_digits<S>(oz_scale2(Xs[(lane + 32 * c) * LDF + rl], -ex), dg);
#pragma unroll
            for (int s = 0; s < S; ++s) d[s * plane + 32 * c] = dg[s];
        }
    }
}

template <int S, int RT>
kfb_status launch_far(double *A, long long ld, int o0, int first, int rows, int m, const double *W,
                      int8_t *dpl, int *dex, const int *skip, cudaStream_t s) {
    using C = FarCfg<RT>;
    static bool attr = false;
    if (!attr) {
        KFB_CUDA_TRY(cudaFuncSetAttribute(chol_far_kernel<S, RT>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)C::SMEM));
        attr = true;
    }
    chol_far_kernel<S, RT><<<(rows + RT - 1) / RT, FAR_THREADS, C::SMEM, s>>>(
        A, ld, o0, first, first + rows, m, W, dpl, dex, skip);
    KFB_CUDA_TRY(cudaGetLastError());
    return KFB_OK;
}

// Rows first .. first + rows - 1 (of the m below the outer panel at o0), RT per CTA.
template <int RT>
kfb_status far_rows(int S, double *A, long long ld, int o0, int first, int rows, int m,
                    const double *W, int8_t *dpl, int *dex, const int *skip, cudaStream_t s) {
    switch (S) {
        case 2: return launch_far<2, RT>(A, ld, o0, first, rows, m, W, dpl, dex, skip, s);
        case 3: return launch_far<3, RT>(A, ld, o0, first, rows, m, W, dpl, dex, skip, s);
        case 4: return launch_far<4, RT>(A, ld, o0, first, rows, m, W, dpl, dex, skip, s);
        case 5: return launch_far<5, RT>(A, ld, o0, first, rows, m, W, dpl, dex, skip, s);
        case 6: return launch_far<6, RT>(A, ld, o0, first, rows, m, W, dpl, dex, skip, s);
        case 7: return launch_far<7, RT>(A, ld, o0, first, rows, m, W, dpl, dex, skip, s);
        default: return set_error(KFB_ERR_INVALID_ARG, "digit planes S=%d", S);
    }
}

}  // namespace

namespace {

// The streams of the look-ahead, per device: the critical path (diagonal
// blocks, the rows and updates the next ones wait for) at the highest priority,
// the rest of a diagonal block's updates beside it, the rows below and the next
// panel's columns after that, the bulk trailing updates at the lowest.
struct CholStreams {
    cudaStream_t crit = nullptr, near = nullptr, far = nullptr, bulk = nullptr;
};

kfb_status chol_streams(CholStreams *&out) {
    static CholStreams per_dev[16];
    int dev = 0;
    KFB_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 16) return set_error(KFB_ERR_UNSUPPORTED, "device index %d", dev);
    CholStreams &cs = per_dev[dev];
    if (!cs.crit) {
        int least = 0, greatest = 0;
        KFB_CUDA_TRY(cudaDeviceGetStreamPriorityRange(&least, &greatest));
        KFB_CUDA_TRY(cudaStreamCreateWithPriority(&cs.crit, cudaStreamNonBlocking, greatest));
        KFB_CUDA_TRY(cudaStreamCreateWithPriority(&cs.near, cudaStreamNonBlocking,
                                                  std::min(greatest + 1, least)));
        KFB_CUDA_TRY(cudaStreamCreateWithPriority(&cs.far, cudaStreamNonBlocking,
                                                  std::min(greatest + 2, least)));
        KFB_CUDA_TRY(cudaStreamCreateWithPriority(&cs.bulk, cudaStreamNonBlocking, least));
    }
    out = &cs;
    return KFB_OK;
}

// Events of one factorisation, destroyed with it.
struct CholEvents {
    cudaEvent_t ev[12] = {};
    kfb_status init() {
        for (auto &e : ev) KFB_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        return KFB_OK;
    }
    ~CholEvents() {
        for (auto &e : ev)
            if (e) cudaEventDestroy(e);
    }
};

}  // namespace

kfb_status chol_dense(double *A, int n, long long ld, int slices, int *info, cudaStream_t s) {
    *info = 0;
    if (n <= 0) return KFB_OK;
    if (slices < 2 || slices > OZ_MAXS)
        return set_error(KFB_ERR_INVALID_ARG, "Cholesky digit planes %d outside 2..%d", slices,
                         OZ_MAXS);
    static bool attr = false;
    if (!attr) {
        KFB_CUDA_TRY(cudaFuncSetAttribute(chol_block64_kernel,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)DBLK_SMEM));
        KFB_CUDA_TRY(cudaFuncSetAttribute(chol_block_kernel,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)BLK_SMEM));
        KFB_CUDA_TRY(cudaFuncSetAttribute(chol_panel_kernel,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)PANEL_SMEM));
        KFB_CUDA_TRY(cudaFuncSetAttribute(chol_update_kernel,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)UPD_SMEM));
        attr = true;
    }
    // the diagonal blocks in FP32 for an FP32-class factor (4 or fewer planes)
    const bool f32blk = slices <= 4;
    CholStreams *cs = nullptr;
    KFB_TRY(chol_streams(cs));
    const cudaStream_t sc = cs->crit, sn = cs->near, sf = cs->far, sb = cs->bulk;
    CholEvents E;
    KFB_TRY(E.init());
    cudaEvent_t ev_start = E.ev[0], ev_panel = E.ev[1], ev_near = E.ev[2], ev_diag = E.ev[3],
                ev_rows = E.ev[4], ev_far = E.ev[5], ev_next = E.ev[6], ev_bulk = E.ev[7];
    cudaEvent_t ev_free[2] = {E.ev[8], E.ev[9]};   // the bulk update has read these digit planes
    cudaEvent_t ev_end = E.ev[10], ev_bulk_end = E.ev[11];
    // everything below is ordered after the caller's work on s
    KFB_CUDA_TRY(cudaEventRecord(ev_start, s));
    KFB_CUDA_TRY(cudaStreamWaitEvent(sc, ev_start, 0));
    // flags: [0] info, [1] skip, [2] GEMM pipeline error
    DevBuf flags, Wd, osl[2], oex[2];
    KFB_TRY(flags.alloc(4 * sizeof(int), sc));
    KFB_TRY(zero(flags.ptr, 4 * sizeof(int), sc));
    int *d_info = flags.as<int>(), *d_skip = d_info + 1, *d_err = d_info + 2;
    // inverted diagonal blocks of two outer panels
    KFB_TRY(Wd.alloc((size_t)2 * NB2 * NB * sizeof(double), sc));
    if (n > NB2)
        for (int b = 0; b < 2; ++b) {
            KFB_TRY(osl[b].alloc((size_t)slices * (n - NB2) * NB2, sc));
            KFB_TRY(oex[b].alloc((size_t)(n - NB2) * sizeof(int), sc));
        }
    // on an early (error) return, let the streams finish before the buffers
    // above are released (destroyed after this guard)
    struct Drain {
        cudaStream_t st[4];
        bool armed = true;
        ~Drain() {
            if (armed)
                for (cudaStream_t t : st) cudaStreamSynchronize(t);
        }
    } drain{{sc, sn, sf, sb}};
    OzEpi epi;
    epi.c = A;
    epi.ldr = 1;
    epi.ldc = ld;
    epi.skip = d_skip;
    epi.mode = OZ_ADD;
    epi.alpha = -1.0;
    epi.tiles_per_cta = 1;
    OzEpi epi_bulk = epi;
    epi_bulk.tiles_per_cta = BULK_TILES;
    bool next_pending = false;   // the columns of this outer panel below its diagonal block
    bool bulk_pending = false;   // a bulk update of later columns
    for (int o0 = 0, P = 0; o0 < n; o0 += NB2, ++P) {
        const int ow = std::min(NB2, n - o0);   // outer panel: columns o0 .. o0 + ow - 1
        double *W = Wd.as<double>() + (size_t)(P & 1) * NB2 * NB;
        // ---- its ow x ow diagonal block
        bool near_pending = false;   // the rest of an update within it
        for (int c0 = o0; c0 < o0 + ow; c0 += NB) {
            const int w = std::min(NB, n - c0);
            const int r0 = c0 + w, m = o0 + ow - r0;
            double *Wj = W + (size_t)((c0 - o0) / NB) * NB * NB;
            if (f32blk)
                chol_block_kernel<<<1, BLK_THREADS, BLK_SMEM, sc>>>(A, ld, c0, w, Wj, d_info,
                                                                    d_skip);
            else
                chol_block64_kernel<<<1, BLK_THREADS, DBLK_SMEM, sc>>>(A, ld, c0, w, Wj, d_info,
                                                                       d_skip);
            KFB_CUDA_TRY(cudaGetLastError());
            // (the block itself was updated ahead of the rest of its columns)
            if (near_pending) KFB_CUDA_TRY(cudaStreamWaitEvent(sc, ev_near, 0));
            near_pending = false;
            if (m == 0) break;
            chol_panel_kernel<<<(m + PR - 1) / PR, PANEL_THREADS, PANEL_SMEM, sc>>>(A, ld, c0, r0, m,
                                                                                   Wj, d_skip);
            KFB_CUDA_TRY(cudaGetLastError());
            // the next 128 x 128 block first, the rest beside its factorisation
            const int nt = (m + UT - 1) / UT, all = nt * (nt + 1) / 2;
            const int head = std::min(all, (NB / UT) * (NB / UT + 1) / 2);
            if (all > head) {
                KFB_CUDA_TRY(cudaEventRecord(ev_panel, sc));
                KFB_CUDA_TRY(cudaStreamWaitEvent(sn, ev_panel, 0));
                chol_update_kernel<<<all - head, PANEL_THREADS, UPD_SMEM, sn>>>(A, ld, c0, r0, m,
                                                                               head, d_skip);
                KFB_CUDA_TRY(cudaGetLastError());
                KFB_CUDA_TRY(cudaEventRecord(ev_near, sn));
                near_pending = true;
            }
            chol_update_kernel<<<head, PANEL_THREADS, UPD_SMEM, sc>>>(A, ld, c0, r0, m, 0, d_skip);
            KFB_CUDA_TRY(cudaGetLastError());
        }
        const int R = o0 + ow, M = n - R;
        if (M <= 0) break;
        // ---- the rows below: those of the next diagonal block on the critical
        // stream, the rest on the far one
        OzSlices O;
        O.d = osl[P & 1].as<int8_t>();
        O.e = oex[P & 1].as<int>();
        O.S = slices;
        O.rows = M;
        O.kp = NB2;
        const int na = std::min(NB2, M);
        if (P >= 2) KFB_CUDA_TRY(cudaStreamWaitEvent(sc, ev_free[P & 1], 0));
        KFB_CUDA_TRY(cudaEventRecord(ev_diag, sc));
        if (next_pending) KFB_CUDA_TRY(cudaStreamWaitEvent(sc, ev_next, 0));
        KFB_TRY(far_rows<8>(slices, A, ld, o0, 0, na, M, W, O.d, O.e, d_skip, sc));
        KFB_CUDA_TRY(cudaEventRecord(ev_rows, sc));
        // ---- the next diagonal block -= L L^T (K = 512); the last bulk update
        // wrote it too
        OzGen g;
        g.mode = OZ_GEN_LOWER;
        g.M = g.N = na;
        g.c_off = (long long)R * ld + R;
        if (bulk_pending) KFB_CUDA_TRY(cudaStreamWaitEvent(sc, ev_bulk, 0));
        KFB_TRY(oz_gemm_gen(O, O, g, epi, d_err, sc));
        next_pending = M > na;
        if (M <= na) continue;
        KFB_CUDA_TRY(cudaStreamWaitEvent(sf, ev_diag, 0));
        KFB_TRY(far_rows<32>(slices, A, ld, o0, na, M - na, M, W, O.d, O.e, d_skip, sf));
        KFB_CUDA_TRY(cudaEventRecord(ev_far, sf));
        // the next outer panel's columns below its diagonal block
        KFB_CUDA_TRY(cudaStreamWaitEvent(sf, ev_rows, 0));
        if (bulk_pending) KFB_CUDA_TRY(cudaStreamWaitEvent(sf, ev_bulk, 0));
        g.mode = OZ_GEN_RECT;
        g.M = M - na;
        g.a_base = na;
        g.c_off += na;
        KFB_TRY(oz_gemm_gen(O, O, g, epi, d_err, sf));
        KFB_CUDA_TRY(cudaEventRecord(ev_next, sf));
        // everything right of them: the columns of the outer panel after the
        // next one first, which is all that the other streams wait for
        KFB_CUDA_TRY(cudaStreamWaitEvent(sb, ev_far, 0));
        g.mode = OZ_GEN_LOWER;
        for (int c = na; c < M; c = c == na && M > na + NB2 ? na + NB2 : M) {
            g.M = M - c;
            g.N = c == na ? std::min(NB2, M - na) : M - c;
            g.a_base = g.b_base = c;
            g.c_off = (long long)(R + c) * ld + (R + c);
            KFB_TRY(oz_gemm_gen(O, O, g, epi_bulk, d_err, sb));
            if (c == na) KFB_CUDA_TRY(cudaEventRecord(ev_bulk, sb));
        }
        KFB_CUDA_TRY(cudaEventRecord(ev_free[P & 1], sb));
        bulk_pending = true;
    }
    // join the streams back into the caller's (the near stream has been waited
    // for; the far one by the critical one)
    KFB_CUDA_TRY(cudaEventRecord(ev_end, sc));
    KFB_CUDA_TRY(cudaStreamWaitEvent(s, ev_end, 0));
    if (bulk_pending) {
        KFB_CUDA_TRY(cudaEventRecord(ev_bulk_end, sb));
        KFB_CUDA_TRY(cudaStreamWaitEvent(s, ev_bulk_end, 0));
    }
    int h[3] = {0, 0, 0};
    KFB_CUDA_TRY(cudaMemcpyAsync(h, d_info, 3 * sizeof(int), cudaMemcpyDeviceToHost, s));
    KFB_CUDA_TRY(cudaStreamSynchronize(s));
    drain.armed = false;   // the streams joined into s, which is idle now
    if (h[2]) return set_error(KFB_ERR_TIMEOUT, "Cholesky: a tensor-core pipeline wait timed out");
    *info = h[0];
    return KFB_OK;
}

}  // namespace kfb
