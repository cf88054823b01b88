// Triangular solves with one right-hand side against a dense FP64 Cholesky
// factor (column-major lower L, leading dimension n): x = (L L^T)^{-1} b as
// L t = b, then L^T x = t.  This is the preconditioner application of the
// refinement loop of the KRR solve; the library call it replaces
// (potrs -> two trsm with one column) walks the factor in dependent column
// panels and ran at about a quarter of the factor's read bandwidth.
//
// Design (64-row blocks, nb = ceil(n / 64)):
//  * the 64 x 64 diagonal blocks are inverted once per factor (block per
//    diagonal block, thread per column), so the solve of a block is a
//    matrix-vector product instead of 64 dependent steps;
//  * one persistent cooperative kernel per direction; block I is owned by CTA
//    I mod grid.  Its CTA accumulates the off-diagonal tiles against the
//    solution blocks as they are published and then applies the inverted
//    diagonal block.  Blocks finish in solve order (block I needs block I-1);
//    that chain, not the factor's bytes, is what bounds the sweep;
//  * the solution vector is its own flag: it is filled with a bit pattern that
//    no result has, and a thread polls the very element that it stages, so a
//    step of the chain has one store and one load in flight (1.6 and 1.5 us a
//    block in the two sweeps of n = 10,000; with a counter published behind a
//    fence and the block read after it 2.4 and 3.1 us);
//  * every wait is bounded: after TRSV_WAIT_NS a thread raises *err and all
//    CTAs leave; the host reads *err once per solve sequence.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels_common.cuh"
#include "trsv.h"

namespace kfb {

namespace {

constexpr int TB = 64;                  // rows per block
constexpr int TRSV_THREADS = 256;       // 64 rows x 4 column groups
constexpr int TB_BATCH = TRSV_THREADS / TB;   // solution blocks staged at once
constexpr unsigned long long TRSV_WAIT_NS = 1000000000ull;   // one second of %globaltimer

// An element that is not published yet: all bits set (a NaN; a result with
// these bits is published as another NaN).
constexpr unsigned long long UNPUBLISHED = ~0ull;

__device__ __forceinline__ bool ld_published(const double *p, double &v) {
    unsigned long long b;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(b) : "l"(p) : "memory");
    v = __longlong_as_double((long long)b);
    return b != UNPUBLISHED;
}

__device__ __forceinline__ void publish(double *p, double v) {
    unsigned long long b = (unsigned long long)__double_as_longlong(v);
    if (b == UNPUBLISHED) b = 0x7ff8000000000000ull;
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(b) : "memory");
}

__device__ __forceinline__ unsigned long long trsv_clock_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Wait for an element; false when the wait gave up (or another CTA gave up).
// The limit is elapsed time on %globaltimer (one second), not a poll count.
__device__ bool wait_published(const double *p, double &v, int *err) {
    for (int i = 0; i < 64; ++i)
        if (ld_published(p, v)) return true;
    const unsigned long long t0 = trsv_clock_ns();
    while (true) {
        for (int i = 0; i < 16; ++i)
            if (ld_published(p, v)) return true;
        if (*reinterpret_cast<volatile int *>(err)) return false;
        if (trsv_clock_ns() - t0 > TRSV_WAIT_NS) break;
    }
    atomicExch(err, 1);
    return false;
}

// Stage up to TB_BATCH solution blocks, thread (r, g) element r of the g-th: it
// is at p (valid: it exists and nblk > g; else the element counts as a zero that
// is there).  The first block is waited for, the others are taken if they are
// there.  Returns the number of leading blocks in xs, -1 when a wait gave up.
__device__ __forceinline__ int stage_blocks(const double *p, bool valid, int nblk, double *xs,
                                            int *state, int *err) {
    const int t = threadIdx.x, g = t / TB;
    double v = 0.0;
    bool ok = true, fail = false;
    if (valid) {
        ok = ld_published(p, v);
        if (!ok && g == 0) {
            ok = wait_published(p, v, err);
            fail = !ok;
        }
    }
    xs[t] = v;
    const bool all = __all_sync(0xffffffffu, ok), bad = __any_sync(0xffffffffu, fail);
    if ((t & 31) == 0) state[t >> 5] = bad ? -1 : all;
    __syncthreads();
    if (state[0] < 0 || state[1] < 0) return -1;
    int d = 1;
    while (d < nblk && state[2 * d] > 0 && state[2 * d + 1] > 0) ++d;
    return d;
}

// Inverse of each 64 x 64 lower diagonal block: dinv[I] column-major
// (dinv[I][r + 64 c] = (L_II^{-1})[r][c]) and dinvt[I] its transpose;
// rows/columns beyond n are the identity.
__global__ void __launch_bounds__(TB) trsv_dinv_kernel(const double *__restrict__ L, int n,
                                                      double *__restrict__ dinv,
                                                      double *__restrict__ dinvt) {
    __shared__ double a[TB][TB + 1];   // a[r][c] = L_II[r][c]
    const int I = blockIdx.x, i0 = I * TB, m = min(TB, n - i0);
    const int c = threadIdx.x;
    for (int r = 0; r < TB; ++r)
        a[r][c] = (r < m && c < m && r >= c) ? L[(size_t)(i0 + r) + (size_t)(i0 + c) * n] : 0.0;
    __syncthreads();
    // column c of the inverse by forward substitution on e_c, kept in dinv
    double *zc = dinv + (size_t)I * TB * TB + (size_t)TB * c;
    for (int r = 0; r < TB; ++r) zc[r] = (r == c && c >= m) ? 1.0 : 0.0;
    if (c < m) {
        zc[c] = 1.0 / a[c][c];
        for (int r = c + 1; r < m; ++r) {
            double s = 0.0;
            for (int j = c; j < r; ++j) s = fma(a[r][j], zc[j], s);
            zc[r] = -s / a[r][r];
        }
    }
    __syncthreads();
    const double *d = dinv + (size_t)I * TB * TB;
    double *dt = dinvt + (size_t)I * TB * TB;
    for (int r = 0; r < TB; ++r) dt[r + TB * c] = d[c + TB * r];   // transpose
}

// L t = b.  Thread (r = t & 63, g = t >> 6) accumulates row r over the
// columns c = g, g + 4, ... of each tile.  Before its first wait a CTA issues
// the loads of what the critical step needs (the inverted diagonal block into
// shared memory, the tile of the block just before it into registers), so
// that once block I-1 is published only x_{I-1} is fetched.
__global__ void __launch_bounds__(TRSV_THREADS) trsv_lower_kernel(
    const double *__restrict__ L, int n, int nb, const double *__restrict__ dinv,
    const double *__restrict__ b, double *t_out, int *err) {
    __shared__ double xs[2][TB_BATCH * TB];   // (two: a batch is staged while the last is read)
    __shared__ int state[2][TRSV_THREADS / 32];
    __shared__ double rhs[TB];
    __shared__ double red[2][4][TB];
    __shared__ double dsm[TB * TB];
    const int t = threadIdx.x, r = t & (TB - 1), g = t >> 6;
    int buf = 0;
    for (int I = blockIdx.x; I < nb; I += gridDim.x) {
        const int i0 = I * TB, row = i0 + r;
        const bool rv = row < n;
        __syncthreads();   // dsm of the previous block consumed
        for (int e = t; e < TB * TB; e += TRSV_THREADS) dsm[e] = dinv[(size_t)I * TB * TB + e];
        double lvl[TB / 4];   // tile (I, I-1)
#pragma unroll
        for (int k = 0; k < TB / 4; ++k)
            lvl[k] = (rv && I > 0) ? L[(size_t)row + (size_t)((I - 1) * TB + g + 4 * k) * n] : 0.0;
        const double bv = t < TB && rv ? b[row] : 0.0;
        double acc = 0.0;
        for (int J = 0; J < I;) {
            // (blocks before I are full)
            const int nblk = min(TB_BATCH, I - J);
            const int d = stage_blocks(t_out + (size_t)J * TB + t, g < nblk, nblk, xs[buf],
                                       state[buf], err);
            if (d < 0) return;
            for (int jj = J; jj < J + d; ++jj) {
                const double *xv = xs[buf] + (jj - J) * TB;
                if (jj == I - 1) {
#pragma unroll
                    for (int k = 0; k < TB / 4; ++k) acc = fma(lvl[k], xv[g + 4 * k], acc);
                    continue;
                }
                const double *col = L + (size_t)row + (size_t)jj * TB * n;
                double lv[TB / 4];
#pragma unroll
                for (int k = 0; k < TB / 4; ++k)
                    lv[k] = rv ? col[(size_t)(g + 4 * k) * n] : 0.0;
#pragma unroll
                for (int k = 0; k < TB / 4; ++k) acc = fma(lv[k], xv[g + 4 * k], acc);
            }
            buf ^= 1;
            J += d;
        }
        red[0][g][r] = acc;
        __syncthreads();
        if (t < TB) rhs[t] = bv - (red[0][0][t] + red[0][1][t] + red[0][2][t] + red[0][3][t]);
        __syncthreads();
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < TB / 4; ++k) s = fma(dsm[r + TB * (g + 4 * k)], rhs[g + 4 * k], s);
        red[1][g][r] = s;
        __syncthreads();
        if (t < TB && rv)
            publish(t_out + row, red[1][0][t] + red[1][1][t] + red[1][2][t] + red[1][3][t]);
    }
}

// L^T x = t, blocks in reverse order (rank q = nb - 1 - I is the publication
// order).  Thread (r, g) accumulates, for the columns c = g, g + 4, ... of
// block I, L[j0 + r][i0 + c] x[j0 + r] over the later blocks J; the row
// partials of each column are summed by warp shuffles and across the two
// warps of a column group.  Prefetches as in the forward sweep (tile of block
// I+1, the transposed inverse of the diagonal block).
__global__ void __launch_bounds__(TRSV_THREADS) trsv_upper_kernel(
    const double *__restrict__ L, int n, int nb, const double *__restrict__ dinvt,
    const double *__restrict__ tv, double *x, int *err) {
    __shared__ double xs[2][TB_BATCH * TB];
    __shared__ int state[2][TRSV_THREADS / 32];
    __shared__ double rhs[TB];
    __shared__ double red[2][TB];   // [half of the rows][column]
    __shared__ double sums[4][TB];
    __shared__ double dsm[TB * TB];
    const int t = threadIdx.x, r = t & (TB - 1), g = t >> 6;
    const int lane = t & 31, half = r >> 5;
    int buf = 0;
    for (int q = blockIdx.x; q < nb; q += gridDim.x) {
        const int I = nb - 1 - q, i0 = I * TB;
        __syncthreads();   // dsm of the previous block consumed
        for (int e = t; e < TB * TB; e += TRSV_THREADS) dsm[e] = dinvt[(size_t)I * TB * TB + e];
        double lvl[TB / 4];   // tile (I+1, I)
        {
            const int j = (I + 1) * TB + r;
            const bool jv = q > 0 && j < n;
#pragma unroll
            for (int k = 0; k < TB / 4; ++k)
                lvl[k] = jv ? L[(size_t)j + (size_t)(i0 + g + 4 * k) * n] : 0.0;
        }
        const double bv = t < TB && i0 + t < n ? tv[i0 + t] : 0.0;
        double acc[TB / 4];
#pragma unroll
        for (int k = 0; k < TB / 4; ++k) acc[k] = 0.0;
        // later blocks J = nb - 1 - p for published ranks p < q
        for (int p = 0; p < q;) {
            const int nblk = min(TB_BATCH, q - p);
            const int je = (nb - 1 - p - g) * TB + r;   // (the last block may be partial)
            const int d = stage_blocks(x + je, g < nblk && je < n, nblk, xs[buf], state[buf], err);
            if (d < 0) return;
            for (int pp = p; pp < p + d; ++pp) {
                const double xr = xs[buf][(pp - p) * TB + r];
                if (pp == q - 1) {   // block I+1
#pragma unroll
                    for (int k = 0; k < TB / 4; ++k) acc[k] = fma(lvl[k], xr, acc[k]);
                    continue;
                }
                const int j = (nb - 1 - pp) * TB + r;
                const bool jv = j < n;
                const double *rowp = L + (size_t)j + (size_t)i0 * n;
                double lv[TB / 4];
#pragma unroll
                for (int k = 0; k < TB / 4; ++k) lv[k] = jv ? rowp[(size_t)(g + 4 * k) * n] : 0.0;
#pragma unroll
                for (int k = 0; k < TB / 4; ++k) acc[k] = fma(lv[k], xr, acc[k]);
            }
            buf ^= 1;
            p += d;
        }
        // sum over the lanes, halving the columns that a lane holds: lane l ends
        // with column 4 (l >> 1) + g
#pragma unroll
        for (int o = 16, len = TB / 8; o > 1; o >>= 1, len >>= 1) {
            const bool up = lane & o;
#pragma unroll
            for (int k = 0; k < len; ++k) {
                const double send = up ? acc[k] : acc[k + len];
                acc[k] = (up ? acc[k + len] : acc[k]) + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
        acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
        if ((lane & 1) == 0) red[half][g + 4 * (lane >> 1)] = acc[0];
        __syncthreads();
        if (t < TB) rhs[t] = bv - (red[0][t] + red[1][t]);
        __syncthreads();
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < TB / 4; ++k) s = fma(dsm[r + TB * (g + 4 * k)], rhs[g + 4 * k], s);
        sums[g][r] = s;
        __syncthreads();
        if (t < TB && i0 + t < n)
            publish(x + i0 + t, sums[0][t] + sums[1][t] + sums[2][t] + sums[3][t]);
    }
}

}  // namespace

kfb_status TrsvPlan::prepare(const double *L, int n_, cudaStream_t s) {
    n = n_;
    nb = (n + TB - 1) / TB;
    if (n <= 0) return KFB_OK;
    KFB_TRY(dinv.alloc((size_t)nb * TB * TB * sizeof(double), s));
    KFB_TRY(dinvt.alloc((size_t)nb * TB * TB * sizeof(double), s));
    KFB_TRY(sync.alloc(sizeof(int), s));
    KFB_TRY(zero(sync.ptr, sizeof(int), s));
    trsv_dinv_kernel<<<nb, TB, 0, s>>>(L, n, dinv.as<double>(), dinvt.as<double>());
    KFB_CUDA_TRY(cudaGetLastError());
    int dev = 0, sms = 0, coop = 0, per_sm_l = 0, per_sm_u = 0;
    KFB_CUDA_TRY(cudaGetDevice(&dev));
    KFB_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    KFB_CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop)
        return set_error(KFB_ERR_UNSUPPORTED, "the triangular solve needs cooperative launches");
    KFB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_l, trsv_lower_kernel,
                                                               TRSV_THREADS, 0));
    KFB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_u, trsv_upper_kernel,
                                                               TRSV_THREADS, 0));
    grid = std::min(nb, sms * std::max(1, std::min(per_sm_l, per_sm_u)));
    return KFB_OK;
}

kfb_status TrsvPlan::solve(const double *L, const double *b, double *tmp, double *x,
                           cudaStream_t s) {
    if (n <= 0) return KFB_OK;
    int *err = sync.as<int>();
    KFB_CUDA_TRY(cudaMemsetAsync(tmp, 0xff, (size_t)n * sizeof(double), s));   // unpublished
    const double *dl = dinv.as<double>(), *du = dinvt.as<double>();
    void *args_l[] = {(void *)&L, (void *)&n, (void *)&nb, (void *)&dl, (void *)&b,
                      (void *)&tmp, (void *)&err};
    KFB_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)trsv_lower_kernel, dim3(grid),
                                             dim3(TRSV_THREADS), args_l, 0, s));
    // (x may be b, which the forward sweep reads)
    KFB_CUDA_TRY(cudaMemsetAsync(x, 0xff, (size_t)n * sizeof(double), s));
    const double *tc = tmp;
    void *args_u[] = {(void *)&L, (void *)&n, (void *)&nb, (void *)&du, (void *)&tc,
                      (void *)&x, (void *)&err};
    KFB_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)trsv_upper_kernel, dim3(grid),
                                             dim3(TRSV_THREADS), args_u, 0, s));
    return KFB_OK;
}

kfb_status TrsvPlan::check(cudaStream_t s) {
    if (n <= 0) return KFB_OK;
    int e = 0;
    KFB_CUDA_TRY(cudaMemcpyAsync(&e, sync.as<int>(), sizeof(int), cudaMemcpyDeviceToHost, s));
    KFB_CUDA_TRY(cudaStreamSynchronize(s));
    if (e != 0)
        return set_error(KFB_ERR_TIMEOUT, "triangular solve: a block wait gave up");
    return KFB_OK;
}

}  // namespace kfb
