// Device code of the scalar kernels without a split (FP64 on mma.sync tiles, FP32
// on CUDA cores), shared by the
// launchers in scalar_simt.cu and scalar_noalloc.cu.
#pragma once

#include "kernels_common.cuh"

namespace kfb {
namespace simt {

constexpr int ST = 64;    // tile edge (rows of A and of B)
constexpr int SK = 16;    // K chunk staged in shared memory
constexpr int SPAD = 1;

// Packed rows, their squared norms and molecules.  With `pos` (packed place of every
// column per label, pack_columns_kernel), only the label's used columns are
// stored; zeros follow up to the next multiple of SK.  The norm is over every
// column; a row with a value that is not finite in a column that is not stored
// has an undefined norm, as its products with that column's zeros would have been.
template <class Tin, class T>
__global__ void pack_rows_kernel(const Tin *__restrict__ x, const int *__restrict__ src, int R,
                                 int rep, int Dp, const int *__restrict__ lab_start, int L,
                                 const int *__restrict__ pos, const int *__restrict__ ncols, int ma,
                                 T *__restrict__ out, T *__restrict__ norm,
                                 int *__restrict__ mol) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= R) return;
    int l = 0;
    while (pos && l + 1 < L && warp >= lab_start[l + 1]) ++l;
    const Tin *xr = x + (size_t)src[warp] * rep;
    const int *pl = pos ? pos + (size_t)l * rep : nullptr;
    T *orow = out + (size_t)warp * Dp;
    double s = 0.0;
    bool bad = false;
    for (int k = lane; k < rep; k += 32) {
        const double v = (double)xr[k];
        const int p = pl ? pl[k] : k;
        if (p >= 0) orow[p] = (T)v;
        bad |= p < 0 && !isfinite(v);
        s += v * v;
    }
    bad = __any_sync(0xffffffffu, bad);
    const int n = pl ? ncols[l] : rep;
    for (int p = n + lane; p < (n + SK - 1) / SK * SK; p += 32) orow[p] = T(0);
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
        norm[warp] = (T)(bad ? s - s : s);
        mol[warp] = src[warp] / ma;
    }
}

// Sums of the tile E (ST x ST, zero outside the valid part) over (molecule
// a) x (molecule b) rectangles, one atomic add each.  Every thread of the block.
template <class T>
__device__ __forceinline__ void tile_rectangles(T (*E)[ST + SPAD], const PairTile &t, int nra,
                                                int nrb, const int *__restrict__ molA,
                                                const int *__restrict__ molB,
                                                const PairSink &sink) {
    __shared__ int rmol[ST], cmol[ST];
    __shared__ int rstart[ST + 1], cstart[ST + 1];
    __shared__ int nrun_r, nrun_c;
    const int tid = threadIdx.x;
    if (tid < ST) rmol[tid] = tid < nra ? molA[t.a0 + tid] : -1;
    else if (tid < 2 * ST) cmol[tid - ST] = (tid - ST) < nrb ? molB[t.b0 + tid - ST] : -1;
    __syncthreads();   // (E is complete too)
    // molecule runs along rows and columns
    if (tid == 0) {
        int k = 0;
        for (int r = 0; r < nra; ++r)
            if (r == 0 || rmol[r] != rmol[r - 1]) rstart[k++] = r;
        rstart[k] = nra;
        nrun_r = k;
    } else if (tid == 32) {
        int k = 0;
        for (int c = 0; c < nrb; ++c)
            if (c == 0 || cmol[c] != cmol[c - 1]) cstart[k++] = c;
        cstart[k] = nrb;
        nrun_c = k;
    }
    __syncthreads();
    const int nr = nrun_r, nc = nrun_c;
    for (int p = tid; p < nr * nc; p += blockDim.x) {
        const int ri = p / nc, ci = p - ri * nc;
        const int r0 = rstart[ri], r1 = rstart[ri + 1];
        const int c0 = cstart[ci], c1 = cstart[ci + 1];
        T s = T(0);
        for (int r = r0; r < r1; ++r)
            for (int c = c0; c < c1; ++c) s += E[r][c];
        emit_pair(sink, rmol[r0], cmol[c0], (double)s, t.diag);
    }
}

// 128 threads: thread (ty = tid / 16, tx = tid % 16) owns rows 8 ty .. 8 ty + 7
// and columns 4 tx .. 4 tx + 3 of the 64 x 64 tile (12 shared loads per 32
// FMAs in the K loop).
constexpr int SIMT_THREADS = 128;

template <class T>
__global__ void __launch_bounds__(SIMT_THREADS) scalar_tile_kernel(
    const T *__restrict__ A, const T *__restrict__ B, int Dp, const int *__restrict__ ncols,
    const T *__restrict__ nA, const T *__restrict__ nB, const int *__restrict__ molA,
    const int *__restrict__ molB, const PairTile *__restrict__ tiles, T coef, PairSink sink) {
    // the staging tiles of the K loop and the e_ij tile of the epilogue share
    // one shared-memory buffer
    constexpr int STAGE_ELEMS = 2 * SK * (ST + SPAD), E_ELEMS = ST * (ST + SPAD);
    __shared__ T smem_buf[STAGE_ELEMS > E_ELEMS ? STAGE_ELEMS : E_ELEMS];
    T (*As)[ST + SPAD] = reinterpret_cast<T (*)[ST + SPAD]>(smem_buf);
    T (*Bs)[ST + SPAD] = reinterpret_cast<T (*)[ST + SPAD]>(smem_buf + SK * (ST + SPAD));
    T (*E)[ST + SPAD] = reinterpret_cast<T (*)[ST + SPAD]>(smem_buf);

    const PairTile t = tiles[blockIdx.x];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;   // ty < 8
    const int nra = min(ST, t.a_end - t.a0);
    const int nrb = min(ST, t.b_end - t.b0);

    T acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = T(0);

    const int lr = tid >> 1, lk = (tid & 1) * 8;  // loader: row, first k
    const int K = ncols ? (ncols[t.lab] + SK - 1) / SK * SK : Dp;
    for (int k0 = 0; k0 < K; k0 += SK) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int k = k0 + lk + u;
            As[lk + u][lr] = (lr < nra && k < Dp) ? A[(size_t)(t.a0 + lr) * Dp + k] : T(0);
            Bs[lk + u][lr] = (lr < nrb && k < Dp) ? B[(size_t)(t.b0 + lr) * Dp + k] : T(0);
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < SK; ++kk) {
            T a[8], b[4];
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = As[kk][ty * 8 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }

    // e_ij into shared memory (zero outside the valid rows / columns)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = ty * 8 + i;
        const T ni = r < nra ? nA[t.a0 + r] : T(0);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = tx * 4 + j;
            T v = T(0);
            if (r < nra && c < nrb) {
                const T d2 = ni + nB[t.b0 + c] - T(2) * acc[i][j];
                v = kexp<T>(coef * d2);
            }
            E[r][c] = v;
        }
    }
    tile_rectangles<T>(E, t, nra, nrb, molA, molB, sink);
}

// FP64 tiles on mma.sync: 128 threads, warp (wm, wn) owns rows 32 wm .. and
// columns 32 wn .. of the 64 x 64 tile as 4 x 4 products of 8 x 8 (8 shared
// loads per 16 products of 256 FMAs; the CUDA-core tile needs 12 loads per 32
// FMAs and was bound by them).  K slices of 16 come by cp.async into two
// buffers; rows of 20 doubles put the fragment loads of a half warp on 16
// different banks.
constexpr int DM_LD = SK + 4;

__device__ __forceinline__ void cp_async16(void *dst, const void *src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                     static_cast<unsigned>(__cvta_generic_to_shared(dst))),
                 "l"(src), "r"(ok ? 16 : 0)
                 : "memory");
}

static __global__ void __launch_bounds__(SIMT_THREADS, 4) scalar_dmma_kernel(
    const double *__restrict__ A, const double *__restrict__ B, int Dp,
    const int *__restrict__ ncols, const double *__restrict__ nA, const double *__restrict__ nB,
    const int *__restrict__ molA, const int *__restrict__ molB,
    const PairTile *__restrict__ tiles, double coef, PairSink sink) {
    // the staging slices and the e_ij tile of the epilogue share one buffer
    __shared__ __align__(16) double buf[2][2][ST][DM_LD];
    double (*E)[ST + SPAD] = reinterpret_cast<double (*)[ST + SPAD]>(&buf[0][0][0][0]);
    static_assert(sizeof(buf) >= sizeof(double) * ST * (ST + SPAD), "epilogue tile");
    const PairTile t = tiles[blockIdx.x];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp & 1, wn = warp >> 1;
    const int nra = min(ST, t.a_end - t.a0), nrb = min(ST, t.b_end - t.b0);
    const int K = ncols ? (ncols[t.lab] + SK - 1) / SK * SK : Dp;
    // staging: thread -> row tid / 2 of both operands, 8 of its 16 columns
    const int lr = tid >> 1, lk = (tid & 1) * 8;
    const bool av = lr < nra, bv = lr < nrb;
    const double *ga = A + (size_t)(t.a0 + (av ? lr : 0)) * Dp + lk;
    const double *gb = B + (size_t)(t.b0 + (bv ? lr : 0)) * Dp + lk;
    auto stage = [&](int s, int k0) {
#pragma unroll
        for (int u = 0; u < 8; u += 2) {
            cp_async16(&buf[s][0][lr][lk + u], ga + k0 + u, av);
            cp_async16(&buf[s][1][lr][lk + u], gb + k0 + u, bv);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    double acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    const bool active = 32 * wm < nra && 32 * wn < nrb;   // warp-uniform
    if (K > 0) stage(0, 0);
    int s = 0;
    for (int k0 = 0; k0 < K; k0 += SK, s ^= 1) {
        if (k0 + SK < K) {
            stage(s ^ 1, k0 + SK);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        if (active) {
#pragma unroll
            for (int kk = 0; kk < SK; kk += 4) {
                const int r = lane >> 2, k = kk + (lane & 3);
                double a[4], b[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = buf[s][0][32 * wm + 8 * i + r][k];
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] = buf[s][1][32 * wn + 8 * j + r][k];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) dmma(acc[i][j], a[i], b[j]);
            }
        }
        __syncthreads();   // the slice is read before it is staged again
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = 32 * wm + 8 * i + (lane >> 2);
        const double ni = r < nra ? nA[t.a0 + r] : 0.0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int c = 32 * wn + 8 * j + 2 * (lane & 3) + u;
                double v = 0.0;
                if (r < nra && c < nrb)
                    v = exp(coef * (ni + nB[t.b0 + c] - 2.0 * acc[i][j][u]));
                E[r][c] = v;
            }
    }
    tile_rectangles<double>(E, t, nra, nrb, molA, molB, sink);
}

}  // namespace simt
}  // namespace kfb
