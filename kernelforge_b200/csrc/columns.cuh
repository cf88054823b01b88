// Descriptor columns that a label's atoms use: device code shared by the scalar
// launchers.
#pragma once

#include <cuda_runtime.h>

namespace kfb {

// used[l][k] = 1 where column k is not zero in one of label l's rows
// src[lab_start[l]] .. (NaN is not zero); grid (rep / 32, row splits, labels),
// 256 threads.
template <class Tin>
__global__ void __launch_bounds__(256) label_columns_kernel(const Tin *__restrict__ x,
                                                            const int *__restrict__ src,
                                                            const int *__restrict__ lab_start,
                                                            int rep, int *__restrict__ used) {
    const int l = blockIdx.z, s = lab_start[l], e = lab_start[l + 1];
    const int chunk = (e - s + gridDim.y - 1) / (int)gridDim.y;
    const int r0 = s + (int)blockIdx.y * chunk, r1 = min(e, r0 + chunk);
    const int k = blockIdx.x * 32 + (threadIdx.x & 31);
    if (k >= rep) return;
    bool nz = false;
    for (int r = r0 + (threadIdx.x >> 5); r < r1; r += 8)
        nz |= !(x[(size_t)src[r] * rep + k] == Tin(0));
    if (nz) used[(size_t)l * rep + k] = 1;
}

// Packed column of every descriptor column, per label (block per label, 256
// threads): used[l][k] becomes the rank of column k among the label's used
// columns, -1 where it is unused; ncols[l] the number of used columns.
//
// A column that is zero in every set-1 row of the label has a zero mean there,
// so its products x_i . x_j are exactly zero and the tiles need not contract
// over it (the norms keep it).  Descriptors have such columns whenever their
// element list holds an element that the molecules do not: 224 of the 720
// default columns belong to sulphur.
static __global__ void __launch_bounds__(256) pack_columns_kernel(int rep, int *__restrict__ used,
                                                           int *__restrict__ ncols) {
    const int l = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __shared__ int wsum[8];
    int *u = used + (size_t)l * rep;
    int base = 0;
    for (int k0 = 0; k0 < rep; k0 += 256) {
        const int k = k0 + threadIdx.x;
        const bool on = k < rep && u[k] != 0;
        const unsigned b = __ballot_sync(0xffffffffu, on);
        if (lane == 0) wsum[w] = __popc(b);
        __syncthreads();
        int before = base, total = 0;
        for (int i = 0; i < 8; ++i) {
            before += i < w ? wsum[i] : 0;
            total += wsum[i];
        }
        if (k < rep) u[k] = on ? before + __popc(b & ((1u << lane) - 1u)) : -1;
        base += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) ncols[l] = base;
}

}  // namespace kfb
