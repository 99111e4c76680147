// fr_fields.cu -- the reference's two field kernels that its registration never calls
// (src/fastreg/cuda/vector_fields.cu:109-136,194-225), on 3-plane FP32 fields in the
// caller's unpadded layout:
//   estimate_inverse_kernel    `sweeps` passes of psi_inv <- -psi o psi_inv, in place.
//                              A voxel's update reads only its own previous value (the
//                              gather is from psi), so each thread runs all the sweeps of
//                              its voxel in registers: one launch instead of the
//                              reference's 48 launches with a device sync after each.
//   interpolate_field_kernel   out = field o pos (the reference's interpolate_gradient)
// Both sample with the unchecked vector trilinear rule of interpolate_field
// (include/cuda/cuda_utils.hpp:86-107), one cell shared by the three components.
#include "fr_common.cuh"
#include "fr_kernels.h"

namespace frg {

__global__ void __launch_bounds__(256) estimate_inverse_kernel(const float* __restrict__ psi, float* psi_inv, int X,
                                                               int Y, int Z, int sweeps) {
    const int N = X * Y * Z, XY = X * Y;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        float p[3] = {psi_inv[i], psi_inv[N + i], psi_inv[2 * N + i]};
        for (int s = 0; s < sweeps; ++s) {
            const Cell32 cl = locate32(X, Y, Z, X, p[0], p[1], p[2]);
#pragma unroll
            for (int c = 0; c < 3; ++c) p[c] = -1.f * tri_unchecked32(psi + (long long)c * N, X, XY, N, cl);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) psi_inv[(long long)c * N + i] = p[c];
    }
}

// A thread owns a column of `depth` slices, a block kFieldThreads consecutive voxels of a slice (rows run on,
// so every warp but the last is full and its rows start where its lanes do).  RUN_ON: blocks run on over slices
// too, into the columns above, where the last block of every slice would be mostly idle (2x2x60000 takes 6.2 us
// and took 45); the loop is not uniform over the block any more then (182x218x182: 65.5 us instead of 64.9).
// The kernel is bound by the gathers' trips through L1, several cache lines per load.  Positions
// are mostly those of a smooth map, so the cell of the next slice is often the one above this
// slice's: its lower four corners are the upper ones already in registers, and a lane loads
// 12 corners instead of 24; all are issued before the arithmetic.  64.7 us on 182x218x182 (36
// bytes per voxel, 39 us at the copy bandwidth); 84 us with three component samples one after
// the other, 80 us with 24 corners loaded together, 70 us on 32 x 8 tiles with the reuse.
template <bool RUN_ON>
__global__ void __launch_bounds__(kFieldThreads, 2) interpolate_field_kernel(const float* __restrict__ field,
                                                                             const float* __restrict__ pos,
                                                                             float* __restrict__ out, int X, int Y,
                                                                             int Z, int depth) {
    const int N = X * Y * Z, XY = X * Y, last = N - 1;
    const int per_slice = (XY + kFieldThreads - 1) / kFieldThreads;  // blocks
    int t = blockIdx.x * kFieldThreads + threadIdx.x, layer = t / XY;
    if (RUN_ON) {
        if (layer > (Z - 1) / depth) return;
        t -= layer * XY;
    } else {
        layer = blockIdx.x / per_slice;
        t -= layer * per_slice * kFieldThreads;
        if (t >= XY) return;
    }
    const int z0 = layer * depth, z1 = Z - z0 > depth ? z0 + depth : Z;  // no overflow near 2^31
    const float* __restrict__ p[3] = {pos, pos + N, pos + 2 * (long long)N};
    const float* __restrict__ F[3] = {field, field + N, field + 2 * (long long)N};
    float* const O[3] = {out, out + N, out + 2 * (long long)N};
    int i = t + XY * z0;
    float n[3], f[3][8];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        n[c] = __ldcs(p[c] + i);
#pragma unroll
        for (int q = 0; q < 8; ++q) f[c][q] = 0.f;
    }
    int above = -1;  // base of the cell whose lower corners are the upper ones in f (-1: none)
    for (int z = z0; z < z1; ++z, i += XY) {
        const Cell32 cl = locate32(X, Y, Z, X, n[0], n[1], n[2]);
        const int b = cl.base;
        if (z + 1 < z1)
#pragma unroll
            for (int c = 0; c < 3; ++c) n[c] = __ldcs(p[c] + i + XY);
        // corners past the last voxel (of weight 0) are clamped, as in tri_unchecked32
        const int o[8] = {min(b + 1 + X + XY, last), min(b + 1 + X, last), min(b + 1 + XY, last), min(b + 1, last),
                          min(b + X + XY, last),     min(b + X, last),     min(b + XY, last),     b};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
#pragma unroll
            for (int q = 0; q < 8; q += 2) {
                f[c][q + 1] = f[c][q];
                f[c][q] = __ldg(F[c] + o[q]);
            }
        }
        if (b != above)
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int q = 1; q < 8; q += 2) f[c][q] = __ldg(F[c] + o[q]);
        above = b + XY;
        float v[3];
        trilerp3(f, cl.a, cl.b, cl.c, v);
#pragma unroll
        for (int c = 0; c < 3; ++c) __stcs(O[c] + i, v[c]);
    }
}

const void* interpolate_field_fn(bool run_on) {
    return run_on ? (const void*)interpolate_field_kernel<true> : (const void*)interpolate_field_kernel<false>;
}

}  // namespace frg
