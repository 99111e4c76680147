// fr_sob.h -- the sobolev solver: SSD data term, Gaussian-smoothed (Sobolev) gradient,
// heavy-ball momentum and a compositional update of the deformation.
//
// One iteration, per voxel x of every pair (phi = positions, m = momentum):
//   W(x)   = S(phi(x))                         trilinear, cell floor clamped to dim-2
//   g(x)   = (W(x) - T(x)) * dW/dphi(x)        exact derivative of the trilinear
//            + lambda * lap(phi - x)(x)        interpolant (0 along a clamped axis);
//                                              lap = graph Laplacian over the grid's
//                                              neighbours, lambda = W_REG
//   gs     = G_sigma * g                       separable Gaussian, SMOOTH_WIDTH taps,
//                                              normalised, replicate boundary, each tap
//                                              a fused multiply-add in the order -R..R
//   m      = DAMPING * m - STEP * gs
//   phi(x) = phi(x) + m(phi(x))                trilinear gather of the new m
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include "fr_common.cuh"

namespace frg {

constexpr int kMaxSmoothWidth = 15;

// The smoothing kernel (fr_smooth.cu): threads per block, and the rows of its 32-column
// tiles.  Tall tiles filter fewer halo rows, short ones give small volumes more warps; the
// autotuner times both.  On the 182x218x182 pair 16 rows take 67 us and 8 rows 77 us at
// radius 3 (56 and 62 us at radius 2); 12 rows 87 us and 8 rows 94 us at radius 4.  On the 64^3
// pair 16 rows take 15.8 us and 8 rows 13.9 us.  From radius 5 the chains of 8 rows fill the
// registers (12 rows at radius 7: 227 us, 8 rows 214 us).
constexpr int kSmoothThreads = 96;
constexpr int sob_smooth_tile_y(int radius, bool tall) { return !tall || radius > 4 ? 8 : radius == 4 ? 12 : 16; }
constexpr bool sob_smooth_has_tall(int radius) { return sob_smooth_tile_y(radius, true) != sob_smooth_tile_y(radius, false); }

struct SobIterArgs {
    const Pair* pairs;
    Pair pair0;      // the pair of a single-pair cohort
    int single;      // npairs == 1: the kernels take tiles and pair from the arguments (take_tile)
    int check_stop;  // max_update_norm can be reached: test for convergence, skip converged pairs
    // each kernel's own table of 32 x 8 x depth tiles (smoothing: its own rows)
    const Tile* tiles_g;
    int ntiles_g, depth_g;
    const Tile* tiles_s;
    int ntiles_s, depth_s;
    const Tile* tiles_b;
    int ntiles_b, depth_b;
    const Tile* tiles_z;  // 32 x 8 x depth tiles of the z filter where it is a launch of its own
    int ntiles_z, depth_z;
    int npairs;
    long long NT;
    const float* S;
    const float* T;
    const float* phi;  // positions (3 planes), read
    const float* m;    // momentum (3 planes), read (unrolled iterations)
    float* phi_n;      // positions, written: phi itself except in unrolled iterations
    float* m_n;        // momentum, written and gathered: m itself except in unrolled iterations
    float* g;          // gradient (3 planes)
    float* mid;        // g filtered along x and y (3 planes), smoothing in two launches
    float damping, step;
    float lambda;  // W_REG; the kernels take each pair's weight from Pair::w_reg
    float taps[kMaxSmoothWidth];
    float fold[kMaxSmoothWidth / 2 + 1];  // transposed smoothing: sum of the taps before tap R - s
    int radius;
    float max_update_norm;
    int iter;
    int* stop;
    unsigned long long* keys;
    unsigned long long* trace;
    unsigned int* counter;
    const CUtensorMap* tmaps;  // [npairs][TM_COUNT] tensor maps (fr_kernels.h), TMA-staged variants
    unsigned int* err;         // device error word (kErrTmaTimeout: a staging wait gave up)
};

// fold[s] = sum of taps[0 .. R - s - 1]: what the transposed replicate boundary adds to the tap
// that an end position takes from position s beside it
void fold_weights(const float* taps, int radius, float* fold);

// Gaussian taps exp(-k^2 / (2 sigma^2)), k = -R..R, normalised; computed in double
// and rounded to float.
void gaussian_taps(float sigma, int width, float* taps);

constexpr int sob_grad_threads(int tma) { return tma ? 288 : 256; }  // with TMA a ninth warp stages
size_t sob_grad_smem_bytes();         // dynamic shared memory of the gradient kernel
const void* sob_grad_fn(int tma);     // the gradient kernel of a staging variant (1: TMA)
// the smoothing kernel instance for a radius, staging variant (1: TMA) and tile height
const void* sob_smooth3_fn(int radius, int tma, bool tall);
// the unrolled registration's (cp.async staging): the momentum from m to m_n, or transposed,
// m_n = G^T g, which needs `fold` and zeros in the pad columns of g
const void* sob_smooth3_unrolled_fn(int radius, bool transposed, bool tall);
// the smoothing in two launches (fr_smooth.cu): every slice along x and y into `mid`, then along z;
// grid: the tiles of the first, 32 columns by the tile height by one slice
enum SmoothForm { kSmoothInPlace, kSmoothUnrolled, kSmoothTransposed };
void sob_smooth_split_fns(int radius, SmoothForm form, bool tall, const void** planes, const void** z);
cudaError_t launch_smooth_split(const SobIterArgs& a, SmoothForm form, bool tall, int grid, cudaStream_t s, bool behind);
// Where the two launches are the faster for N packed voxels, one launch -> two.  Unrolled (20
// iterations), radius 2: 64^3 0.97 -> 0.93 ms, 96^3 1.96 -> 1.99; radius 3: 64^3 1.33 -> 1.10, 112^3 3.74 ->
// 3.67, 128^3 4.83 -> 4.85; radius 4: 64^3 1.46 -> 1.07, 182x218x182 14.5 -> 14.2; radius 5: 128^3 5.99 ->
// 5.47, 182x218x182 the same; radius 7: 128^3 9.04 -> 6.30, 182x218x182 20.6 -> 17.6.  Registrations (200
// iterations), whose other kernels take more of L2, radius 2: 60x64x60 3.3 -> 3.0 ms; radius 3: 64^3 4.1 ->
// 3.3, 112^3 the same, 128^3 13.2 -> 14.8; radius 4: 96^3 7.9 -> 6.8, 128^3 14.8 -> 15.4; radius 5: 91x109x91
// 5.2 -> 4.6, 128^3 19.0 -> 16.5, from 160^3 on one launch (the autotuner times both).
constexpr bool sob_smooth_split(int radius, long long N, bool unrolled) {
    return radius >= (unrolled ? 4 : 5) || (radius >= 3 && N <= 3 << 19) || (radius == 2 && N <= 1 << 18);
}
// Whether any size is smoothed in two launches, and any unrolled one in one: the forms that fr_smooth.cu instantiates.
constexpr bool sob_smooth_ever_split(int radius) {
    return sob_smooth_split(radius, 1, false) || sob_smooth_split(radius, 1, true);
}
constexpr bool sob_smooth_ever_one_unrolled(int radius) { return !sob_smooth_split(radius, 1LL << 62, true); }
// slices per tile of the z filter: as many, up to 32, as leave two blocks for every SM
inline int sob_smooth_z_depth(long long columns, int Z, int sms) {  // columns: 32 x 8, of all pairs
    const long long d = 3 * columns * Z / (2LL * (sms > 0 ? sms : 1));
    return d < 2 ? 2 : d > 32 ? 32 : (int)d;
}
// box of one component of the smoothing kernel's staged slice for radius R: x extent, rows
inline void sob_smooth_box(int R, bool tall, int* wx, int* rows) {
    *wx = kTileX + 2 * ((R + 3) / 4 * 4);
    *rows = sob_smooth_tile_y(R, tall) + 2 * R;
}
const void* sob_pass_b_fn(bool unrolled);  // the update kernel
constexpr int kUnrolled = 4;  // variant bit: the unrolled registration's kernel (separate in and out states)
constexpr int kSplit = 8;     // variant bit of the smoothing: in two launches

// one of them: k = 0 gradient, 1 smoothing, 2 update
cudaError_t launch_sob_kernel(int k, const SobIterArgs& a, int grid, int variant, cudaStream_t s, bool behind);

// grids: {grad, smooth, pass_b}; variants: of {grad, smooth, pass_b} (bit 0: TMA
// staging, bit 1 of smooth: tall tiles); with `ev`
// (4 events) each launch is bracketed
cudaError_t launch_sob_iter(const SobIterArgs& a, const int* grids, const int* variants, cudaStream_t s,
                            bool behind, cudaEvent_t* ev = nullptr);

// Cell for the sobolev solver: clamp to [0, dim-1], floor clamped to dim-2 so that
// both corners of every axis are inside the grid; in_x, in_y, in_z: the position was not
// clamped (a clamped axis has derivative 0).
struct SobCell {
    int base;
    int gx, gy, gz;
    float a, b, c;
    bool in_x, in_y, in_z;
};

__device__ __forceinline__ SobCell sob_locate(const Pair& P, float px, float py, float pz) {
    SobCell s;
    const float cx = fminf(fmaxf(0.f, px), (float)(P.X - 1));
    const float cy = fminf(fmaxf(0.f, py), (float)(P.Y - 1));
    const float cz = fminf(fmaxf(0.f, pz), (float)(P.Z - 1));
    s.gx = min((int)floorf(cx), P.X - 2);
    s.gy = min((int)floorf(cy), P.Y - 2);
    s.gz = min((int)floorf(cz), P.Z - 2);
    s.a = cx - (float)s.gx;
    s.b = cy - (float)s.gy;
    s.c = cz - (float)s.gz;
    s.in_x = cx == px;  // false for a NaN
    s.in_y = cy == py;
    s.in_z = cz == pz;
    s.base = s.gx + P.Xp * (s.gy + P.Y * s.gz);
    return s;
}

}  // namespace frg
