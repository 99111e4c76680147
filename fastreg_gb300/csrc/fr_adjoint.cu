// fr_adjoint.cu -- the differentiated sobolev registration.
//
// J(v0, lambda) = 0.5 * sum (S(phi_K) - T)^2 + 0.1 * sum |m_K|^2 after K iterations of the
// sobolev solver (fr_sob.h) started from phi_0 = identity and m_0 = v0, with the
// displacement regulariser weighted by lambda:
//   g       = (S(phi) - T) dS(phi) + lambda * lap(phi - x)
//   m'      = damping * m - step * G g
//   phi'    = phi + m'(phi)
// The reverse sweep runs hand-written adjoint kernels for each line: the compositional
// update (gather of dm'/dphi, scatter-add into m'), the momentum, the transposed
// separable Gaussian (replicate boundary), the regulariser (the graph Laplacian is
// symmetric) and the data gradient (the trilinear interpolant's gradient and Hessian).
// Forward states are checkpointed every `checkpoint_every` iterations and each segment
// is recomputed before it is reversed (the last one as part of the forward sweep).
//
// The workspace holds one pair in the packed layout of the cohort (fr_common.cuh), so the
// forward iterations are the cohort's own three kernels (the same bits as a registration),
// with a separate input and output state per iteration: a checkpoint or a segment's state is
// written where it is kept and never copied.  The reverse iteration is four kernels: the
// update's adjoint, the momentum's, the transposed smoothing (the smoothing kernel's
// transposed form, or two) and the gradient's.  fr_warp_adjoint works on the caller's unpadded planes.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "../../include/fastreg_gb300.h"
#include "fr_columns.h"
#include "fr_common.cuh"
#include "fr_kernels.h"
#include "fr_limits.h"
#include "fr_sob.h"

namespace frg {

#define GRID_STRIDE(i, n) for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += gridDim.x * blockDim.x)

// One pair of the workspace.
struct AdjPair {
    int X, Y, Z, Xp, XYp;  // extents, row and slice pitch
    int N;                 // XYp * Z
    long long NT;          // plane stride of vector fields
};

// The caller's fields into the packed workspace: S, T, phi = identity, m = v0; pad columns zero.
__global__ void __launch_bounds__(256) adj_pack_kernel(AdjPair A, const float* __restrict__ S, const float* __restrict__ T,
                                                       const float* __restrict__ v0, float* Sp, float* Tp, float* phi,
                                                       float* m) {
    const long long nu = (long long)A.X * A.Y * A.Z;
    GRID_STRIDE(i, A.N) {
        const int row = i / A.Xp, x = i - row * A.Xp, z = row / A.Y, y = row - z * A.Y;
        const bool in = x < A.X;
        const long long u = x + (long long)A.X * row;
        Sp[i] = in ? __ldg(S + u) : 0.f;
        Tp[i] = in ? __ldg(T + u) : 0.f;
        const float pos[3] = {(float)x, (float)y, (float)z};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            phi[c * A.NT + i] = pos[c];
            m[c * A.NT + i] = in ? __ldg(v0 + c * nu + u) : 0.f;
        }
    }
}

// The result: the adjoint of v0 out of the interleaved accumulator.
__global__ void __launch_bounds__(256) adj_unpack_kernel(AdjPair A, const float4* mbar, float* out) {
    pdl_wait();
    const long long nu = (long long)A.X * A.Y * A.Z;
    GRID_STRIDE(i, A.N) {
        const int row = i / A.Xp, x = i - row * A.Xp;
        if (x >= A.X) continue;
        const float4 v = chain_load(mbar + i);
        const long long u = x + (long long)A.X * row;
        out[u] = v.x;
        out[nu + u] = v.y;
        out[2 * nu + u] = v.z;
    }
}

// The trilinear interpolant at a cell: corners f in the order 111, 110, 101, 100, 011, 010, 001,
// 000 (x, y, z), fractions a, b, c.
__device__ __forceinline__ void tri_grad(const float f[8], const SobCell& s, float d[3], float* val, float H[3]) {
    const float e11 = lerpf_(f[0], f[1], s.c), e10 = lerpf_(f[2], f[3], s.c);
    const float e01 = lerpf_(f[4], f[5], s.c), e00 = lerpf_(f[6], f[7], s.c);
    const float A1 = lerpf_(e11, e10, s.b), A0 = lerpf_(e01, e00, s.b);
    const float d11 = f[0] - f[1], d10 = f[2] - f[3], d01 = f[4] - f[5], d00 = f[6] - f[7];
    const float z1 = lerpf_(d11, d10, s.b), z0 = lerpf_(d01, d00, s.b);
    d[0] = s.in_x ? A1 - A0 : 0.f;
    d[1] = s.in_y ? lerpf_(e11 - e10, e01 - e00, s.a) : 0.f;
    d[2] = s.in_z ? lerpf_(z1, z0, s.a) : 0.f;
    if (val) *val = lerpf_(A1, A0, s.a);
    if (H) {  // mixed second derivatives xy, xz, yz (the pure ones are 0)
        H[0] = s.in_x && s.in_y ? (e11 - e10) - (e01 - e00) : 0.f;
        H[1] = s.in_x && s.in_z ? z1 - z0 : 0.f;
        H[2] = s.in_y && s.in_z ? lerpf_(d11 - d10, d01 - d00, s.a) : 0.f;
    }
}

__device__ __forceinline__ void load_corners(const float* __restrict__ F, int b, int X, int XY, float f[8]) {
    f[0] = __ldg(F + b + 1 + X + XY);
    f[1] = __ldg(F + b + 1 + X);
    f[2] = __ldg(F + b + 1 + XY);
    f[3] = __ldg(F + b + 1);
    f[4] = __ldg(F + b + X + XY);
    f[5] = __ldg(F + b + X);
    f[6] = __ldg(F + b + XY);
    f[7] = __ldg(F + b);
}

__device__ __forceinline__ Pair as_pair(const AdjPair& A) {
    Pair P{};
    P.X = A.X;
    P.Y = A.Y;
    P.Z = A.Z;
    P.Xp = A.Xp;
    return P;
}

// J and the adjoint seeds: pbar = r dS(phi_K), mbar = 0.2 m_K (0 in the pad columns).  Every term
// is a product of two FP32 values, exact in FP64, added by one fused multiply-add.
__global__ void __launch_bounds__(256) adj_loss_kernel(AdjPair A, const float* __restrict__ S, const float* __restrict__ T,
                                                       const float* phi, const float* m,
                                                       float* pbar, float4* mbar, double* loss) {
    pdl_wait();
    __shared__ double red[32];
    const Pair P = as_pair(A);
    double er = 0.0, em = 0.0;
    GRID_STRIDE(i, A.N) {
        if (i % A.Xp >= A.X) {
            mbar[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            continue;
        }
        const SobCell s = sob_locate(P, chain_load(phi + i), chain_load(phi + A.NT + i), chain_load(phi + 2 * A.NT + i));
        float f[8], d[3], W;
        load_corners(S, s.base, A.Xp, A.XYp, f);
        tri_grad(f, s, d, &W, nullptr);
        const float r = W - __ldg(T + i);
        er = fma((double)r, (double)r, er);
        float mc[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            mc[c] = chain_load(m + c * A.NT + i);
            em = fma((double)mc[c], (double)mc[c], em);
            pbar[c * A.NT + i] = r * d[c];
        }
        mbar[i] = make_float4(0.2f * mc[0], 0.2f * mc[1], 0.2f * mc[2], 0.f);
    }
    const double e = block_sum_f64(0.5 * er + 0.1 * em, red);
    if (threadIdx.x == 0) atomicAdd(loss, e);
}

// Adds the contributions v[0..3] to the corners 00, 10, 01, 11 (x, y) of the face at `b` of the
// interleaved field F: one 16-byte reduction per corner for the three components, and the x
// corners that neighbouring lanes share added once: the lanes of a warp hold consecutive
// voxels of a row, whose cells are usually consecutive along x, so lane k adds lane k - 1's x + 1
// contribution to its own x one.  All 32 lanes must call it; inactive lanes pass act = false.
__device__ __forceinline__ void red_add4(float4* p, float3 v) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(0.f)
                 : "memory");
}
__device__ __forceinline__ void scatter_face_warp(float4* F, int b, const float3 v[4], bool act, int X) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int bprev = __shfl_up_sync(full, act ? b : -4, 1);
    const bool merge = act && lane > 0 && bprev == b - 1;
    const bool next_merges = __shfl_down_sync(full, (int)merge, 1) != 0 && lane < 31;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const float3 c1 = v[2 * j + 1];
        float3 c0 = v[2 * j];
        const float px = __shfl_up_sync(full, c1.x, 1), py = __shfl_up_sync(full, c1.y, 1),
                    pz = __shfl_up_sync(full, c1.z, 1);
        if (merge) c0 = make_float3(c0.x + px, c0.y + py, c0.z + pz);
        if (act) {
            red_add4(F + b + j * X, c0);
            if (!next_merges) red_add4(F + b + 1 + j * X, c1);
        }
    }
}

// phi' = phi + m'(phi): pbar += (dm'/dphi)^T pbar (in place: a voxel reads only its own), mbar +=
// scatter(w * pbar).
//
// A thread owns a column (Columns).  The reductions bound the kernel (about one lane's
// reduction a cycle and SM whatever its width), so they are made few and wide: mbar is
// interleaved, a 16-byte reduction per corner serves the three components; neighbouring lanes
// share corners (scatter_face_warp); and the upper face of a voxel's cell, which is the lower
// face of the next slice's cell where the cell moves up by exactly one slice, is held back and
// added there.  The gathered corners are kept the same way, as in sob_pass_b_kernel.  On the
// 128^3 pair 42 us from a smooth momentum, 75 us from white noise, whose cells share little; with one 4-byte
// reduction per corner and component, lanes merged, 144 us.
template <int SHAPE>
__global__ void __launch_bounds__(256) adj_update_kernel(AdjPair A, Columns C, const float* phi, const float* mn,
                                                         float* pbar, float4* mbar) {
    pdl_wait();
    const Pair P = as_pair(A);
    int x, y, z0, z1;
    C.place<SHAPE>(blockIdx.x, threadIdx.x, A.Z, x, y, z0, z1);
    const bool act = x < A.X && y < A.Y && (SHAPE != kLayeredColumns || z0 < z1);
    const int Xp = A.Xp, XY = A.XYp;
    int i = act ? x + Xp * y + XY * z0 : 0;
    float f[3][8];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int q = 0; q < 8; ++q) f[c][q] = 0.f;
    float3 held[4];  // the upper face's contributions of the previous slice's cell
#pragma unroll
    for (int q = 0; q < 4; ++q) held[q] = make_float3(0.f, 0.f, 0.f);
    int above = -1;  // base of the cell above the previous slice's cell (-1: none)
    float np[3], nb[3];  // phi and pbar of the next slice, loaded while this one's gathers are in flight
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        np[c] = chain_load(phi + c * A.NT + i);
        nb[c] = pbar[c * A.NT + i];
    }
    for (int z = z0; z < z1; ++z, i += act ? XY : 0) {
        const SobCell s = sob_locate(P, np[0], np[1], np[2]);
        const int b = s.base;
        const bool on = b == above;
        float acc[3], pb[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float* F = mn + c * A.NT;
            f[c][1] = f[c][0];
            f[c][3] = f[c][2];
            f[c][5] = f[c][4];
            f[c][7] = f[c][6];
            f[c][0] = chain_load(F + b + 1 + Xp + XY);
            f[c][2] = chain_load(F + b + 1 + XY);
            f[c][4] = chain_load(F + b + Xp + XY);
            f[c][6] = chain_load(F + b + XY);
            if (!on) {
                f[c][1] = chain_load(F + b + 1 + Xp);
                f[c][3] = chain_load(F + b + 1);
                f[c][5] = chain_load(F + b + Xp);
                f[c][7] = chain_load(F + b);
            }
            acc[c] = pb[c] = nb[c];
        }
        if (act && z + 1 < z1)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                np[c] = chain_load(phi + c * A.NT + i + XY);
                nb[c] = pbar[c * A.NT + i + XY];
            }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            float d[3];
            tri_grad(f[c], s, d, nullptr, nullptr);
#pragma unroll
            for (int k = 0; k < 3; ++k) acc[k] += pb[c] * d[k];
        }
        if (act)
#pragma unroll
            for (int c = 0; c < 3; ++c) pbar[c * A.NT + i] = acc[c];
        // what the cell does not take over from the slice below is added where it belongs
        const bool flush = act && !on && above >= 0;
        if (__any_sync(0xffffffffu, flush)) scatter_face_warp(mbar, above, held, flush, Xp);
        float3 low[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float w = ((q & 1) ? s.a : 1.f - s.a) * ((q & 2) ? s.b : 1.f - s.b);
            const float w0 = w * (1.f - s.c), w1 = w * s.c;
            low[q] = make_float3(w0 * pb[0], w0 * pb[1], w0 * pb[2]);
            if (on) low[q] = make_float3(low[q].x + held[q].x, low[q].y + held[q].y, low[q].z + held[q].z);
            held[q] = make_float3(w1 * pb[0], w1 * pb[1], w1 * pb[2]);
        }
        scatter_face_warp(mbar, b, low, act, Xp);
        above = b + XY;
    }
    scatter_face_warp(mbar, above, held, act && above >= 0, Xp);
}

// m' = damping * m - step * gs: gs = -step * mbar (planes), mbar = damping * mbar; zero pad columns stay zero
__global__ void __launch_bounds__(256) adj_momentum_kernel(AdjPair A, float damping, float step, float4* mbar, float* gs) {
    pdl_wait();
    GRID_STRIDE(i, A.N) {
        const float4 v = mbar[i];
        gs[i] = -step * v.x;
        gs[A.NT + i] = -step * v.y;
        gs[2 * A.NT + i] = -step * v.z;
        mbar[i] = make_float4(damping * v.x, damping * v.y, damping * v.z, 0.f);
    }
}

// s + c += a * b with the product and the sum exact to about twice the FP32 precision (the
// compensated dot product Dot2 of Ogita, Rump and Oishi, 2005).  Its error terms are exact only for products
// in kDotLeast .. kDotMost (and for a zero factor): below, the product's last bits, 47 places
// under its first, fall under the smallest FP32 number, 2^-149; above, a few dozen sums could overflow.
// False for any other product, and for a NaN.
constexpr float kDotLeast = 0x1p-100f, kDotMost = 0x1p100f;
__device__ __forceinline__ bool dot2(float a, float b, float& s, float& c) {
    const float p = a * b, e = fmaf(a, b, -p), size = fabsf(p);
    const float t = s + p, u = t - s;
    c += e + ((s - (t - u)) + (p - u));
    s = t;
    return ((size >= kDotLeast) & (size <= kDotMost)) | ((p == 0.f) & ((a == 0.f) | (b == 0.f)));
}

// The sum of gbar . lap(phi - x) over one column of adj_grad_kernel in FP64, terms and order as there.
__device__ __forceinline__ double lambda_sum_f64(const AdjPair& A, const float* phi, const float* gbar, int x, int y, int z0,
                                              int z1) {
    const bool ok[6] = {x > 0, x < A.X - 1, y > 0, y < A.Y - 1, true, true};
    const int off[6] = {-1, 1, -A.Xp, A.Xp, -A.XYp, A.XYp};
    double sum = 0.0;
    int i = x + A.Xp * y + A.XYp * z0;
    for (int z = z0; z < z1; ++z, i += A.XYp)
        for (int c = 0; c < 3; ++c) {
            const float* P = phi + c * A.NT + i;
            const float pc = chain_load(P);
            float l = 0.f;
            for (int k = 0; k < 6; ++k) {
                if (k < 4 ? !ok[k] : k == 4 ? z == 0 : z == A.Z - 1) continue;
                const float d = pc - chain_load(P + off[k]);
                l += k / 2 == c ? d + ((k & 1) ? 1.f : -1.f) : d;
            }
            sum = fma((double)chain_load(gbar + c * A.NT + i), (double)l, sum);
        }
    return sum;
}

// g = (S(phi) - T) dS(phi) + lambda lap(phi - x): pbar += lambda lap^T(gbar) + (gbar . dS) dS + r H
// gbar; lambda_bar += gbar . lap.  A thread owns a column (Columns); its own
// column of phi and gbar stays in registers from slice to slice, the neighbours along x and y
// come through L1, and the Laplacians' terms across a z face are formed once (sob_grad_kernel).
// The kernel waits on its loads, so a voxel's are issued together (64 us on
// the 128^3 pair when each neighbour was loaded where it was used), and it is held to five blocks per SM (48
// registers): 40 us, 46 us with four of 54.  lambda_bar is
// summed in compensated FP32 per thread and in FP64 beyond, as the FP64 pipe of this GPU takes
// 16 cycles per warp and operation (78 us with six FP64 operations and six conversions a voxel); a column with a
// product outside dot2's range is summed in FP64 (lambda_sum_f64).
template <int SHAPE>
__global__ void __launch_bounds__(256, SHAPE == kLayeredColumns ? 3 : 5) adj_grad_kernel(AdjPair A, Columns C, const float* __restrict__ S,
                                                          const float* __restrict__ T, const float* phi, float lambda,
                                                          const float* gbar, float* pbar, double* lbar) {
    pdl_wait();
    __shared__ double red[32];
    const Pair P = as_pair(A);
    int x, y, z0, z1;
    C.place<SHAPE>(blockIdx.x, threadIdx.x, A.Z, x, y, z0, z1);
    const int Xp = A.Xp, XY = A.XYp;
    double lsum = 0.0;
    if (x < A.X && y < A.Y && (SHAPE != kLayeredColumns || z0 < z1)) {
        const bool xl = x > 0, xr = x < A.X - 1, yl = y > 0, yr = y < A.Y - 1;
        int i = x + Xp * y + XY * z0;
        float ls = 0.f, lc = 0.f;
        bool held = true;  // every product of the column was in dot2's range
        float p[3], g[3], pz[3], gz[3];  // phi and gbar here, and their terms across the face below
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            p[c] = chain_load(phi + c * A.NT + i);
            g[c] = chain_load(gbar + c * A.NT + i);
            pz[c] = gz[c] = 0.f;
            if (z0 > 0) {
                pz[c] = chain_load(phi + c * A.NT + i - XY) - p[c];
                if (c == 2) pz[c] += 1.f;
                gz[c] = chain_load(gbar + c * A.NT + i - XY) - g[c];
            }
        }
        for (int z = z0; z < z1; ++z, i += XY) {
            const bool zr = z < A.Z - 1;
            const SobCell s = sob_locate(P, p[0], p[1], p[2]);
            float f[8], add[3], gb[3], pn[3][5], gn[3][5], old[3];
            // every load of the voxel before the arithmetic: neighbours -x, +x, -y, +y, +z (its own
            // value where there is none), corners, T and pbar
            load_corners(S, s.base, Xp, XY, f);
            const float tv = __ldg(T + i);
            const int off[5] = {xl ? -1 : 0, xr ? 1 : 0, yl ? -Xp : 0, yr ? Xp : 0, zr ? XY : 0};
#pragma unroll
            for (int c = 0; c < 3; ++c) {
#pragma unroll
                for (int k = 0; k < 5; ++k) {
                    pn[c][k] = chain_load(phi + c * A.NT + i + off[k]);
                    gn[c][k] = chain_load(gbar + c * A.NT + i + off[k]);
                }
                old[c] = pbar[c * A.NT + i];
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float pc = p[c], gc = g[c];
                gb[c] = gc;
                float l = 0.f;
                if (xl) l += c == 0 ? (pc - pn[c][0]) - 1.f : pc - pn[c][0];
                if (xr) l += c == 0 ? (pc - pn[c][1]) + 1.f : pc - pn[c][1];
                if (yl) l += c == 1 ? (pc - pn[c][2]) - 1.f : pc - pn[c][2];
                if (yr) l += c == 1 ? (pc - pn[c][3]) + 1.f : pc - pn[c][3];
                l -= pz[c];
                pz[c] = !zr ? 0.f : c == 2 ? (pc - pn[c][4]) + 1.f : pc - pn[c][4];
                l += pz[c];
                const float t = (((gc - gn[c][0]) + (gc - gn[c][1])) + (gc - gn[c][2])) + (gc - gn[c][3]);
                const float up = gc - gn[c][4];
                add[c] = lambda * ((t - gz[c]) + up);
                gz[c] = up;
                p[c] = pn[c][4];
                g[c] = gn[c][4];
                held &= dot2(gc, l, ls, lc);
            }
            float d[3], W, H[3];
            tri_grad(f, s, d, &W, H);
            const float r = W - tv;
            const float gd = (gb[0] * d[0] + gb[1] * d[1]) + gb[2] * d[2];
            const float h[3] = {gb[1] * H[0] + gb[2] * H[1], gb[0] * H[0] + gb[2] * H[2], gb[0] * H[1] + gb[1] * H[2]};
#pragma unroll
            for (int k = 0; k < 3; ++k) pbar[k * A.NT + i] = old[k] + (add[k] + (gd * d[k] + r * h[k]));
        }
        lsum = held ? (double)ls + (double)lc : lambda_sum_f64(A, phi, gbar, x, y, z0, z1);
    }
    const double lb = block_sum_f64(lsum, red);
    if (threadIdx.x == 0) atomicAdd(lbar, lb);
}

}  // namespace frg

namespace {

// The device workspace of fr_sobolev_loss_grad (checkpoints, segment states and adjoint
// fields, about 40 fields of 3 N floats for 50 iterations), kept per device and reused by
// later calls that need as much or less: an unrolled registration is typically
// differentiated many times in a row (hypergradient steps), and a fresh cudaMalloc /
// cudaFree of a gigabyte per call costs milliseconds and synchronises the device.  A call
// that finds the workspace busy (another host thread's call on the same device) uses a
// private allocation instead.
std::mutex g_ws_mu;
struct Workspace {
    float* ptr = nullptr;
    size_t floats = 0;
    bool busy = false;
};
Workspace g_ws[64];

// a workspace of at least `floats` floats on device `dev`; *cached says whether it is the
// shared one (released with release_workspace) or private (freed by the caller)
float* acquire_workspace(int dev, size_t floats, bool* cached) {
    *cached = false;
    if (dev >= 0 && dev < 64) {
        std::lock_guard<std::mutex> lk(g_ws_mu);
        Workspace& w = g_ws[dev];
        if (!w.busy) {
            if (w.floats < floats) {
                if (w.ptr) cudaFree(w.ptr);
                w.ptr = nullptr;
                w.floats = 0;
                if (cudaMalloc((void**)&w.ptr, floats * sizeof(float)) == cudaSuccess)
                    w.floats = floats;
                else {
                    cudaGetLastError();
                    w.ptr = nullptr;
                }
            }
            if (w.ptr) {
                w.busy = true;
                *cached = true;
                return w.ptr;
            }
        }
    }
    float* p = nullptr;
    if (cudaMalloc((void**)&p, floats * sizeof(float)) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return p;
}

void release_workspace(int dev, float* p, bool cached) {
    if (!cached) {
        cudaFree(p);
        return;
    }
    std::lock_guard<std::mutex> lk(g_ws_mu);
    g_ws[dev].busy = false;
}

int grid_for(long long n) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    long long want = (n + 255) / 256;
    return (int)std::max(1LL, std::min<long long>(want, (long long)std::max(sms, 1) * 8));
}

}  // namespace

namespace frg {
void set_global_error(const char* msg);
}

extern "C" int fr_sobolev_loss_grad(const float* d_T, const float* d_S, const int dims[3], const float* d_v0,
                                    float lambda, int iters, int checkpoint_every, float damping, float step,
                                    float smooth_sigma, int smooth_width, double* loss, float* d_grad_v0,
                                    double* grad_lambda, void* stream) {
    using namespace frg;
    set_global_error("");
    if (!d_T || !d_S || !dims || !d_v0 || !loss) {
        set_global_error("fr_sobolev_loss_grad: NULL argument");
        return FR_ERR_INVALID_ARG;
    }
    if (dims[0] < 4 || dims[1] < 4 || dims[2] < 4 || iters < 1 || checkpoint_every < 1 || smooth_width < 1 ||
        smooth_width > kMaxSmoothWidth || (smooth_width & 1) == 0 || !(smooth_sigma > 0.f)) {
        set_global_error("fr_sobolev_loss_grad: invalid size or parameter");
        return FR_ERR_INVALID_ARG;
    }
    const long long N64 = (long long)dims[0] * dims[1] * dims[2];
    if (N64 > (1LL << 30)) {
        set_global_error("fr_sobolev_loss_grad: volume too large (limit 2^30 voxels)");
        return FR_ERR_INVALID_ARG;
    }
    AdjPair A{};
    A.X = dims[0];
    A.Y = dims[1];
    A.Z = dims[2];
    A.Xp = (A.X + 3) / 4 * 4;
    A.XYp = A.Xp * A.Y;
    A.N = A.XYp * A.Z;
    A.NT = ((long long)A.N + 31) / 32 * 32;
    const size_t N3 = 3 * (size_t)A.NT;
    const int K = iters, ck = std::min(checkpoint_every, iters), nseg = (K + ck - 1) / ck;
    cudaStream_t s = (cudaStream_t)stream;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        set_global_error("fr_sobolev_loss_grad: no current CUDA device");
        return FR_ERR_CUDA;
    }
    const int R = smooth_width / 2;
    // Tiles of the gradient, the smoothing, the update and the transposed smoothing, and the reverse
    // kernels' columns.  A tile of d slices takes d + extra steps; blocks
    // beyond `per_sm` per SM slow one another down instead of filling idle issue slots.  With the
    // blocks per SM below the depth chosen is within 4% of the best one measured at 45x54x45,
    // 64^3, 96^3 and 128^3 (20 iterations); the column kernels gain from many small tiles (128^3:
    // 6.15 ms at 6 slices, 6.48 at 13), so theirs are held to 6 slices.
    auto best_depth = [&](auto blocks, int per_sm, int extra, int most, double* cost) {
        int best = 1;
        *cost = 1e300;
        for (int d = 1; d <= std::min(A.Z, most); ++d) {
            const double c = std::max(1.0, (double)blocks(d) / ((double)sms * per_sm)) * (d + extra);
            if (c < *cost) {
                *cost = c;
                best = d;
            }
        }
        return best;
    };
    struct Cut {
        int rows, depth, count;
    };
    auto cut = [&](int per_sm, int rows, int extra, int most, double* cost) {
        const long long cols = (long long)((A.X + kTileX - 1) / kTileX) * ((A.Y + rows - 1) / rows);
        auto tiles = [&](int d) { return cols * ((A.Z + d - 1) / d); };
        const int d = best_depth(tiles, per_sm, extra, most, cost);
        *cost *= rows + extra;
        return Cut{rows, d, (int)tiles(d)};
    };
    double cost = 0.0, cost_tall = 0.0;
    Cut cuts[4];
    cuts[0] = cut(6, kTileY, 2, 128, &cost);
    cuts[2] = cut(4, kTileY, 1, 6, &cost);
    const Cut low = cut(3, sob_smooth_tile_y(R, false), 2 * R + 1, 128, &cost);
    const Cut high = cut(3, sob_smooth_tile_y(R, true), 2 * R + 1, 128, &cost_tall);
    const long long columns8 = (long long)((A.X + kTileX - 1) / kTileX) * ((A.Y + kTileY - 1) / kTileY);
    // smoothing in two launches where it is the faster (sob_smooth_z_kernel)
    const bool split = sob_smooth_split(R, A.N, true);
    auto slices = [&](bool tall) {  // tiles of one slice each
        const int rows = sob_smooth_tile_y(R, tall);
        return Cut{rows, 1, (A.X + kTileX - 1) / kTileX * ((A.Y + rows - 1) / rows) * A.Z};
    };
    const bool tall = split ? slices(true).count >= 2 * sms : cost_tall < cost;
    cuts[1] = cuts[3] = split ? slices(tall) : tall ? high : low;
    Columns columns(A.Xp, A.X, A.Y);
    columns.depth = best_depth(
        [&](int d) {
            columns.depth = d;
            return columns.blocks(A.Z);
        },
        4, 1, 6, &cost);

    // the workspace: checkpoints (phi, m) x nseg, the states of a segment (phi, m) x ck, two
    // working states, g, gbar, pbar, the interleaved mbar, S and T; and a small head
    auto round_up = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t head = round_up(sizeof(Pair)) + round_up(64);
    const size_t plane = round_up(N3 * sizeof(float)), scalar = round_up((size_t)A.NT * sizeof(float));
    const size_t bytes = head + plane * (2 * nseg + 2 * ck + 4 + 3) + round_up((size_t)A.NT * sizeof(float4)) + 2 * scalar;
    bool cached = false;
    char* blk = reinterpret_cast<char*>(acquire_workspace(dev, (bytes + 3) / 4, &cached));
    if (!blk) {
        set_global_error("fr_sobolev_loss_grad: device allocation failed");
        return FR_ERR_ALLOC;
    }
    char* at = blk;
    auto take = [&](size_t b) {
        char* p = at;
        at += round_up(b);
        return p;
    };
    Pair* pair = (Pair*)take(sizeof(Pair));
    double* dd = (double*)take(64);  // loss and lambda_bar
    auto field = [&]() { return (float*)take(N3 * sizeof(float)); };
    struct State {
        float *phi, *m;
    };
    std::vector<State> ckpt(nseg), seg(ck);  // seg[j]: the state after iteration j of a segment
    for (State& c : ckpt) c = State{field(), field()};
    for (State& c : seg) c = State{field(), field()};
    State work[2] = {{field(), field()}, {field(), field()}};
    float *g = field(), *gbar = field(), *pbar = field();
    float4* mbar = (float4*)take((size_t)A.NT * sizeof(float4));
    float *Sp = (float*)take((size_t)A.NT * sizeof(float)), *Tp = (float*)take((size_t)A.NT * sizeof(float));

    SobIterArgs a{};
    a.pairs = pair;
    a.single = 1;  // tiles and pair from the arguments, no convergence test
    a.pair0.X = A.X;
    a.pair0.Y = A.Y;
    a.pair0.Z = A.Z;
    a.pair0.Xp = A.Xp;
    a.pair0.N = A.N;
    a.pair0.w_reg = lambda;
    a.ntiles_g = cuts[0].count;
    a.depth_g = cuts[0].depth;
    a.depth_z = sob_smooth_z_depth(columns8, A.Z, sms);
    a.ntiles_z = (int)(columns8 * ((A.Z + a.depth_z - 1) / a.depth_z));
    a.ntiles_b = cuts[2].count;
    a.depth_b = cuts[2].depth;
    a.npairs = 1;
    a.NT = A.NT;
    a.S = Sp;
    a.T = Tp;
    a.g = g;
    a.damping = damping;
    a.step = step;
    a.lambda = lambda;
    gaussian_taps(smooth_sigma, smooth_width, a.taps);
    a.radius = R;
    fold_weights(a.taps, R, a.fold);
    const int grid = grid_for(A.N), column_blocks = (int)columns.blocks(A.Z);
    const void* const update_fns[] = {(const void*)adj_update_kernel<kTileColumns>, (const void*)adj_update_kernel<kFlatColumns>,
                                      (const void*)adj_update_kernel<kLayeredColumns>};
    const void* const grad_fns[] = {(const void*)adj_grad_kernel<kTileColumns>, (const void*)adj_grad_kernel<kFlatColumns>,
                                    (const void*)adj_grad_kernel<kLayeredColumns>};
    const void *update_fn = update_fns[columns.shape], *grad_fn = grad_fns[columns.shape];
    int rc = FR_OK;
    auto ok = [&](cudaError_t e) {
        if (e != cudaSuccess) rc = FR_ERR_CUDA;
        return rc == FR_OK;
    };
    // iteration k (0-based) from one state to another
    auto forward = [&](int k, const State& from, const State& to) {
        a.iter = k + 1;
        a.phi = from.phi;
        a.m = from.m;
        a.phi_n = to.phi;
        a.m_n = to.m;
        a.ntiles_s = cuts[1].count;
        a.depth_s = cuts[1].depth;
        ok(launch_sob_kernel(0, a, cuts[0].count, 0, s, k > 0));  // the first one behind adj_pack_kernel (pdl_wait)
        a.mid = gbar;  // free until the reverse iteration's smoothing
        ok(launch_sob_kernel(1, a, cuts[1].count, kUnrolled | (tall ? 2 : 0) | (split ? kSplit : 0), s, true));
        ok(launch_sob_kernel(2, a, cuts[2].count, kUnrolled, s, true));
    };
    // the reverse kernels' blocks are placed while the kernel ahead drains, as the forward ones' are: short
    // kernels gain most (45x54x45, 20 iterations: 1.93 -> 1.69 ms; 128^3, 50 iterations: 13.3 -> 12.7 ms, of
    // which 0.25 ms is a segment's last state taken from the checkpoint)
    auto reverse = [&](const void* fn, int blocks, auto... v) {
        void* args[] = {&v...};
        ok(launch_kernel(fn, blocks, 256, 0, args, s, true));
    };
    auto smooth_adjoint = [&]() {  // gbar = G^T g
        SobIterArgs t = a;
        t.m_n = gbar;
        t.ntiles_s = cuts[3].count;
        t.depth_s = cuts[3].depth;
        t.mid = work[0].phi;  // the forward sweep is done with it
        if (split) {
            ok(launch_smooth_split(t, kSmoothTransposed, tall, cuts[3].count, s, true));
            return;
        }
        void* args[1] = {&t};
        ok(launch_kernel(sob_smooth3_unrolled_fn(R, true, tall), cuts[3].count, kSmoothThreads, 0, args, s, true));
    };
    do {
        if (!ok(cudaMemcpyAsync(pair, &a.pair0, sizeof(Pair), cudaMemcpyHostToDevice, s))) break;
        if (!ok(cudaMemsetAsync(dd, 0, 64, s))) break;
        adj_pack_kernel<<<grid, 256, 0, s>>>(A, d_S, d_T, d_v0, Sp, Tp, ckpt[0].phi, ckpt[0].m);
        // forward: a segment's first state is its checkpoint, and the last segment's states stay
        State st = ckpt[0];
        for (int k = 0; k < K && rc == FR_OK; ++k) {
            const int j = k % ck;
            const bool last_segment = k / ck == nseg - 1;
            const State to = last_segment ? seg[j] : j == ck - 1 ? ckpt[k / ck + 1] : work[k & 1];
            forward(k, st, to);
            st = to;
        }
        reverse((const void*)adj_loss_kernel, grid, A, Sp, Tp, st.phi, st.m, pbar, mbar, dd);
        if (!d_grad_v0) break;
        // reverse, one segment at a time
        for (int q = nseg - 1; q >= 0 && rc == FR_OK; --q) {
            const int s0 = q * ck, s1 = std::min(s0 + ck, K);
            if (q < nseg - 1) {
                st = ckpt[q];
                for (int k = s0; k < s1 - 1; ++k) {
                    forward(k, st, seg[k - s0]);
                    st = seg[k - s0];
                }
            }
            for (int k = s1 - 1; k >= s0; --k) {
                const float* phik = k == s0 ? ckpt[q].phi : seg[k - s0 - 1].phi;
                // a segment's last state is the next one's checkpoint
                const float* mn = k == s1 - 1 && q < nseg - 1 ? ckpt[q + 1].m : seg[k - s0].m;
                reverse(update_fn, column_blocks, A, columns, phik, mn, pbar, mbar);
                reverse((const void*)adj_momentum_kernel, grid, A, damping, step, mbar, g);
                smooth_adjoint();
                reverse(grad_fn, column_blocks, A, columns, Sp, Tp, phik, lambda, gbar, pbar, dd + 1);
            }
        }
        reverse((const void*)adj_unpack_kernel, grid, A, mbar, d_grad_v0);
    } while (0);
    double host[2] = {0.0, 0.0};
    if (rc == FR_OK) {
        if (cudaGetLastError() != cudaSuccess || cudaMemcpyAsync(host, dd, sizeof host, cudaMemcpyDeviceToHost, s) !=
                                                     cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess)
            rc = FR_ERR_CUDA;
    }
    if (rc != FR_OK) cudaStreamSynchronize(s);  // nothing may still use the workspace
    release_workspace(dev, reinterpret_cast<float*>(blk), cached);
    if (rc != FR_OK) {
        cudaGetLastError();
        set_global_error("fr_sobolev_loss_grad: a CUDA call failed");
        return rc;
    }
    *loss = host[0];
    if (grad_lambda) *grad_lambda = host[1];
    return FR_OK;
}

namespace frg {
// scatter_face_warp of one channel
__device__ __forceinline__ void scatter_face_warp(float* F, int b, const float v[4], bool act, int X) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int bprev = __shfl_up_sync(full, act ? b : -4, 1);
    const bool merge = act && lane > 0 && bprev == b - 1;
    const bool next_merges = __shfl_down_sync(full, (int)merge, 1) != 0 && lane < 31;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const float c1 = v[2 * j + 1], c1prev = __shfl_up_sync(full, c1, 1);
        if (act) {
            atomicAdd(F + b + j * X, merge ? v[2 * j] + c1prev : v[2 * j]);
            if (!next_merges) atomicAdd(F + b + 1 + j * X, c1);
        }
    }
}

// pos_bar = wbar * d img/d pos, img_bar += the trilinear weights times wbar, on the caller's
// unpadded planes.  A thread owns a column (Columns): the corners and the upper
// face of a cell that the next slice's cell stands on are kept and held back as in
// adj_update_kernel, as the reductions bound the kernel: 57 us on 160x192x160, where eight
// corners per voxel, lanes merged, took 83 us.
template <int SHAPE>
__global__ void __launch_bounds__(256) warp_adjoint_kernel(Pair P, Columns C, const float* __restrict__ pos,
                                                           const float* __restrict__ img,
                                                           const float* __restrict__ wbar, float* pos_bar,
                                                           float* img_bar) {
    const int X = P.X, XY = P.X * P.Y;
    const long long N = P.N;
    int x, y, z0, z1;
    C.place<SHAPE>(blockIdx.x, threadIdx.x, P.Z, x, y, z0, z1);
    const bool act = x < P.X && y < P.Y && (SHAPE != kLayeredColumns || z0 < z1);
    int i = act ? x + X * y + XY * z0 : 0;
    float f[8] = {}, held[4] = {};
    int above = -1;  // base of the cell above the previous slice's cell (-1: none)
    float np[3], nw = __ldg(wbar + i);  // the next slice's position and wbar
#pragma unroll
    for (int c = 0; c < 3; ++c) np[c] = __ldg(pos + c * N + i);
    for (int z = z0; z < z1; ++z, i += act ? XY : 0) {
        const SobCell s = sob_locate(P, np[0], np[1], np[2]);
        const float w = nw;
        const int b = s.base;
        const bool on = b == above;
        if (pos_bar) {
            f[1] = f[0];
            f[3] = f[2];
            f[5] = f[4];
            f[7] = f[6];
            f[0] = __ldg(img + b + 1 + X + XY);
            f[2] = __ldg(img + b + 1 + XY);
            f[4] = __ldg(img + b + X + XY);
            f[6] = __ldg(img + b + XY);
            if (!on) {
                f[1] = __ldg(img + b + 1 + X);
                f[3] = __ldg(img + b + 1);
                f[5] = __ldg(img + b + X);
                f[7] = __ldg(img + b);
            }
        }
        if (act && z + 1 < z1) {
            nw = __ldg(wbar + i + XY);
#pragma unroll
            for (int c = 0; c < 3; ++c) np[c] = __ldg(pos + c * N + i + XY);
        }
        if (pos_bar) {
            float d[3];
            tri_grad(f, s, d, nullptr, nullptr);
            if (act)
#pragma unroll
                for (int c = 0; c < 3; ++c) __stcs(pos_bar + c * N + i, w * d[c]);
        }
        if (img_bar) {  // uniform: every lane calls the warp scatter
            const bool flush = act && !on && above >= 0;
            if (__any_sync(0xffffffffu, flush)) scatter_face_warp(img_bar, above, held, flush, X);
            float low[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float k = ((q & 1) ? s.a : 1.f - s.a) * ((q & 2) ? s.b : 1.f - s.b);
                low[q] = (k * (1.f - s.c)) * w;
                if (on) low[q] += held[q];
                held[q] = (k * s.c) * w;
            }
            scatter_face_warp(img_bar, b, low, act, X);
        }
        above = b + XY;
    }
    if (img_bar) scatter_face_warp(img_bar, above, held, act && above >= 0, X);
}
}  // namespace frg

extern "C" int fr_warp_adjoint(const float* d_pos, const float* d_img, const float* d_wbar, const int dims[3],
                               float* d_pos_bar, float* d_img_bar, void* stream) {
    using namespace frg;
    set_global_error("");
    if (!d_pos || !d_img || !d_wbar || !dims || (!d_pos_bar && !d_img_bar)) {
        set_global_error("fr_warp_adjoint: NULL argument");
        return FR_ERR_INVALID_ARG;
    }
    if (dims[0] < 2 || dims[1] < 2 || dims[2] < 2 || !frg::fits_index32(dims[0], dims[1], dims[2])) {
        set_global_error("fr_warp_adjoint: invalid dims (each >= 2, N + 2 X Y + 2 X + 2 <= 2^31-1)");
        return FR_ERR_INVALID_ARG;
    }
    Pair P{};
    P.X = P.Xp = dims[0];
    P.Y = dims[1];
    P.Z = dims[2];
    P.N = (long long)dims[0] * dims[1] * dims[2];
    cudaStream_t s = (cudaStream_t)stream;
    if (d_img_bar && cudaMemsetAsync(d_img_bar, 0, sizeof(float) * (size_t)P.N, s) != cudaSuccess) {
        cudaGetLastError();
        set_global_error("fr_warp_adjoint: memset failed");
        return FR_ERR_CUDA;
    }
    // long columns hold more faces back, short ones fill the GPU: up to 16 slices while there are
    // eight blocks per SM
    Columns C(P.X, P.X, P.Y);
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    C.depth = (int)std::max(1LL, std::min(16LL, C.blocks(P.Z) / (8LL * std::max(sms, 1))));
    auto fn = C.shape == kTileColumns   ? warp_adjoint_kernel<kTileColumns>
              : C.shape == kFlatColumns ? warp_adjoint_kernel<kFlatColumns>
                                        : warp_adjoint_kernel<kLayeredColumns>;
    fn<<<(unsigned)C.blocks(P.Z), 256, 0, s>>>(P, C, d_pos, d_img, d_wbar, d_pos_bar, d_img_bar);
    if (cudaGetLastError() != cudaSuccess) {
        set_global_error("fr_warp_adjoint: launch failed");
        return FR_ERR_CUDA;
    }
    return FR_OK;
}
