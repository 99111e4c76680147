// fr_common.cuh -- shared device-side types and helpers of the fastreg GB300 kernels.
//
// Layout in HBM (all pairs of a cohort packed into one allocation per field):
//   scalar field  f[off_p + i]                    i = x + Xp*(y + Y*z), x fastest
//   vector field  f[c*NT + off_p + i], c = 0,1,2  three planes (SoA), NT = packed voxels
// Xp is X rounded up to a multiple of 4 (rows start on 16-byte boundaries); the pad
// columns are zero and never written.  off_p, the voxel offset of pair p, is a
// multiple of 32 (128 B).  The caller's buffers keep the reference's unpadded layout
// x + X*(y + Y*z); pack_init_kernel and finalize_kernel convert.
//
// Arithmetic contract (mirrored by the CPU oracle): the library is compiled with
// --fmad=false, so a*b+c is never contracted; the only fused multiply-adds are the
// explicit fmaf() calls of lerp (include/cuda/cuda_utils.hpp:43-46 of the reference).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace frg {

// Launches `fn`; with `behind` its blocks may be placed before the kernel ahead of it in the stream
// has ended, and wait in pdl_wait.
inline cudaError_t launch_kernel(const void* fn, int grid, int threads, size_t smem, void** args, cudaStream_t s,
                                 bool behind) {
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = behind ? 1 : 0;
    return cudaLaunchKernelExC(&c, fn, args);
}

// One registration pair inside a packed cohort.
struct Pair {
    int X, Y, Z;
    int Xp;         // row pitch in the packed arrays (X rounded up to a multiple of 4)
    long long off;  // voxel offset into the packed arrays
    long long N;    // Xp*Y*Z: the pair's extent in the packed arrays
    float w_reg;    // regularisation weight of this pair (W_REG unless set per pair)
    int pad_;
};

// A tile of work: pair index and the tile origin (x0, y0, z0).
typedef int4 Tile;

constexpr int kTileX = 32;  // threads along x (one warp per row)
constexpr int kTileY = 8;   // rows per block
// The solver kernels walk their own tile tables of 32 x 8 x depth tiles; the depth of
// each table and the kernel's blocks per SM are chosen on the host (fr_api.cu: defaults,
// or the autotuner's choice for the cohort's size class).

__device__ __forceinline__ long long lin(const Pair& P, int x, int y, int z) {
    return (long long)x + (long long)P.Xp * ((long long)y + (long long)P.Y * z);
}

// index of (x, y, z) in the caller's unpadded layout
__device__ __forceinline__ long long user_lin(const Pair& P, int x, int y, int z) {
    return (long long)x + (long long)P.X * ((long long)y + (long long)P.Y * z);
}

// Reads a field that an earlier kernel of a chain of programmatic launches writes (pdl_wait), and this one does
// not: an ordinary load.  __ldg and const __restrict__ kernel parameters make non-coherent loads, which are
// defined only for memory that nothing writes as long as the kernel is resident, and which the
// compiler may move above the wait.  Written out, the loads keep their place among the volatile statements,
// the wait included; as plain C++ they are put off to their use, behind the stores before it (pass A
// 0.163 instead of 0.161 ms on 182x218x182, the sobolev update 0.3545 instead of 0.3532 on 8 x 160x192x160).
__device__ __forceinline__ float chain_load(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 chain_load(const float4* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// lerp(v0, v1, t) = fma(t, v0, fma(-t, v1, v1))
__device__ __forceinline__ float lerpf_(float v0, float v1, float t) { return fmaf(t, v0, fmaf(-t, v1, v1)); }

// Sample cell: clamp to [0, dim-1], floor corner, fractional weights
// (interpolate_intensity / interpolate_field, include/cuda/cuda_utils.hpp:60-136).
struct Cell {
    long long base;  // linear index of the floor corner
    int gx, gy, gz;
    float a, b, c;
};

__device__ __forceinline__ Cell locate(const Pair& P, float px, float py, float pz) {
    Cell cl;
    float cx = fminf(fmaxf(0.f, px), (float)(P.X - 1));
    float cy = fminf(fmaxf(0.f, py), (float)(P.Y - 1));
    float cz = fminf(fmaxf(0.f, pz), (float)(P.Z - 1));
    cl.gx = (int)floorf(cx);
    cl.gy = (int)floorf(cy);
    cl.gz = (int)floorf(cz);
    cl.a = cx - (float)cl.gx;
    cl.b = cy - (float)cl.gy;
    cl.c = cz - (float)cl.gz;
    cl.base = lin(P, cl.gx, cl.gy, cl.gz);
    return cl;
}

// Trilinear sample with the unchecked corner addressing of the reference's
// Volume/VectorField operator(): the +1 corner of a cell on the upper face aliases
// to the next row/slice (weight 0 there); an index past the last voxel is clamped.
// F points at the pair's plane (already offset by off_p).
__device__ __forceinline__ float tri_unchecked(const float* __restrict__ F, const Pair& P, const Cell& cl) {
    const long long X = P.Xp, XY = (long long)P.Xp * P.Y, last = P.N - 1;
    const long long b = cl.base;
    auto at = [&](long long d) -> float {
        long long j = b + d;
        return __ldg(F + (j < last ? j : last));
    };
    float f111 = at(1 + X + XY), f110 = at(1 + X), f101 = at(1 + XY), f100 = at(1);
    float f011 = at(X + XY), f010 = at(X), f001 = at(XY), f000 = __ldg(F + b);
    return lerpf_(lerpf_(lerpf_(f111, f110, cl.c), lerpf_(f101, f100, cl.c), cl.b),
                  lerpf_(lerpf_(f011, f010, cl.c), lerpf_(f001, f000, cl.c), cl.b), cl.a);
}

// ---- 32-bit variants used inside one pair (N < 2^31) ----

struct Cell32 {
    int base;  // linear index of the floor corner inside the pair
    int gx, gy, gz;
    float a, b, c;
};

// X, Y, Z: grid extents; Xp: row pitch of the array the cell indexes
__device__ __forceinline__ Cell32 locate32(int X, int Y, int Z, int Xp, float px, float py, float pz) {
    Cell32 cl;
    const float cx = fminf(fmaxf(0.f, px), (float)(X - 1));
    const float cy = fminf(fmaxf(0.f, py), (float)(Y - 1));
    const float cz = fminf(fmaxf(0.f, pz), (float)(Z - 1));
    cl.gx = (int)floorf(cx);
    cl.gy = (int)floorf(cy);
    cl.gz = (int)floorf(cz);
    cl.a = cx - (float)cl.gx;
    cl.b = cy - (float)cl.gy;
    cl.c = cz - (float)cl.gz;
    cl.base = cl.gx + Xp * (cl.gy + Y * cl.gz);
    return cl;
}

__device__ __forceinline__ float trilerp(float f111, float f110, float f101, float f100, float f011, float f010,
                                         float f001, float f000, float a, float b, float c) {
    return lerpf_(lerpf_(lerpf_(f111, f110, c), lerpf_(f101, f100, c), b),
                  lerpf_(lerpf_(f011, f010, c), lerpf_(f001, f000, c), b), a);
}

// Two lerps as one packed FP32 pair: per lane exactly lerpf_(v0, v1, t) (both fused
// multiply-adds of a lane are the lane's own, rounded once each).  nt = -t, passed in so
// that a cell's negated weights are formed once.
__device__ __forceinline__ float2 lerp2_(float2 v0, float2 v1, float2 t, float2 nt) {
    return __ffma2_rn(t, v0, __ffma2_rn(nt, v1, v1));
}

// two trilerps as one packed pair, each lane with its own corner values and weights
__device__ __forceinline__ float2 trilerp2w(float2 f111, float2 f110, float2 f101, float2 f100, float2 f011,
                                            float2 f010, float2 f001, float2 f000, float2 ta, float2 tb, float2 tc) {
    const float2 na = make_float2(-ta.x, -ta.y), nb = make_float2(-tb.x, -tb.y), nc = make_float2(-tc.x, -tc.y);
    return lerp2_(lerp2_(lerp2_(f111, f110, tc, nc), lerp2_(f101, f100, tc, nc), tb, nb),
                  lerp2_(lerp2_(f011, f010, tc, nc), lerp2_(f001, f000, tc, nc), tb, nb), ta, na);
}

// trilerp of two fields at one cell as one packed pair (lane 0: field 0, lane 1: field 1)
__device__ __forceinline__ float2 trilerp2(float2 f111, float2 f110, float2 f101, float2 f100, float2 f011,
                                           float2 f010, float2 f001, float2 f000, float a, float b, float c) {
    return trilerp2w(f111, f110, f101, f100, f011, f010, f001, f000, make_float2(a, a), make_float2(b, b),
                     make_float2(c, c));
}

// trilerp of three fields' corners f[k][0..7] (order 111, 110, 101, 100, 011, 010, 001, 000)
// at one cell: fields 0 and 1 as one packed pair, field 2 alone; per field exactly trilerp
__device__ __forceinline__ void trilerp3(const float f[3][8], float a, float b, float c, float out[3]) {
    auto p = [&](int q) { return make_float2(f[0][q], f[1][q]); };
    const float2 r = trilerp2(p(0), p(1), p(2), p(3), p(4), p(5), p(6), p(7), a, b, c);
    out[0] = r.x;
    out[1] = r.y;
    out[2] = trilerp(f[2][0], f[2][1], f[2][2], f[2][3], f[2][4], f[2][5], f[2][6], f[2][7], a, b, c);
}

// tri_unchecked with 32-bit indices: corners past the last voxel (only possible when
// the cell touches the end of the array) are clamped on a slow path.  X, XY, N are the
// strides and extent of the array (pitched for the packed arrays).
__device__ __forceinline__ float tri_unchecked32(const float* __restrict__ F, int X, int XY, int N, const Cell32& cl) {
    const int b = cl.base;
    if (b + 1 + X + XY <= N - 1) {
        return trilerp(__ldg(F + b + 1 + X + XY), __ldg(F + b + 1 + X), __ldg(F + b + 1 + XY), __ldg(F + b + 1),
                       __ldg(F + b + X + XY), __ldg(F + b + X), __ldg(F + b + XY), __ldg(F + b), cl.a, cl.b, cl.c);
    }
    const int last = N - 1;
    return trilerp(__ldg(F + min(b + 1 + X + XY, last)), __ldg(F + min(b + 1 + X, last)),
                   __ldg(F + min(b + 1 + XY, last)), __ldg(F + min(b + 1, last)), __ldg(F + min(b + X + XY, last)),
                   __ldg(F + min(b + X, last)), __ldg(F + min(b + XY, last)), __ldg(F + b), cl.a, cl.b, cl.c);
}

// The three components of a vector field (planes F0, F1, F2) at one cell with get_global_idx
// addressing (include/cuda/cuda_utils.hpp:31-37, 109-136): a corner outside the grid reads element 0.
// X, Y, Z: grid extents; Xp, XYp: strides of the array.  Components 0 and 1 are interpolated as one
// packed pair.  The field is one that the chain of launches writes (chain_load).
__device__ __forceinline__ void tri_checked32_3(const float* F0, const float* F1,
                                                const float* F2, int X, int Y, int Z, int Xp, int XYp,
                                                const Cell32& cl, float out[3]) {
    const int b = cl.base;
    const bool ox = cl.gx + 1 < X, oy = cl.gy + 1 < Y, oz = cl.gz + 1 < Z;
    const float* const F[3] = {F0, F1, F2};
    float f[3][8];
    if (ox && oy && oz) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            f[k][0] = chain_load(F[k] + b + 1 + Xp + XYp);
            f[k][1] = chain_load(F[k] + b + 1 + Xp);
            f[k][2] = chain_load(F[k] + b + 1 + XYp);
            f[k][3] = chain_load(F[k] + b + 1);
            f[k][4] = chain_load(F[k] + b + Xp + XYp);
            f[k][5] = chain_load(F[k] + b + Xp);
            f[k][6] = chain_load(F[k] + b + XYp);
            f[k][7] = chain_load(F[k] + b);
        }
    } else {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float f0 = chain_load(F[k]);
            f[k][0] = (ox && oy && oz) ? chain_load(F[k] + b + 1 + Xp + XYp) : f0;
            f[k][1] = (ox && oy) ? chain_load(F[k] + b + 1 + Xp) : f0;
            f[k][2] = (ox && oz) ? chain_load(F[k] + b + 1 + XYp) : f0;
            f[k][3] = ox ? chain_load(F[k] + b + 1) : f0;
            f[k][4] = (oy && oz) ? chain_load(F[k] + b + Xp + XYp) : f0;
            f[k][5] = oy ? chain_load(F[k] + b + Xp) : f0;
            f[k][6] = oz ? chain_load(F[k] + b + XYp) : f0;
            f[k][7] = chain_load(F[k] + b);
        }
    }
    trilerp3(f, cl.a, cl.b, cl.c, out);
}

// tri_unchecked32 on an interleaved 4-channel field (one 16-byte load per corner) that the
// chain of launches writes (chain_load)
__device__ __forceinline__ float4 tri_unchecked32_f4(const float4* F, int X, int XY, int N,
                                                     const Cell32& cl) {
    const int b = cl.base;
    int o111 = b + 1 + X + XY, o110 = b + 1 + X, o101 = b + 1 + XY, o100 = b + 1;
    int o011 = b + X + XY, o010 = b + X, o001 = b + XY;
    if (o111 > N - 1) {
        const int last = N - 1;
        o111 = min(o111, last);
        o110 = min(o110, last);
        o101 = min(o101, last);
        o100 = min(o100, last);
        o011 = min(o011, last);
        o010 = min(o010, last);
        o001 = min(o001, last);
    }
    const float4 f111 = chain_load(F + o111), f110 = chain_load(F + o110), f101 = chain_load(F + o101), f100 = chain_load(F + o100);
    const float4 f011 = chain_load(F + o011), f010 = chain_load(F + o010), f001 = chain_load(F + o001), f000 = chain_load(F + b);
    // channels (x, y) and (z, w) as packed pairs: per channel exactly trilerp
    auto lo = [](float4 v) { return make_float2(v.x, v.y); };
    auto hi = [](float4 v) { return make_float2(v.z, v.w); };
    const float2 r0 = trilerp2(lo(f111), lo(f110), lo(f101), lo(f100), lo(f011), lo(f010), lo(f001), lo(f000), cl.a,
                               cl.b, cl.c);
    const float2 r1 = trilerp2(hi(f111), hi(f110), hi(f101), hi(f100), hi(f011), hi(f010), hi(f001), hi(f000), cl.a,
                               cl.b, cl.c);
    return make_float4(r0.x, r0.y, r1.x, r1.y);
}

// Programmatic dependent launch: waits until the kernels that this one was launched behind have
// completed and their writes are visible (an ordinary launch has nothing to wait for).  The kernels
// leave the trigger to their blocks' exits: it saves part of the launch latency between two
// kernels (64^3: 22.1 -> 21.5 us per iteration), while triggering early places blocks that hold
// SM room and wait (27.6 us).
//
// A kernel launched this way may be resident before the one ahead has completed, so what the kernels of
// a chain write is read with chain_load, by asynchronous copies or by plain loads, and every thread
// waits before its first access.  __ldg is for what stays as it is for the whole chain: the
// images, the labels and the pair table.  The first kernel behind the one that packs the images
// is therefore an ordinary launch, or has a copy or a clearing between the two.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The t-th tile of a kernel's table of 32 x rows x depth tiles and its pair; false if the pair has
// converged.  A cohort's tiles, pairs and stop words are read from memory.  Of a single pair (args.single)
// the tile follows from t and the pair from the kernel's arguments, and without a convergence
// test (args.check_stop) there is no stop word to read: two dependent loads less before a block's
// first useful one.  The pair's weight always comes from the table, where it may change between
// launches of a captured graph; nothing waits for it here.
template <typename Args>
__device__ __forceinline__ bool take_tile(const Args& a, const Tile* tiles, int t, int rows, int depth, Tile& tl, Pair& P) {
    if (a.single) {
        if (a.check_stop && a.stop[0]) return false;
        P = a.pair0;
        P.w_reg = __ldg(&a.pairs[0].w_reg);
        const int nx = (P.X + kTileX - 1) / kTileX, ny = (P.Y + rows - 1) / rows;
        const int row = t / nx, z = row / ny;
        tl = make_int4(0, (t - row * nx) * kTileX, (row - z * ny) * rows, z * depth);
        return true;
    }
    tl = tiles[t];
    if (a.check_stop && a.stop[tl.x]) return false;
    P = a.pairs[tl.x];
    return true;
}

// The update kernels' last step for a tile: the pair's largest update norm of this iteration.
// Without a convergence test it is recorded at once; with one, the last block does
// (record_and_test).
template <typename Args>
__device__ __forceinline__ void note_max(const Args& a, int pair, unsigned long long key) {
    if (key) atomicMax(a.check_stop ? a.keys + pair : a.trace + (long long)(a.iter - 1) * a.npairs + pair, key);
}

// With a convergence test: the last block of the grid to finish records the iteration's largest
// norms and stops the pairs whose norm is small enough.
template <typename Args>
__device__ __forceinline__ void record_and_test(const Args& a) {
    if (!a.check_stop) return;
    __shared__ bool last;
    const int tid = threadIdx.x;
    __threadfence();
    __syncthreads();
    if (tid == 0) last = (atomicAdd(a.counter, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int p = tid; p < a.npairs; p += blockDim.x) {
        if (a.stop[p]) continue;
        const unsigned long long k = atomicExch(a.keys + p, 0ull);
        a.trace[(long long)(a.iter - 1) * a.npairs + p] = k;
        const float mx = __uint_as_float((unsigned)(k >> 32));
        if (mx <= a.max_update_norm) a.stop[p] = a.iter;
    }
    if (tid == 0) *a.counter = 0u;
}

// Hint that the 128-byte line holding *p will be read soon: it is fetched into L2 with
// no register written and nothing waited for (p must point into an allocation).
__device__ __forceinline__ void prefetch_l2(const void* p) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// ---- asynchronous global -> shared copies (cp.async, 4 bytes each) ----
__device__ __forceinline__ void cp_async4(float* smem, const float* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
// 16-byte copy that bypasses L1; both addresses 16-byte aligned
__device__ __forceinline__ void cp_async16(float* smem, const float* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
// the same, or 16 bytes of zeros (nothing is read then)
__device__ __forceinline__ void cp_async16_or_zero(float* smem, const float* gmem, bool copy) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(copy ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int Pending>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(Pending) : "memory");
}

// ---- slices of a 32 x 8 column tile staged in shared memory ----
// A staged slice of a plane with y halo H is 8 + 2H rows (y0 - H .. y0 + 7 + H) of
// kStageChunks aligned 16-byte chunks (columns x0 - 4 .. x0 + 35; column x0 + tx sits at
// row offset tx + kStageXO).  Thread e copies chunk e of every slice and component of the
// tile: its shared-memory offset is 4e floats, and its offset inside a slice, fixed for
// the tile, is returned here (-1: no chunk, or the chunk lies outside the padded volume,
// where no voxel of the tile reads).
constexpr int kStageXO = 4, kStageW = kTileX + 2 * kStageXO, kStageChunks = kStageW / 4;
template <int H>
__device__ __forceinline__ int stage_offset(int e, int Y, int Xp, int x0, int y0) {
    constexpr int R = kTileY + 2 * H;
    static_assert(R * kStageChunks <= 256, "one chunk per thread of a 256-thread block");
    if (e >= R * kStageChunks) return -1;
    const int r = e / kStageChunks, k = e - r * kStageChunks;
    const int y = y0 - H + r, x = x0 - kStageXO + 4 * k;
    if (y < 0 || y >= Y || x < 0 || x >= Xp) return -1;
    return Xp * y + x;
}

// sqrt rounded toward -inf (reference norm(), include/cuda/cuda_utils.hpp:251-253)
__device__ __forceinline__ float norm3_rd(float x, float y, float z) {
    return __fsqrt_rd((x * x + y * y) + z * z);
}

// (norm, index) packed so that a larger key means a larger norm and, for equal
// norms, a lower linear index.  norm >= 0, so its IEEE bits order like the value.
__device__ __forceinline__ unsigned long long norm_key(float nrm, long long idx) {
    return ((unsigned long long)__float_as_uint(nrm) << 32) | (unsigned long long)(0xffffffffu - (unsigned)idx);
}

// Block-wide max of a 64-bit key; every thread must call it.  Returns the block max
// in thread 0.
__device__ __forceinline__ unsigned long long block_max_u64(unsigned long long k, unsigned long long* smem) {
    for (int o = 16; o > 0; o >>= 1) {
        unsigned long long other = __shfl_xor_sync(0xffffffffu, k, o);
        k = other > k ? other : k;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) smem[warp] = k;
    __syncthreads();
    const int nw = blockDim.x >> 5;
    if (warp == 0) {
        k = lane < nw ? smem[lane] : 0ull;
        for (int o = 16; o > 0; o >>= 1) {
            unsigned long long other = __shfl_xor_sync(0xffffffffu, k, o);
            k = other > k ? other : k;
        }
    }
    __syncthreads();
    return k;
}

__device__ __forceinline__ double block_sum_f64(double v, double* smem) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) smem[warp] = v;
    __syncthreads();
    const int nw = blockDim.x >> 5;
    if (warp == 0) {
        v = lane < nw ? smem[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    __syncthreads();
    return v;
}

}  // namespace frg
