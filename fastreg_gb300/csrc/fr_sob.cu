// fr_sob.cu -- kernels of the sobolev solver (see fr_sob.h for the iteration).
//
// Launches per iteration: sob_grad_kernel (W, residual, exact trilinear gradient, graph
// Laplacian), sob_smooth3_kernel (fr_smooth.cu: separable Gaussian along x, y, z
// fused with the momentum update), sob_pass_b_kernel (compositional update, max update norm,
// on-device convergence test).
#include <cmath>
#include <type_traits>

#include "fr_common.cuh"
#include "fr_kernels.h"
#include "fr_sob.h"
#include "fr_tma.cuh"

namespace frg {

void gaussian_taps(float sigma, int width, float* taps) {
    const int R = width / 2;
    double w[kMaxSmoothWidth];
    double sum = 0.0;
    for (int k = -R; k <= R; ++k) {
        w[k + R] = std::exp(-(double)k * (double)k / (2.0 * (double)sigma * (double)sigma));
        sum += w[k + R];
    }
    for (int k = 0; k < width; ++k) taps[k] = (float)(w[k] / sum);
}

void fold_weights(const float* taps, int radius, float* fold) {
    for (int k = 0; k <= radius; ++k) {
        double sum = 0.0;
        for (int q = 0; q < radius - k; ++q) sum += (double)taps[q];
        fold[k] = (float)sum;
    }
}

// W = S o phi, r = W - T, g = r * (exact trilinear gradient of the interpolant) + w_reg * (graph
// Laplacian of u = phi - x).
//
// A block owns a 32 x 8 column tile and marches z, one voxel per thread and slice.  phi's three
// components (the tile and a 1-voxel halo) and T are staged slice by slice in a ring of kGS
// shared-memory slots; the eight corners of S are gathered through L1.  A thread keeps its own
// column of phi in registers from slice to slice, and the Laplacian's term across a z face is
// formed once and enters the next slice's sum negated: (p - q) + d and (q - p) - d differ in
// sign only, and adding the zero of either sign to a sum that is not -0 gives the same bits
// (a sum that starts from +0 is never -0).
//
// With TMA staging a ninth warp fills the ring, two tensor copies per slice, and warps do not
// wait on one another: each waits for a slice's full barrier and arrives on its empty barrier
// when it has read the slot, and the filling thread waits for the slot's eight arrivals.  The
// cp.async variant stages one chunk per thread and component, with a block barrier per slice.
//
// Bound by issue slots (73% used, 59 million warp instructions on the 182x218x182 pair) and by
// the corner loads' latency: 70.6 us there, where every thread waiting at a block barrier per
// slice, seven shared-memory reads per component and an FP64 sum that nothing read took 82.5 us
// (72.6 million instructions; 32 bytes per voxel are 34 us at the copy bandwidth).  Four blocks
// (56 registers) with TMA: five need 40 registers, spill and take 100 us; six cp.async blocks
// 75 us, five 79 us.  Four slots: three take 73 us, five 71 us.  Warps that own four rows
// each, with the rows' values in registers, execute 42 million instructions but hold only 16
// warps per SM and take 78 us.
namespace {
constexpr int kGS = 4;                               // ring slots: slices z and z + 1, the others in flight
constexpr int kGW = kStageW, kGPlane = kGW * (kTileY + 2);  // box row and plane (floats)
constexpr int kGTOff = (3 * kGPlane + 31) / 32 * 32;  // T's offset in a slot (128-byte aligned)
constexpr int kGSlot = kGTOff + kTileX * kTileY;
constexpr unsigned kGBytes = sizeof(float) * (3 * kGPlane + kTileX * kTileY);
static_assert(kGSlot % 32 == 0, "slots on 128-byte boundaries");
}  // namespace

size_t sob_grad_smem_bytes() { return sizeof(float) * kGS * kGSlot + 2 * sizeof(uint64_t) * kGS; }

template <bool TMA>
__global__ void __launch_bounds__(sob_grad_threads(TMA), TMA ? 4 : 6) sob_grad_kernel(SobIterArgs a) {
    pdl_wait();
    extern __shared__ __align__(128) unsigned char grad_raw[];
    float* ring = reinterpret_cast<float*>(grad_raw);
    if (TMA && !ring_aligned(ring, a.err)) return;
    uint64_t* full = reinterpret_cast<uint64_t*>(ring + kGS * kGSlot);
    uint64_t* empty = full + kGS;
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
    if (TMA) {
        if (tid == 0) {
            for (int k = 0; k < kGS; ++k) {
                mbar_init(full + k, 1);
                mbar_init(empty + k, 8);
            }
            mbar_fence_init();
        }
        __syncthreads();
        if (ty == 8) {  // the filling warp: one thread copies every slice of the block's tiles in order
            if (tx != 0) return;
            unsigned n = 0;  // fills: fill n goes to slot n % kGS, the (n / kGS)-th of that slot
            bool ok = true;
            for (int t = blockIdx.x; t < a.ntiles_g && ok; t += gridDim.x) {
                Tile tl;
                Pair P;
                if (!take_tile(a, a.tiles_g, t, kTileY, a.depth_g, tl, P)) continue;
                const CUtensorMap* maps = a.tmaps + (long long)tl.x * TM_COUNT;
                const int z1 = min(tl.w + a.depth_g, P.Z);
                for (int z = tl.w - 1; z <= z1 && ok; ++z, ++n) {
                    const int k = SliceRing<kGS>::slot(n);
                    // the slot's previous reader has released it (an unused slot counts as released)
                    ok = mbar_wait_bounded(empty + k, SliceRing<kGS>::parity(n) ^ 1u);
                    if (!ok) break;
                    mbar_arrive_expect_tx(full + k, kGBytes);
                    tma_load_4d(ring + k * kGSlot, maps + TM_LAP_PSI, tl.y - 4, tl.z - 1, z, 0, full + k);
                    tma_load_3d(ring + k * kGSlot + kGTOff, maps + TM_LAP_T, tl.y, tl.z, z, full + k);
                }
            }
            // the copies in flight end (bounded) before this thread, and with it the block's shared memory, goes:
            // also when it saw no failure itself, as a warp that gave up on one of the last fills has left
            drain_fills<kGS>(n, [&](int k, unsigned parity) { mbar_wait_bounded(full + k, parity); });
            if (!ok) atomicOr(a.err, kErrTmaTimeout);
            return;
        }
    }
    int slot = 0;           // slots are read in order
    unsigned full_ph = 0u;  // bit k: parity of slot k's next fill
    bool failed = false;

    for (int t = blockIdx.x; t < a.ntiles_g && !failed; t += gridDim.x) {
        Tile tl;
        Pair P;
        if (!take_tile(a, a.tiles_g, t, kTileY, a.depth_g, tl, P)) continue;  // uniform over the block
        const int X = P.X, Y = P.Y, Z = P.Z, Xp = P.Xp, XYp = P.Xp * P.Y;  // strides of the packed arrays
        const long long NT = a.NT;
        const float* __restrict__ S = a.S + P.off;
        const int x = tl.y + tx, y = tl.z + ty;
        const bool inside = x < X && y < Y;
        const int z0 = tl.w, z1 = min(tl.w + a.depth_g, Z);  // slices z0 - 1 .. z1 are staged
        // cp.async: this thread's chunk of a slice of phi, and of T (threads below 64)
        const int gq = TMA ? -1 : stage_offset<1>(tid, Y, Xp, tl.y, tl.z);
        const int tr = tid >> 3, tk = tid & 7;
        const int gt = !TMA && tid < 64 && tl.z + tr < Y && tl.y + 4 * tk < Xp ? Xp * (tl.z + tr) + tl.y + 4 * tk : -1;
        auto stage = [&](int z, int k) {  // cp.async: slice z into slot k (one group)
            if (TMA) return;
            if (z >= 0 && z < Z && z <= z1) {
                float* dst = ring + k * kGSlot;
                if (gq >= 0)
#pragma unroll
                    for (int c = 0; c < 3; ++c)
                        cp_async16(dst + c * kGPlane + 4 * tid, a.phi + c * NT + P.off + gq + XYp * z);
                if (gt >= 0) cp_async16(dst + kGTOff + 4 * tid, a.T + P.off + gt + XYp * z);
            }
            cp_async_commit();
        };
        auto next_slice = [&]() {  // the next slice in order has landed; its slot
            const int k = slot;
            if (TMA) {
                const bool ok = mbar_wait_bounded(full + k, (full_ph >> k) & 1u);
                if (!__all_sync(0xffffffffu, ok)) failed = true;
                full_ph ^= 1u << k;
            } else {
                cp_async_wait<kGS - 3>();
                __syncthreads();
            }
            slot = slot + 1 == kGS ? 0 : slot + 1;
            return k;
        };
        auto release = [&](int k) {  // this warp has read slot k
            if (TMA) {
                __syncwarp();
                if (tx == 0) mbar_arrive(empty + k);
            }
        };
        if (!TMA) {
            __syncthreads();  // the previous tile is done with the ring
            slot = 0;
#pragma unroll
            for (int k = 0; k < kGS - 1; ++k) stage(z0 - 1 + k, k);
        }
        const bool xl = x > 0, xr = x < X - 1;
        const bool y_edge = y == 0 || y >= Y - 1;  // uniform over the warp
        const int c0 = (ty + 1) * kGW + tx + kStageXO;
        // phi of this column at the slice computed, and the Laplacian's terms across the
        // voxel's z face towards the slice above
        float cur[3], up[3];
        int at = next_slice();
#pragma unroll
        for (int c = 0; c < 3; ++c) up[c] = ring[at * kGSlot + c0 + c * kGPlane];
        release(at);
        stage(z0 - 1 + kGS - 1, kGS - 1);
        at = next_slice();
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            cur[c] = ring[at * kGSlot + c0 + c * kGPlane];
            up[c] = c == 2 ? (up[c] - cur[c]) + 1.f : up[c] - cur[c];
        }
        int i = x + Xp * y + XYp * z0;
        float* const G[3] = {a.g + P.off, a.g + NT + P.off, a.g + 2 * NT + P.off};
        for (int z = z0; z < z1; ++z, i += XYp) {
            const float* q0 = ring + at * kGSlot;
            const int above = next_slice();
            if (TMA && failed) break;
            stage(z - 1 + kGS, at == 0 ? kGS - 1 : at - 1);  // the slot of slice z - 1
            if (inside) {
                const float* qp = ring + above * kGSlot + c0;
                const SobCell s = sob_locate(P, cur[0], cur[1], cur[2]);
                const float* b = S + s.base;
                const float f000 = __ldg(b), f100 = __ldg(b + 1);
                const float f010 = __ldg(b + Xp), f110 = __ldg(b + 1 + Xp);
                const float f001 = __ldg(b + XYp), f101 = __ldg(b + 1 + XYp);
                const float f011 = __ldg(b + Xp + XYp), f111 = __ldg(b + 1 + Xp + XYp);
                // neighbours inside the grid, in the order -x, +x, -y, +y, -z, +z
                // (shared-memory work placed between the corner loads and their use)
                float lap[3];
                auto laplacian = [&](auto edge) {
                    constexpr bool kEdge = decltype(edge)::value;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const float* q = q0 + c0 + c * kGPlane;
                        const float p = cur[c], n = qp[c * kGPlane];
                        const float dx = p - q[-1], ux = p - q[1], dy = p - q[-kGW], uy = p - q[kGW], uz = p - n;
                        float acc = 0.f;
                        if (xl) acc = acc + (c == 0 ? dx - 1.f : dx);
                        if (xr) acc = acc + (c == 0 ? ux + 1.f : ux);
                        if (!kEdge || y > 0) acc = acc + (c == 1 ? dy - 1.f : dy);
                        if (!kEdge || y < Y - 1) acc = acc + (c == 1 ? uy + 1.f : uy);
                        if (!kEdge || z > 0) acc = acc - up[c];
                        up[c] = c == 2 ? uz + 1.f : uz;
                        if (!kEdge || z < Z - 1) acc = acc + up[c];
                        lap[c] = acc;
                        cur[c] = n;
                    }
                };
                if (y_edge || z == 0 || z == Z - 1)
                    laplacian(std::true_type{});
                else
                    laplacian(std::false_type{});
                const float tv = q0[kGTOff + ty * kTileX + tx];
                const float e11 = lerpf_(f111, f110, s.c), e10 = lerpf_(f101, f100, s.c);
                const float e01 = lerpf_(f011, f010, s.c), e00 = lerpf_(f001, f000, s.c);
                const float A1 = lerpf_(e11, e10, s.b), A0 = lerpf_(e01, e00, s.b);
                const float W = lerpf_(A1, A0, s.a);
                const float dWa = s.in_x ? A1 - A0 : 0.f;
                const float dWb = s.in_y ? lerpf_(e11 - e10, e01 - e00, s.a) : 0.f;
                const float dWc = s.in_z ? lerpf_(lerpf_(f111 - f110, f101 - f100, s.b),
                                                  lerpf_(f011 - f010, f001 - f000, s.b), s.a)
                                         : 0.f;
                const float r = W - tv;
                G[0][i] = (r * dWa) + (P.w_reg * lap[0]);
                G[1][i] = (r * dWb) + (P.w_reg * lap[1]);
                G[2][i] = (r * dWc) + (P.w_reg * lap[2]);
            }
            release(at);
            at = above;
        }
        if (!failed) release(at);
        if (!TMA) cp_async_wait<0>();
    }
    if (TMA && failed && tx == 0) atomicOr(a.err, kErrTmaTimeout);
}

const void* sob_grad_fn(int tma) {
    return tma ? (const void*)sob_grad_kernel<true> : (const void*)sob_grad_kernel<false>;
}

// phi += m o phi with the max update norm.  phi is smooth, so the cell of slice z + 1 is often
// the one above this slice's: its lower corners are then the upper ones already in registers,
// and a lane loads 12 corners instead of 24.  The kernel is bound by the gathers' trips through
// L1 (its data pipe 68% busy with 24 corners, several cache lines per load), then by their
// latency: 80 us on the 182x218x182 pair, where 24 corners and an L2 prefetch of the next
// cell's rows took 92 us (86 us with the reuse and the prefetch: it only adds to the L1
// queue now).  Four blocks of 64 registers; five would spill the kept corners, three take 81 us.
// The reference solver's pass B, whose psi stays near the grid, gains nothing from the
// reuse (73 against 66 us): its loads mostly hit the same lines, and it needs the warps.
// UNROLLED: from phi to phi_n, without the update norm and the convergence test; else in place.
template <bool UNROLLED>
__global__ void __launch_bounds__(256, 4) sob_pass_b_kernel(SobIterArgs a) {
    pdl_wait();
    constexpr bool NORM = !UNROLLED;
    __shared__ unsigned long long red[32];
    for (int t = blockIdx.x; t < a.ntiles_b; t += gridDim.x) {
        Tile tl;
        Pair P;
        if (!take_tile(a, a.tiles_b, t, kTileY, a.depth_b, tl, P)) continue;  // uniform over the block
        const int x = tl.y + (int)(threadIdx.x & 31), y = tl.z + (int)(threadIdx.x >> 5);
        unsigned long long best = 0ull;
        if (x < P.X && y < P.Y) {
            const long long NT = a.NT;
            const int X = P.Xp, XY = P.Xp * P.Y;  // strides of the packed arrays
            float* phi_n[3] = {a.phi_n + P.off, a.phi_n + NT + P.off, a.phi_n + 2 * NT + P.off};
            const float* phi[3] = {phi_n[0], phi_n[1], phi_n[2]};
            if (UNROLLED)
                for (int c = 0; c < 3; ++c) phi[c] = a.phi + c * NT + P.off;
            const float* mc[3] = {a.m_n + P.off, a.m_n + NT + P.off, a.m_n + 2 * NT + P.off};
            const int z1 = min(tl.w + a.depth_b, P.Z);
            int i = x + X * y + XY * tl.w;
            // phi of the next slice is loaded while this slice's gathers are in flight
            float nx = phi[0][i], ny = phi[1][i], nz = phi[2][i];
            float f[3][8];  // corners 111, 110, 101, 100, 011, 010, 001, 000 (x, y, z) of m's components
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int q = 0; q < 8; ++q) f[c][q] = 0.f;
            int above = -1;  // base of the cell whose lower corners are the upper ones in f (-1: none)
            for (int z = tl.w; z < z1; ++z, i += XY) {
                const float px = nx, py = ny, pz = nz;
                if (z + 1 < z1) {
                    nx = phi[0][i + XY];
                    ny = phi[1][i + XY];
                    nz = phi[2][i + XY];
                }
                const SobCell s = sob_locate(P, px, py, pz);
                float u[3];
                const int b = s.base;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    f[c][1] = f[c][0];
                    f[c][3] = f[c][2];
                    f[c][5] = f[c][4];
                    f[c][7] = f[c][6];
                    const float* F = mc[c];
                    f[c][0] = chain_load(F + b + 1 + X + XY);
                    f[c][2] = chain_load(F + b + 1 + XY);
                    f[c][4] = chain_load(F + b + X + XY);
                    f[c][6] = chain_load(F + b + XY);
                }
                if (b != above)
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const float* F = mc[c];
                        f[c][1] = chain_load(F + b + 1 + X);
                        f[c][3] = chain_load(F + b + 1);
                        f[c][5] = chain_load(F + b + X);
                        f[c][7] = chain_load(F + b);
                    }
                above = b + XY;
                trilerp3(f, s.a, s.b, s.c, u);
                phi_n[0][i] = px + u[0];
                phi_n[1][i] = py + u[1];
                phi_n[2][i] = pz + u[2];
                const float nrm = NORM ? norm3_rd(u[0], u[1], u[2]) : 0.f;
                if (NORM && nrm == nrm) {
                    const unsigned long long k = norm_key(nrm, i);
                    best = k > best ? k : best;
                }
            }
        }
        if (!NORM) continue;
        const unsigned long long bm = block_max_u64(best, red);
        if (threadIdx.x == 0) note_max(a, tl.x, bm);
    }
    if (NORM) record_and_test(a);
}

const void* sob_pass_b_fn(bool unrolled) {
    return unrolled ? (const void*)sob_pass_b_kernel<true> : (const void*)sob_pass_b_kernel<false>;
}

cudaError_t launch_sob_kernel(int k, const SobIterArgs& a, int grid, int variant, cudaStream_t s, bool behind) {
    void* args[1] = {const_cast<SobIterArgs*>(&a)};
    if (k == 0) return launch_kernel(sob_grad_fn(variant), grid, sob_grad_threads(variant), sob_grad_smem_bytes(), args, s, behind);
    if (k == 1 && (variant & kSplit))
        return launch_smooth_split(a, variant & kUnrolled ? kSmoothUnrolled : kSmoothInPlace, variant & 2, grid, s, behind);
    if (k == 1)
        return launch_kernel(variant & kUnrolled ? sob_smooth3_unrolled_fn(a.radius, false, variant & 2)
                                                 : sob_smooth3_fn(a.radius, variant & 1, variant & 2),
                             grid, kSmoothThreads, 0, args, s, behind);
    return launch_kernel(sob_pass_b_fn(variant & kUnrolled), grid, 256, 0, args, s, behind);
}

cudaError_t launch_sob_iter(const SobIterArgs& a, const int* grids, const int* variants, cudaStream_t s,
                            bool behind, cudaEvent_t* ev) {
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < 3 && e == cudaSuccess; ++k) {
        if (ev) cudaEventRecord(ev[k], s);
        e = launch_sob_kernel(k, a, grids[k], variants[k], s, behind);
    }
    if (ev) cudaEventRecord(ev[3], s);
    return e;
}

}  // namespace frg
