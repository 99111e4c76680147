// fr_ref.cu -- reference-mode solver kernels (the accelerated PDE flow of fastreg).
//
// One iteration of estimate_psi (src/fastreg/cuda/solver.cu:329-433) is three
// launches over a packed cohort of pairs:
//   ref_laplacian_kernel  L = -Laplacian(psi) on the interior    (vector_fields.cu:275-300)
//   ref_pass_a_kernel     divergence + density, J(psi_inv) and its determinant, the
//                         potential gradient with L o psi_inv and T o psi_inv gathered
//                         on the fly, (Dv)v, the upwind velocity Laplacian, the
//                         velocity update and the psi_inv update -- all fused
//                         (solver.cu:56-289, vector_fields.cu:231-404,503-535)
//   ref_pass_b_kernel     psi += alpha * v o psi with the max-update-norm reduction
//                         and the on-device convergence test (solver.cu:230-247,
//                         reductor.cu:426-539, solver.cu:407-421)
// rho, v and psi_inv are double-buffered because pass A reads neighbours of the old
// values while writing the new ones; psi is updated in place (pass B reads psi only
// at the voxel it writes).  Boundary voxels are never written, as in the reference.
#include "fr_common.cuh"
#include "fr_kernels.h"
#include "fr_tma.cuh"

namespace frg {

// det(Mat4f) as written in the reference (include/cuda/cuda_utils.hpp:389-396)
__device__ __forceinline__ float det_ref(const float m[3][3]) {
    float first = ((m[0][0] * m[1][1]) * m[2][2] + (m[1][0] * m[2][1]) * m[0][2]) + (m[2][0] * m[0][1]) * m[1][2];
    float second = ((m[0][2] * m[1][1]) + m[2][0]) * ((m[1][2] * m[2][1]) * m[0][0]) + (m[2][2] * m[0][1]) * m[1][0];
    return first - second;
}

// entropy flux of the (Dv)v diagonal term (vector_fields.cu:376-378): max(c,0)^2 - min(c,0)^2
// + min(n,0)^2 - max(n,0)^2.  The first difference is c |c|: one square is zero, a zero of
// either sign vanishes in the sum, and where c is a NaN the row's other terms are NaN too.
__device__ __forceinline__ float entropy_flux(float c, float n) {
    return (c * fabsf(c) + fminf(n, 0.f) * fminf(n, 0.f)) - fmaxf(n, 0.f) * fmaxf(n, 0.f);
}

// ----------------------------------------------------------------------------------
// fused pass A
//
// A block owns a 32 x 8 column tile and marches z.  Every stencil operand is staged in
// shared-memory ring buffers by 16-byte cp.async one slice ahead of the compute: v with
// a 2-voxel halo over a 5-slice window, and psi_inv, rho and S with a 1-voxel halo over a
// 3-slice window (one ring of five components), so the stencil reads are shared-memory
// loads and the global traffic is one coalesced pass per field.  T o psi_inv and
// L o psi_inv are gathered from the interleaved LT field (eight 16-byte loads per voxel).
// The LT rows of the next slice's cell are prefetched into L2 (the kernel is latency-bound).
// ----------------------------------------------------------------------------------
namespace {
// prefetch distance: slices in flight ahead of the one being computed
constexpr int kAhead = 1;
// Staged rows cover x0 - 4 .. x0 + 35 (stage_offset): column x0 + tx sits at row offset
// tx + kXO.  v has a 2-row y halo, psi_inv a 1-row one.
constexpr int kXO = kStageXO;
constexpr int kVH = 2, kVW = kTileX + 2 * kXO, kVR = kTileY + 2 * kVH, kVS = 5 + kAhead;  // v: halo, width, rows, slots
constexpr int kQH = 1, kQW = kTileX + 2 * kXO, kQR = kTileY + 2 * kQH, kQS = 3 + kAhead;  // psi_inv
constexpr int kVPlane = kVW * kVR, kQPlane = kQW * kQR;
constexpr int kQC = 5;  // the psi_inv ring also holds rho and S (same halo and window)
constexpr int kPassASmemFloats = 3 * kVS * kVPlane + kQC * kQS * kQPlane;  // v x3, psi_inv x3, rho, S
constexpr size_t kPassASmemBytes = sizeof(float) * kPassASmemFloats;

struct PassASmem {
    float* v;  // [3][kVS][kVR][kVW]
    float* q;  // [kQC][kQS][kQR][kQW]: psi_inv x, y, z, rho, S
};

}  // namespace

size_t ref_pass_a_smem_bytes() { return kPassASmemBytes; }

// ----------------------------------------------------------------------------------
// LT = (-(sum of 6 neighbours - 6 psi), T) on the interior; the boundary keeps the
// (0, 0, 0, T) that pack_init_kernel wrote
//
// A block owns a 32 x 8 column tile and marches z.  psi's three components (tile rows
// plus a 1-voxel halo, the psi_inv ring's geometry) and T are staged slice by slice into
// a shared-memory ring by 16-byte cp.async three slices ahead of the compute, so each
// slice of psi is fetched once per tile instead of once per stencil tap (11% faster than
// 7-point reads through L1; one slice ahead or T read per voxel gained nothing).
// ----------------------------------------------------------------------------------
namespace {
constexpr int kLAhead = 3;        // slices in flight ahead of the one computed
constexpr int kLS = 3 + kLAhead;  // ring slots: slices z - 1, z, z + 1 and those in flight
constexpr bool kLStageT = true;   // T staged with psi (else read per voxel)
constexpr int kTPlane = kTileX * kTileY;
}

size_t ref_laplacian_smem_bytes() { return sizeof(float) * kLS * (3 * kQPlane + (kLStageT ? kTPlane : 0)); }

__global__ void __launch_bounds__(256) ref_laplacian_kernel(RefIterArgs a) {
    pdl_wait();
    extern __shared__ __align__(16) float ring[];  // psi [3][kLS][kQR][kQW], then T [kLS][8][32]
    float* tring = ring + 3 * kLS * kQPlane;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int t = blockIdx.x; t < a.ntiles_l; t += gridDim.x) {
        Tile tl;
        Pair P;
        if (!take_tile(a, a.tiles_l, t, kTileY, a.depth_l, tl, P)) continue;  // uniform over the block
        const int X = P.X, Y = P.Y, Z = P.Z, Xp = P.Xp, XYp = P.Xp * P.Y;  // strides of the packed arrays
        const int zs0 = max(tl.w, 1), zs1 = min(tl.w + a.depth_l, Z - 1);
        if (zs0 >= zs1 || tl.y + kTileX <= 1 || tl.z + kTileY <= 1 || tl.y >= X - 1 || tl.z >= Y - 1) continue;
        const long long NT = a.NT;
        const float* Qg[3] = {a.psi + P.off, a.psi + NT + P.off, a.psi + 2 * NT + P.off};
        const float* __restrict__ Tg = a.T + P.off;
        float4* LT = a.LT + P.off;
        const int x = tl.y + tx, y = tl.z + ty;
        const bool active = x >= 1 && x <= X - 2 && y >= 1 && y <= Y - 2;
        const int g = stage_offset<1>(threadIdx.x, Y, Xp, tl.y, tl.z);
        // T: thread e < 64 copies chunk e & 7 of tile row e >> 3 (x0 is a multiple of 32)
        const int tr = (int)threadIdx.x >> 3, tk = (int)threadIdx.x & 7;
        const int gt = (kLStageT && threadIdx.x < 64 && tl.z + tr < Y && tl.y + 4 * tk < Xp)
                           ? Xp * (tl.z + tr) + tl.y + 4 * tk : -1;
        auto stage = [&](int zs, int sl) {  // slice zs of psi's three components (and T) into slot sl
            if (g >= 0) {
                float* dst = ring + sl * kQPlane + 4 * threadIdx.x;
                const int off = g + XYp * zs;
#pragma unroll
                for (int c = 0; c < 3; ++c) cp_async16(dst + c * kLS * kQPlane, Qg[c] + off);
            }
            if (kLStageT && gt >= 0) cp_async16(tring + sl * kTPlane + 4 * threadIdx.x, Tg + gt + XYp * zs);
        };
        __syncthreads();  // the previous tile is done with the ring
        // prologue: slices zs0 - 1 .. zs0 + 1 (one group), then one group per slice ahead
        stage(zs0 - 1, 0);
        stage(zs0, 1);
        stage(zs0 + 1, 2);
        cp_async_commit();
#pragma unroll
        for (int k = 1; k < kLAhead; ++k) {
            if (zs0 + 1 + k <= zs1) stage(zs0 + 1 + k, 2 + k);
            cp_async_commit();
        }
        int sm = 0;  // slot of slice z - 1 (z, z + 1 follow it in the ring)
        const int c0 = (ty + 1) * kQW + tx + kXO;
        for (int z = zs0; z < zs1; ++z) {
            cp_async_wait<kLAhead - 1>();  // slice z + 1 has landed ...
            __syncthreads();               // ... for every thread, and slice z - 2's slot is free
            {
                int sl = sm + 2 + kLAhead;  // the slot of slice z - 2
                sl = sl >= kLS ? sl - kLS : sl;
                if (z + 1 + kLAhead <= zs1) stage(z + 1 + kLAhead, sl);  // reads reach zs1
                cp_async_commit();
            }
            const int s0 = sm + 1 >= kLS ? sm + 1 - kLS : sm + 1;
            const int sp = s0 + 1 >= kLS ? s0 + 1 - kLS : s0 + 1;
            if (active) {
                const int i = x + Xp * y + XYp * z;
                float l[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const float* q = ring + (c * kLS + s0) * kQPlane + c0;
                    const float* qm = ring + (c * kLS + sm) * kQPlane + c0;
                    const float* qp = ring + (c * kLS + sp) * kQPlane + c0;
                    float s = -6.f * q[0];
                    s = s + q[1];
                    s = s + q[-1];
                    s = s + q[kQW];
                    s = s + q[-kQW];
                    s = s + qp[0];
                    s = s + qm[0];
                    l[c] = -1.f * s;
                }
                const float tv = kLStageT ? tring[s0 * kTPlane + ty * kTileX + tx] : __ldg(Tg + i);
                LT[i] = make_float4(l[0], l[1], l[2], tv);
            }
            sm = s0;
        }
        cp_async_wait<0>();
    }
}

// ----------------------------------------------------------------------------------
// The same Laplacian with TMA staging.  Per slice, one thread issues two tensor copies
// into the slot's shared memory -- psi's box of 40 columns x 10 rows x 3 components (the
// tile plus a 1-voxel halo, x0 - 4 .. x0 + 35, y0 - 1 .. y0 + 8; out-of-volume parts read
// as zero and are never used) and T's 32 x 8 box -- completing on the slot's mbarrier; no
// other thread computes an address or issues a copy.  A six-slot ring keeps three slices
// ahead of the one computed (slices z - 1, z, z + 1 are read), and one block barrier per
// slice frees the slot of slice z - 2 for the next copy.  Every wait is bounded (about a
// second); a block that gives up sets the device error word, waits (bounded) for its own
// copies in flight and returns.
// ----------------------------------------------------------------------------------
namespace {
constexpr int kTLAhead = 3;
constexpr int kTLS = 3 + kTLAhead;                      // ring slots
constexpr int kTQW = 40, kTQR = 10, kTQPlane = kTQW * kTQR;  // psi box: row, rows, plane (floats)
constexpr int kTTOff = 1216;                            // T box offset in a slot (floats, 128-byte aligned)
constexpr int kTSlot = kTTOff + kTileX * kTileY;        // slot stride: 1472 floats = 5888 bytes
constexpr unsigned kTLBytes = sizeof(float) * (3 * kTQPlane + kTileX * kTileY);  // copied per slice
static_assert(3 * kTQPlane <= kTTOff && (kTTOff * 4) % 128 == 0 && (kTSlot * 4) % 128 == 0, "slot layout");
}  // namespace

size_t ref_laplacian_tma_smem_bytes() { return sizeof(float) * kTLS * kTSlot + sizeof(uint64_t) * kTLS; }

__global__ void __launch_bounds__(256) ref_laplacian_tma_kernel(RefIterArgs a) {
    pdl_wait();
    extern __shared__ __align__(128) unsigned char lap_raw[];
    float* ring = reinterpret_cast<float*>(lap_raw);
    if (!ring_aligned(ring, a.err)) return;
    uint64_t* full = reinterpret_cast<uint64_t*>(ring + kTLS * kTSlot);
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
    if (tid == 0) {
        for (int k = 0; k < kTLS; ++k) mbar_init(full + k, 1);
        mbar_fence_init();
    }
    __syncthreads();
    // The block's slices go through the ring in one sequence n = 0, 1, 2, ... across its
    // tiles (slot n % kTLS, the (n / kTLS)-th fill of that slot), issued by thread 0 and
    // waited for by every thread in the same order; both walk it with counters instead of
    // dividing: the next slot to issue (islot), the next slot to wait for (wslot), and per
    // slot the parity of its next completion (bit k of wph).
    unsigned issued = 0;  // slices issued so far (thread 0's count)
    int islot = 0, wslot = 0;
    unsigned wph = 0u;
    bool failed = false;
    for (int t = blockIdx.x; t < a.ntiles_l && !failed; t += gridDim.x) {
        Tile tl;
        Pair P;
        if (!take_tile(a, a.tiles_l, t, kTileY, a.depth_l, tl, P)) continue;  // uniform over the block
        const int X = P.X, Y = P.Y, Z = P.Z, Xp = P.Xp, XYp = P.Xp * P.Y;
        const int zs0 = max(tl.w, 1), zs1 = min(tl.w + a.depth_l, Z - 1);
        if (zs0 >= zs1 || tl.y + kTileX <= 1 || tl.z + kTileY <= 1 || tl.y >= X - 1 || tl.z >= Y - 1) continue;
        const CUtensorMap* mpsi = a.tmaps + (long long)tl.x * TM_COUNT + TM_LAP_PSI;
        const CUtensorMap* mT = a.tmaps + (long long)tl.x * TM_COUNT + TM_LAP_T;
        float4* LT = a.LT + P.off;
        const int x = tl.y + tx, y = tl.z + ty;
        const bool active = x >= 1 && x <= X - 2 && y >= 1 && y <= Y - 2;
        const int nsl = zs1 - zs0 + 2;  // slices zs0 - 1 .. zs1, all issued and all waited for
        auto issue = [&](int j) {       // slice zs0 - 1 + j of the tile (thread 0)
            float* dst = ring + islot * kTSlot;
            uint64_t* bar = full + islot;
            mbar_arrive_expect_tx(bar, kTLBytes);
            tma_load_4d(dst, mpsi, tl.y - 4, tl.z - 1, zs0 - 1 + j, 0, bar);
            tma_load_3d(dst + kTTOff, mT, tl.y, tl.z, zs0 - 1 + j, bar);
            islot = islot + 1 == kTLS ? 0 : islot + 1;
            ++issued;
        };
        auto wait_next = [&]() {  // the next slice of the sequence has landed
            const bool ok = mbar_wait_bounded(full + wslot, (wph >> wslot) & 1u);
            wph ^= 1u << wslot;
            wslot = wslot + 1 == kTLS ? 0 : wslot + 1;
            return ok;
        };
        __syncthreads();  // the previous tile is done with the ring
        if (tid == 0) {
            tma_prefetch_map(mpsi);
            tma_prefetch_map(mT);
            for (int j = 0; j < min(nsl, kTLS); ++j) issue(j);
        }
        const int c0 = (ty + 1) * kTQW + tx + 4;
        int sm = 0, s0 = 0, sp = 0;  // slots of slices j0, j0 + 1 and j0 + 2 of the tile
        for (int j0 = 0; j0 + 2 < nsl; ++j0) {
            // slices j0, j0 + 1 and j0 + 2 of the tile are read; j0 + 2 is the newest
            bool ok;
            if (j0 == 0) {
                sm = wslot;
                ok = wait_next();
                s0 = wslot;
                ok = wait_next() && ok;
                sp = wslot;
                ok = wait_next() && ok;
            } else {
                sm = s0;
                s0 = sp;
                sp = wslot;
                ok = wait_next();
            }
            // every thread is past step j0 - 1 (the slot of slice j0 - 1 is free), and the
            // block agrees on whether any wait gave up
            if (__syncthreads_or(!ok)) {
                failed = true;
                break;
            }
            if (tid == 0 && j0 >= 1 && j0 - 1 + kTLS < nsl) issue(j0 - 1 + kTLS);
            if (active) {
                const int z = zs0 + j0;
                const float* qm = ring + sm * kTSlot + c0;
                const float* q0 = ring + s0 * kTSlot;
                const float* qp = ring + sp * kTSlot + c0;
                float l[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const float* q = q0 + c0 + c * kTQPlane;
                    float s = -6.f * q[0];
                    s = s + q[1];
                    s = s + q[-1];
                    s = s + q[kTQW];
                    s = s + q[-kTQW];
                    s = s + qp[c * kTQPlane];
                    s = s + qm[c * kTQPlane];
                    l[c] = -1.f * s;
                }
                const float tv = q0[kTTOff + ty * kTileX + tx];
                LT[x + Xp * y + XYp * z] = make_float4(l[0], l[1], l[2], tv);
            }
        }
    }
    if (failed && tid == 0) {
        // the copies in flight end (bounded) before the block's shared memory goes away
        drain_fills<kTLS>(issued, [&](int k, unsigned parity) { mbar_wait_bounded(full + k, parity); });
        atomicOr(a.err, kErrTmaTimeout);
    }
}

// One voxel of pass A (i = x + Xp (y + Y z), an interior voxel).  vb[k]: this thread's
// column in the staged slice z - 2 + k of v (component c at + c VC); qb[k]: in the staged
// slice z - 1 + k of psi_inv (component c at + c QC), rho (at + QR) and S (at + QS); RW is
// the staged row length.  The arithmetic is the reference's, operation for operation.
template <int VC, int QC, int QR, int QS, int RW>
__device__ __forceinline__ void pass_a_voxel(const RefIterArgs& a, const Pair& P, int X, int Y, int Z, int N, int Xp,
                                             int XYp, int y, int z, int i, bool dv_xy, const float* const vb[5],
                                             const float* const qb[3], const float4* LT,
                                             const float* __restrict__ Tg, const float* const* Vg,
                                             float* rho_n,
                                             float* const* Vn, float* const* Qn) {
    auto V = [&](int k, int c) { return vb[k] + c * VC; };
    auto Q = [&](int k, int c) { return qb[k] + (c < 3 ? c * QC : (c == 3 ? QR : QS)); };
    // T o psi_inv and L o psi_inv, gathered at psi_inv(x)
    const float q[3] = {Q(1, 0)[0], Q(1, 1)[0], Q(1, 2)[0]};
    const Cell32 cl = locate32(X, Y, Z, Xp, q[0], q[1], q[2]);
    const float4 lt = tri_unchecked32_f4(LT, Xp, XYp, N, cl);
    // psi_inv is smooth: the cell of slice z + 1 is about this one plus a slice, so
    // the rows it adds (two slices above the floor corner) are fetched into L2 now
    prefetch_l2(LT + min(cl.base + 2 * XYp, N - 1));
    prefetch_l2(LT + min(cl.base + 2 * XYp + Xp, N - 1));

    // Jacobian of psi_inv, row r = d(psi_inv_r)/d(x, y, z), and its determinant
    float M[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        M[r][0] = (Q(1, r)[1] - Q(1, r)[-1]) * 0.5f;
        M[r][1] = (Q(1, r)[RW] - Q(1, r)[-RW]) * 0.5f;
        M[r][2] = (Q(2, r)[0] - Q(0, r)[0]) * 0.5f;
    }
    const float det = det_ref(M);

    // central-difference gradient of S and the potential gradient
    const float Si = Q(1, 4)[0];
    const float gs[3] = {(Q(1, 4)[1] - Q(1, 4)[-1]) * 0.5f,
                         (Q(1, 4)[RW] - Q(1, 4)[-RW]) * 0.5f,
                         (Q(2, 4)[0] - Q(0, 4)[0]) * 0.5f};

    // velocity and its 6 neighbours (vb[2] is slice z)
    float vc[3], vxm[3], vxp[3], vym[3], vyp[3], vzm[3], vzp[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        vc[c] = V(2, c)[0];
        vxm[c] = V(2, c)[-1];
        vxp[c] = V(2, c)[1];
        vym[c] = V(2, c)[-RW];
        vyp[c] = V(2, c)[RW];
        vzm[c] = V(1, c)[0];
        vzp[c] = V(3, c)[0];
    }
    const float vx = vc[0], vy = vc[1], vz = vc[2];

    // divergence of rho*v (upwind) and the density update
    const float* rb = Q(1, 3);
    const float p = rb[0];
    const float t11 = (vx > 0.f) ? (-vx) * p : (-vx) * rb[1];
    const float t12 = (vxm[0] > 0.f) ? vxm[0] * rb[-1] : vxm[0] * p;
    const float t21 = (vy > 0.f) ? (-vy) * p : (-vy) * rb[RW];
    const float t22 = (vym[1] > 0.f) ? vym[1] * rb[-RW] : vym[1] * p;
    const float t31 = (vz > 0.f) ? (-vz) * p : (-vz) * Q(2, 3)[0];
    const float t32 = (vzm[2] > 0.f) ? vzm[2] * Q(0, 3)[0] : vzm[2] * p;
    const float div = ((((t11 + t12) + t21) + t22) + t31) + t32;
    const float rho_new = p + a.alpha * div;
    rho_n[i] = rho_new;

    // (Dv)v: entropy scheme on the diagonal, upwind off the diagonal
    const float ax1 = entropy_flux(vx, vxp[0]);
    const float ax2 = (vy > 0.f) ? vy * (vx - vym[0]) : vy * (vyp[0] - vx);
    const float ax3 = (vz > 0.f) ? vz * (vx - vzm[0]) : vz * (vzp[0] - vx);
    const float ay1 = (vx > 0.f) ? vx * (vy - vxm[1]) : vx * (vxp[1] - vy);
    const float ay2 = entropy_flux(vy, vyp[1]);
    const float ay3 = (vz > 0.f) ? vz * (vy - vzm[1]) : vz * (vzp[1] - vy);
    const float az1 = (vx > 0.f) ? vx * (vz - vxm[2]) : vx * (vxp[2] - vz);
    const float az2 = (vy > 0.f) ? vy * (vz - vym[2]) : vy * (vyp[2] - vz);
    const float az3 = entropy_flux(vz, vzp[2]);
    const float dvv[3] = {(0.5f * ax1 + ax2) + ax3, (ay1 + 0.5f * ay2) + ay3,
                          (az1 + az2) + 0.5f * az3};

    // negated upwind second differences of v (x in [2,X-3], y in [2,Y-2],
    // z in [2,Z-3]); the y and z forward branches read (+2, -1, 0) as the
    // reference does; y+2 at y = Y-2 reads index i + 2 rows (voxel (x, 0, z+1))
    // from global memory, as the reference's unchecked read does
    float dv[3] = {0.f, 0.f, 0.f};
    if (dv_xy && z >= 2 && z <= Z - 3) {
        const bool y_edge = y + 2 > Y - 1;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float xx = (vx < 0.f) ? (V(2, c)[2] - 2.f * vxp[c]) + vc[c]
                                        : (vc[c] - 2.f * vxm[c]) + V(2, c)[-2];
            const float vyp2 = y_edge ? chain_load(Vg[c] + i + 2 * Xp) : V(2, c)[2 * RW];
            const float yy = (vy < 0.f) ? (vyp2 - 2.f * vym[c]) + vc[c]
                                        : (vc[c] - 2.f * vym[c]) + V(2, c)[-2 * RW];
            const float zz = (vz < 0.f) ? (V(4, c)[0] - 2.f * vzm[c]) + vc[c]
                                        : (vc[c] - 2.f * vzm[c]) + V(0, c)[0];
            dv[c] = -1.f * ((xx + yy) + zz);
        }
    }

    // the potential gradient, from the gathered (L, T) o psi_inv: used as late as the
    // arithmetic allows, so that the work above overlaps the gather's latency
    const float Tq = a.first_iter ? __ldg(Tg + i) : lt.w;
    const float Lq[3] = {lt.x, lt.y, lt.z};
    const float diff = Si - Tq;
    float gU[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) gU[c] = ((diff * gs[c]) + (P.w_reg * Lq[c])) * det;

    // velocity update (solver.cu:198-209) and psi_inv update (solver.cu:275-277)
    const float qd = a.m2 / (fabsf(rho_new) + 1e-5f);
    float vn[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float friction = a.f1 * vc[c];
        const float diffusion = a.tau * dv[c];
        const float potential = qd * gU[c];
        const float acc = ((friction + dvv[c]) - diffusion) + potential;
        vn[c] = vc[c] - a.alpha * acc;
        Vn[c][i] = vn[c];
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const float jv = ((M[r][0] * vn[0]) + (M[r][1] * vn[1])) + (M[r][2] * vn[2]);
        Qn[r][i] = q[r] - a.alpha * jv;
    }
}

__global__ void __launch_bounds__(256, 3) ref_pass_a_kernel(RefIterArgs a) {
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    PassASmem sm;
    sm.v = smem;
    sm.q = sm.v + 3 * kVS * kVPlane;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;

    for (int t = blockIdx.x; t < a.ntiles_a; t += gridDim.x) {
        Tile tl;
        Pair P;
        if (!take_tile(a, a.tiles_a, t, kTileY, a.depth_a, tl, P)) continue;  // uniform over the block
        const int X = P.X, Y = P.Y, Z = P.Z, N = (int)P.N;
        const int Xp = P.Xp, XYp = P.Xp * P.Y;  // strides of the packed arrays
        const int zs0 = max(tl.w, 1), zs1 = min(tl.w + a.depth_a, Z - 1);
        if (zs0 >= zs1 || tl.y + kTileX <= 1 || tl.z + kTileY <= 1 || tl.y >= X - 1 || tl.z >= Y - 1) continue;
        const long long NT = a.NT;
        const float* Vg[3] = {a.v + P.off, a.v + NT + P.off, a.v + 2 * NT + P.off};
        const float* Qg[3] = {a.pinv + P.off, a.pinv + NT + P.off, a.pinv + 2 * NT + P.off};
        const float* Rg = a.rho + P.off;
        const float* __restrict__ Sg = a.S + P.off;
        const float* __restrict__ Tg = a.T + P.off;
        const float4* LT = a.LT + P.off;
        float* rho_n = a.rho_n + P.off;
        float* Vn[3] = {a.v_n + P.off, a.v_n + NT + P.off, a.v_n + 2 * NT + P.off};
        float* Qn[3] = {a.pinv_n + P.off, a.pinv_n + NT + P.off, a.pinv_n + 2 * NT + P.off};
        const int x0 = tl.y, y0 = tl.z;
        const int x = x0 + tx, y = y0 + ty;
        const bool active = x >= 1 && x <= X - 2 && y >= 1 && y <= Y - 2;
        const bool dv_xy = x >= 2 && x <= X - 3 && y >= 2 && y <= Y - 2;

        auto vslot = [](int zs) { return ((zs % kVS) + kVS) % kVS; };
        auto qslot = [](int zs) { return ((zs % kQS) + kQS) % kQS; };
        const int gv = stage_offset<kVH>(threadIdx.x, Y, Xp, x0, y0);
        const int gq = stage_offset<kQH>(threadIdx.x, Y, Xp, x0, y0);
        auto stage_v_at = [&](int zs, int sl) {  // slice zs of v's three components into slot sl
            if (gv < 0 || zs < 0 || zs >= Z) return;
            float* dst = sm.v + sl * kVPlane + 4 * threadIdx.x;
            const int off = gv + XYp * zs;
#pragma unroll
            for (int c = 0; c < 3; ++c) cp_async16(dst + c * kVS * kVPlane, Vg[c] + off);
        };
        auto stage_v = [&](int zs) { stage_v_at(zs, vslot(zs)); };
        auto stage_q_at = [&](int zs, int sl) {  // slice zs of psi_inv's three components, rho and S
            if (gq < 0 || zs < 0 || zs >= Z) return;
            float* dst = sm.q + sl * kQPlane + 4 * threadIdx.x;
            const int off = gq + XYp * zs;
#pragma unroll
            for (int c = 0; c < 3; ++c) cp_async16(dst + c * kQS * kQPlane, Qg[c] + off);
            cp_async16(dst + 3 * kQS * kQPlane, Rg + off);
            cp_async16(dst + 4 * kQS * kQPlane, Sg + off);
        };
        auto stage_q = [&](int zs) { stage_q_at(zs, qslot(zs)); };

        __syncthreads();  // the previous tile is done with the ring buffers
        // prologue: everything slice zs0 needs, then what each of the next kAhead - 1
        // slices adds (one commit group per slice)
        for (int zs = zs0 - 2; zs <= zs0 + 2; ++zs) stage_v(zs);
        for (int zs = zs0 - 1; zs <= zs0 + 1; ++zs) stage_q(zs);
        cp_async_commit();
#pragma unroll
        for (int k = 1; k < kAhead; ++k) {
            if (zs0 + 2 + k <= zs1 + 1) stage_v(zs0 + 2 + k);
            if (zs0 + 1 + k <= zs1) stage_q(zs0 + 1 + k);
            cp_async_commit();
        }

        // this thread's column in the staged slices z - 2 .. z + 2 of v and z - 1 .. z + 1 of
        // psi_inv/rho/S, rotated by one slice per step; with one slice in flight, the slice
        // staged at step z (z + 3 of v, z + 2 of psi_inv) goes into the slot of slice z - 3 /
        // z - 2, and that slot is the newest one read at step z + 1
        static_assert(kAhead == 1 && kVS == 6 && kQS == 4, "the slot rotation below assumes these rings");
        const int vc0 = (ty + kVH) * kVW + tx + kXO;
        const int qc0 = (ty + kQH) * kQW + tx + kXO;
        const float* vb[5];
        const float* qb[3];
#pragma unroll
        for (int k = 0; k < 5; ++k) vb[k] = sm.v + vslot(zs0 - 2 + k) * kVPlane + vc0;
#pragma unroll
        for (int k = 0; k < 3; ++k) qb[k] = sm.q + qslot(zs0 - 1 + k) * kQPlane + qc0;
        int sv = vslot(zs0 - 3), sq = qslot(zs0 - 2);  // the slots step zs0 stages into
        for (int z = zs0; z < zs1; ++z) {
            cp_async_wait<kAhead - 1>();  // slice z's group has landed (the newer ones may not)
            __syncthreads();              // ... for every thread, and slice z - 3 / z - 2 is no longer read
            // prefetch what slice z + 1 adds, into the slots of slices z - 3 (v) and z - 2
            if (z + 3 <= zs1 + 1) stage_v_at(z + 3, sv);  // the last slice reads v up to zs1 + 1
            if (z + 2 <= zs1) stage_q_at(z + 2, sq);      // and psi_inv up to zs1
            cp_async_commit();
            if (active) {
                const int i = x + Xp * y + XYp * z;
                pass_a_voxel<kVS * kVPlane, kQS * kQPlane, 3 * kQS * kQPlane, 4 * kQS * kQPlane, kVW>(
                    a, P, X, Y, Z, N, Xp, XYp, y, z, i, dv_xy, vb, qb, LT, Tg, Vg, rho_n, Vn, Qn);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) vb[k] = vb[k + 1];
            vb[4] = sm.v + sv * kVPlane + vc0;
            qb[0] = qb[1];
            qb[1] = qb[2];
            qb[2] = sm.q + sq * kQPlane + qc0;
            sv = sv + 1 == kVS ? 0 : sv + 1;
            sq = (sq + 1) & 3;
        }
        cp_async_wait<0>();
    }
}

// ----------------------------------------------------------------------------------
// Pass A with TMA staging.  Fill n of a tile holds v's slice zs0 - 2 + n (a box of 40 columns x 12
// rows x 3 components, 2-voxel halo) in a slot of the v ring and, from n = 2 on, slice zs0 - 3 + n
// of psi_inv (40 x 10 x 3), rho and S (40 x 10) in a slot of the q ring, all copied by one thread
// and completing on one barrier.  Slice zs0 + j reads v's fills j .. j + 4 and the q ring's
// j + 2 .. j + 4; one block barrier per slice frees the slots of slices z - 3 / z - 2 for the next
// fill.  Out-of-volume parts of a box read as zero and are never used (the stencils
// that reach them are masked, as in the cp.async kernel).  Waits are bounded as in
// ref_laplacian_tma_kernel.  The voxel arithmetic is pass_a_voxel, shared with
// ref_pass_a_kernel.
//
// Bound by issue slots (three blocks of 80 registers, 600 instructions per voxel of which 250 are
// the reference's arithmetic) and by the LT gather's latency.  163 us on the 182x218x182 pair
// (76 bytes per voxel, 82 us at the copy bandwidth) and 384 us on four 160x192x160 pairs, 180 and
// 431 us with cp.async staging, whose threads each form eight staging addresses per slice.
// With a barrier per field, ring slots by division and generic addressing this kernel took
// 193 us; per-slot empty barriers in place of the block barrier 220 us (the extra state
// spills); the LT rows prefetched by one tensor copy instead of per thread 165 us, not
// prefetched 170 us; rho and S three slices ahead prefetched as well 167 us.
// ----------------------------------------------------------------------------------
namespace {
constexpr int kPVS = 6, kPQS = 4;                 // ring slots: v (5 + 1), psi_inv/rho/S (3 + 1)
constexpr int kPW = 40;                           // staged row: columns x0 - 4 .. x0 + 35
constexpr int kPVPlane = kPW * 12, kPVSlot = 3 * kPVPlane;  // 1440 floats = 5760 bytes
constexpr int kPQPlane = kPW * 10;
constexpr int kPQR = 1216, kPQSo = 1632, kPQSlot = 2048;    // rho, S offsets; slot (floats)
constexpr unsigned kPVBytes = sizeof(float) * kPVSlot;
constexpr unsigned kPQBytes = sizeof(float) * (3 * kPQPlane + 2 * kPQPlane);
static_assert((kPVSlot * 4) % 128 == 0 && (kPQR * 4) % 128 == 0 && (kPQSo * 4) % 128 == 0 &&
                  3 * kPQPlane <= kPQR && kPQR + kPQPlane <= kPQSo && kPQSo + kPQPlane <= kPQSlot,
              "slot layout");
}  // namespace

size_t ref_pass_a_tma_smem_bytes() {
    return sizeof(float) * (kPVS * kPVSlot + kPQS * kPQSlot) + sizeof(uint64_t) * kPVS;
}

__global__ void __launch_bounds__(256, 3) ref_pass_a_tma_kernel(RefIterArgs a) {
    pdl_wait();
    extern __shared__ __align__(128) unsigned char pa_raw[];
    float* vring = reinterpret_cast<float*>(pa_raw);
    if (!ring_aligned(vring, a.err)) return;
    float* qring = vring + kPVS * kPVSlot;
    uint64_t* full = reinterpret_cast<uint64_t*>(qring + kPQS * kPQSlot);
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
    if (tid == 0) {
        for (int k = 0; k < kPVS; ++k) mbar_init(full + k, 1);
        mbar_fence_init();
    }
    __syncthreads();
    // fills go through the rings in order, across the block's tiles: the next slots to fill
    // (thread 0) and to read, and per slot the parity of its next completion
    int fv = 0, fq = 0, rv = 0, rq = 0;
    unsigned phase = 0u;
    unsigned issued = 0;  // fills so far (thread 0)
    bool failed = false;
    for (int t = blockIdx.x; t < a.ntiles_a && !failed; t += gridDim.x) {
        Tile tl;
        Pair P;
        if (!take_tile(a, a.tiles_a, t, kTileY, a.depth_a, tl, P)) continue;  // uniform over the block
        const int X = P.X, Y = P.Y, Z = P.Z, N = (int)P.N;
        const int Xp = P.Xp, XYp = P.Xp * P.Y;
        const int zs0 = max(tl.w, 1), zs1 = min(tl.w + a.depth_a, Z - 1);
        if (zs0 >= zs1 || tl.y + kTileX <= 1 || tl.z + kTileY <= 1 || tl.y >= X - 1 || tl.z >= Y - 1) continue;
        const long long NT = a.NT;
        const float* Vg[3] = {a.v + P.off, a.v + NT + P.off, a.v + 2 * NT + P.off};
        const float* __restrict__ Tg = a.T + P.off;
        const float4* LT = a.LT + P.off;
        float* rho_n = a.rho_n + P.off;
        float* Vn[3] = {a.v_n + P.off, a.v_n + NT + P.off, a.v_n + 2 * NT + P.off};
        float* Qn[3] = {a.pinv_n + P.off, a.pinv_n + NT + P.off, a.pinv_n + 2 * NT + P.off};
        const int x = tl.y + tx, y = tl.z + ty;
        const bool active = x >= 1 && x <= X - 2 && y >= 1 && y <= Y - 2;
        const bool dv_xy = x >= 2 && x <= X - 3 && y >= 2 && y <= Y - 2;
        const int nfill = zs1 - zs0 + 4;
        auto issue = [&](int n) {  // thread 0
            const CUtensorMap* maps = a.tmaps + (long long)tl.x * TM_COUNT;
            const int src = (a.iter - 1) & 1, zv = zs0 - 2 + n;  // src: the buffers this iteration reads
            uint64_t* bar = full + fv;
            mbar_arrive_expect_tx(bar, n >= 2 ? kPVBytes + kPQBytes : kPVBytes);
            tma_load_4d(vring + fv * kPVSlot, maps + TM_PA_V0 + src, tl.y - 4, tl.z - 2, zv, 0, bar);
            if (n >= 2) {
                float* dst = qring + fq * kPQSlot;
                tma_load_4d(dst, maps + TM_PA_Q0 + src, tl.y - 4, tl.z - 1, zv - 1, 0, bar);
                tma_load_3d(dst + kPQR, maps + TM_PA_R0 + src, tl.y - 4, tl.z - 1, zv - 1, bar);
                tma_load_3d(dst + kPQSo, maps + TM_PA_S, tl.y - 4, tl.z - 1, zv - 1, bar);
                fq = fq + 1 == kPQS ? 0 : fq + 1;
            }
            fv = fv + 1 == kPVS ? 0 : fv + 1;
            ++issued;
        };
        __syncthreads();  // the previous tile is done with the rings
        if (tid == 0)
            for (int n = 0; n < min(nfill, kPVS); ++n) issue(n);

        const int vc0 = (ty + 2) * kPW + tx + 4, qc0 = (ty + 1) * kPW + tx + 4;
        const float* vb[5];  // this thread's column in the slices read, rotated by one per step
        const float* qb[3];
        bool ok = true;
        auto land = [&]() {  // waits for the next fill
            ok = mbar_wait_bounded(full + rv, (phase >> rv) & 1u) && ok;
            phase ^= 1u << rv;
        };
        auto next_v = [&](int k) {
            vb[k] = vring + rv * kPVSlot + vc0;
            rv = rv + 1 == kPVS ? 0 : rv + 1;
        };
        auto next_q = [&](int k) {
            qb[k] = qring + rq * kPQSlot + qc0;
            rq = (rq + 1) & (kPQS - 1);
        };
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            land();
            next_v(k + 1);
            if (k >= 2) next_q(k - 1);
        }
        for (int z = zs0; z < zs1; ++z) {
            land();
            // every thread is past slice z - 1, whose oldest fill is free, and the block agrees on
            // whether any wait gave up
            if (__syncthreads_or(!ok)) {
                failed = true;
                break;
            }
            if (tid == 0 && z > zs0 && z - zs0 - 1 + kPVS < nfill) issue(z - zs0 - 1 + kPVS);
#pragma unroll
            for (int k = 0; k < 4; ++k) vb[k] = vb[k + 1];
            qb[0] = qb[1];
            qb[1] = qb[2];
            next_v(4);
            next_q(2);
            if (active) {
                const int i = x + Xp * y + XYp * z;
                pass_a_voxel<kPVPlane, kPQPlane, kPQR, kPQSo, kPW>(a, P, X, Y, Z, N, Xp, XYp, y, z, i, dv_xy, vb, qb,
                                                                   LT, Tg, Vg, rho_n, Vn, Qn);
            }
        }
    }
    if (failed && tid == 0) {
        // the copies in flight end (bounded) before the block's shared memory goes; every fill is one of
        // the v ring, whose barriers the q ring's copies complete on too
        drain_fills<kPVS>(issued, [&](int k, unsigned parity) { mbar_wait_bounded(full + k, parity); });
        atomicOr(a.err, kErrTmaTimeout);
    }
}

// ----------------------------------------------------------------------------------
// pass B: psi += alpha * v o psi, max update norm, convergence
//
// One thread per column of a 32 x 4 tile (128-thread blocks): the kernel waits on its
// gathers, and 9 blocks of 128 threads at 56 registers hold 36 warps per SM where 256-thread
// blocks held 32 (at 64 registers; at 48, for 5 blocks of 256, it spills).
// ----------------------------------------------------------------------------------
__global__ void __launch_bounds__(kPassBThreads, 9) ref_pass_b_kernel(RefIterArgs a) {
    pdl_wait();
    __shared__ unsigned long long red[32];
    const int tid = threadIdx.x;
    for (int t = blockIdx.x; t < a.ntiles_b; t += gridDim.x) {
        Tile tl;
        Pair P;
        if (!take_tile(a, a.tiles_b, t, kPassBTileY, a.depth_b, tl, P)) continue;  // uniform over the block
        const int x = tl.y + (int)(threadIdx.x & 31), y = tl.z + (int)(threadIdx.x >> 5);
        unsigned long long best = 0ull;
        if (x >= 1 && x <= P.X - 2 && y >= 1 && y <= P.Y - 2) {
            const int X = P.X, Y = P.Y, Z = P.Z, Xp = P.Xp, XYp = P.Xp * P.Y;
            const long long NT = a.NT;
            // the velocity pass A just wrote
            const float* V[3] = {a.v_n + P.off, a.v_n + NT + P.off, a.v_n + 2 * NT + P.off};
            float* Q[3] = {a.psi + P.off, a.psi + NT + P.off, a.psi + 2 * NT + P.off};
            const int z0 = max(tl.w, 1), z1 = min(tl.w + a.depth_b, P.Z - 1);
            int i = x + Xp * y + XYp * z0;
            // psi of the next slice is loaded while this slice's gathers are in flight
            float nx = 0.f, ny = 0.f, nz = 0.f;
            if (z0 < z1) {
                nx = Q[0][i];
                ny = Q[1][i];
                nz = Q[2][i];
            }
            for (int z = z0; z < z1; ++z, i += XYp) {
                const float px = nx, py = ny, pz = nz;
                if (z + 1 < z1) {
                    nx = Q[0][i + XYp];
                    ny = Q[1][i + XYp];
                    nz = Q[2][i + XYp];
                }
                const Cell32 cl = locate32(X, Y, Z, Xp, px, py, pz);
                float vp[3];
                tri_checked32_3(V[0], V[1], V[2], X, Y, Z, Xp, XYp, cl, vp);
                const float ux = a.alpha * vp[0];
                const float uy = a.alpha * vp[1];
                const float uz = a.alpha * vp[2];
                Q[0][i] = px + ux;
                Q[1][i] = py + uy;
                Q[2][i] = pz + uz;
                const float nrm = norm3_rd(ux, uy, uz);
                if (nrm == nrm) {  // NaN norms never win, as in the reference's '>' test
                    const unsigned long long k = norm_key(nrm, i);
                    best = k > best ? k : best;
                }
            }
        }
        const unsigned long long bm = block_max_u64(best, red);
        if (tid == 0) note_max(a, tl.x, bm);
    }

    record_and_test(a);
}

}  // namespace frg
