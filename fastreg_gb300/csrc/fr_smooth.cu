// fr_smooth.cu -- the sobolev solver's separable Gaussian (x, y, z) fused with the momentum
// update m = damping * m - step * gs, one launch over the cohort (two for small volumes and wide
// filters: sob_smooth_z_kernel).
//
// A warp owns one component of a 32-column x TY-row tile and marches z; a block is the three
// components of a tile, and its warps never wait on one another.  Per slice the warp stages
// its own box of g (the rows plus an R halo, columns x0 - HX .. x0 + 31 + HX with HX = R
// rounded up to 4) in a ring of shared-memory slots, by one TMA tensor copy or by 16-byte
// cp.async per lane, and then keeps everything else in registers: each lane filters its own
// column of every staged row along x, filters the results along y from a window of 2R + 2
// rows, and feeds each row's value into the z filter of that row.
//
//   - The z filter is kept as 2R partial sums per row instead of the last 2R + 1 values: the
//     chain of output slice z is fma(w_2R, y_z+R, ... fma(w_0, y_z-R, 0)), so slice k's value
//     extends the 2R chains in flight by one tap each and starts a new one, and the shift to
//     the next chain position is the destination register of the fma.  (A ring of values needs
//     2R register moves per row and slice.)
//   - Rows are taken in pairs, so that the taps of all three axes run as packed FP32 pairs
//     (per lane the same fused multiply-adds as the scalar chain).
//   - No block barrier and no second shared-memory array: exchanging the x pass through shared
//     memory between two barriers per slice took 80 million warp instructions on the
//     182x218x182 pair at radius 3, this takes 36 million: 67 us instead of 94 us (36 bytes per
//     voxel, 39 us at the copy bandwidth), 274 instead of 403 us on eight pairs of 160x192x160,
//     214 instead of 231 us at radius 7.
//
// What bounds it now: 12 warps per SM (164 registers: the chains of 16 rows) that wait on the
// fixed latency of dependent multiply-adds (issue slots 50% used), with the shared-memory
// loads of the x filter (one per tap and row, 36 us of LSU time) and HBM (39 us) close behind.
//
// The taps of every output are taken in the order -R..R for each axis, acc = fma(w, v, acc)
// from 0, with the replicate boundary: slices outside the volume are the clamped slice, and
// on tiles at an x or y edge the staged box is completed in shared memory (fix_edges).
#include "fr_common.cuh"
#include "fr_kernels.h"
#include "fr_sob.h"
#include "fr_tma.cuh"

namespace frg {
namespace {

constexpr int kILP = 2;  // row pairs whose chains are interleaved: radius 2 takes 56 us instead of 62, others the same

template <int R, int TY>
struct SmoothGeom {
    static constexpr int K = 2 * R + 1;
    static constexpr int HX = (R + 3) / 4 * 4, WS = kTileX + 2 * HX, H = TY + 2 * R;
    static constexpr int BOX = H * WS;                // floats of a staged slice
    static constexpr int SLOT = (BOX + 31) / 32 * 32;  // slot stride: 128-byte multiple
    // slots per warp: as many (up to 4) as keep the block's shared memory within 48 KB
    static constexpr int NS = 3 * (4 * SLOT * 4 + 32) <= 48 * 1024 ? 4 : 3;
    static_assert(TY % 2 == 0, "rows are taken in pairs");
    static_assert(3 * (NS * SLOT * 4 + 8 * NS) <= 48 * 1024, "static shared memory");
};

// The replicate boundary of a staged slice (whole warp): the R columns beyond an x edge take
// the edge column, then, where rows outside the volume were not staged from the clamped row
// (TMA fills them with zeros), the R rows beyond a y edge take the edge row.  Only columns
// and rows that outputs inside the volume read are written; what else the box holds reaches
// outputs that are never stored.
template <int R, bool TMA, int TY>
__device__ __forceinline__ void fix_edges(float* box, int x0, int y0, int X, int Y) {
    using G = SmoothGeom<R, TY>;
    if constexpr (R > 0) {
        const int lane = threadIdx.x & 31;
        if (x0 == 0) {  // x0 is a multiple of 32, so only the first tile has x = 0 in its halo
            for (int w = lane; w < G::H * R; w += 32) {
                float* row = box + (w / R) * G::WS;
                row[G::HX - R + w % R] = row[G::HX];
            }
        }
        const int hi = X - 1 - x0 + G::HX;  // staged column of x = X - 1
        if (hi + 1 < G::WS) {
            for (int w = lane; w < G::H * R; w += 32) {
                float* row = box + (w / R) * G::WS;
                const int c = hi + 1 + w % R;
                if (c < G::WS) row[c] = row[hi];
            }
        }
        if constexpr (TMA) {
            const int top = R - y0, bottom = Y - 1 - (y0 - R);  // staged rows of y = 0 and y = Y - 1
            __syncwarp();
            if (top > 0)
                for (int w = lane; w < top * G::WS; w += 32) box[w] = box[top * G::WS + w % G::WS];
            if (bottom + 1 < G::H) {
                const int end = min(bottom + R, G::H - 1);
                for (int w = lane; w < (end - bottom) * G::WS; w += 32)
                    box[(bottom + 1) * G::WS + w] = box[bottom * G::WS + w % G::WS];
            }
            // these generic-proxy writes come before the tensor copy that refills the slot
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncwarp();
    }
}

// The transpose, with cp.async staging.  Inside the volume it is the same filter
// (the taps are symmetric) of g continued by zeros, since a tap that the forward pass clamps
// lands on the first or last position of its axis; those positions take, from the position s
// beside them, all taps up to tap R - s instead of that tap alone: fold[s] more.
// MODE: what the filter feeds.
enum SmoothMode {
    kInPlace,    // the momentum, updated in place (m_n is m; a second pointer costs the TMA kernel 4%)
    kOutOfPlace, // the momentum, read from m and written to m_n
    kTranspose,  // m_n = G^T g
    kPlanes,     // mid = g filtered along x and y only (sob_smooth_z_kernel does the rest)
    kPlanesTranspose
};
constexpr int kPlaneSlots = 1;  // the plane forms take one slice per tile
template <int R, bool TMA, int TY, SmoothMode MODE>
__global__ void __launch_bounds__(kSmoothThreads) sob_smooth3_kernel(SobIterArgs a) {
    pdl_wait();
    using G = SmoothGeom<R, TY>;
    constexpr bool ADJ = MODE == kTranspose || MODE == kPlanesTranspose;
    constexpr bool kPlane = MODE == kPlanes || MODE == kPlanesTranspose, kMomentum = !ADJ && !kPlane;
    constexpr int RZ = kPlane ? 0 : R;  // slices read beyond a tile's ends
    constexpr int K = G::K, WS = G::WS, NS = kPlane ? kPlaneSlots : G::NS, NP = TY / 2;
    __shared__ __align__(128) float rings[3][NS][G::SLOT];
    __shared__ __align__(8) uint64_t bars[3][NS];
    const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;  // this warp's component
    float(*ring)[G::SLOT] = rings[c];
    uint64_t* full = bars[c];
    if (TMA) {
        if (lane == 0) {
            for (int k = 0; k < NS; ++k) mbar_init(full + k, 1);
            mbar_fence_init();
        }
        __syncwarp();
    }
    unsigned phase = 0u;  // TMA: parity of each slot's next completion
    int issue_slot = 0, slot = 0, pending = 0;  // slots filled and read in order; fills not yet read
    bool failed = false;

    for (int t = blockIdx.x; t < a.ntiles_s && !failed; t += gridDim.x) {
        // The kernels of large cohorts read the table even for a single pair: with the tile and
        // pair chosen between table and arguments the tall TMA kernel takes 75 instead of 66 us.  Neither
        // registers (166, 164) nor blocks per SM (4, 4) tell the two apart; the compiler orders the march differently,
        // so another compiler may need another choice.
        constexpr bool kTable = MODE == kInPlace && (TMA || TY != sob_smooth_tile_y(R, false));
        Tile tl;
        Pair P;
        if (kTable) {
            tl = a.tiles_s[t];
            if (a.check_stop && a.stop[tl.x]) continue;  // uniform over the block
            P = a.pairs[tl.x];
        } else if (!take_tile(a, a.tiles_s, t, TY, a.depth_s, tl, P)) {
            continue;
        }
        const int X = P.X, Y = P.Y, Z = P.Z, Xp = P.Xp, XY = P.Xp * P.Y;
        const int x0 = tl.y, y0 = tl.z, zt0 = tl.w, zt1 = min(tl.w + a.depth_s, Z);
        const int nsl = (zt1 - zt0) + 2 * RZ;
        const bool edge = x0 == 0 || x0 + kTileX - 1 + R > X - 1 || y0 == 0 || y0 + TY - 1 + R > Y - 1;
        const float* gc = a.g + c * a.NT + P.off;
        const CUtensorMap* mg = a.tmaps + (long long)tl.x * TM_COUNT + (TY == sob_smooth_tile_y(R, false) ? TM_SOB_G : TM_SOB_G_TALL);

        // cp.async: chunk f = lane + 32 j of the box is (row f / (WS / 4), chunk f % (WS / 4));
        // its offset inside a slice is fixed for the tile (-1: outside the padded row)
        constexpr int NF = G::H * (WS / 4), NJ = TMA ? 1 : (NF + 31) / 32;
        int goff[NJ];
        if (!TMA) {
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const int f = lane + 32 * j, r = f / (WS / 4), x = x0 - G::HX + 4 * (f % (WS / 4));
                const int yr = y0 - R + r;
                const bool in = f < NF && x >= 0 && x < Xp && (!ADJ || (yr >= 0 && yr < Y));
                goff[j] = in ? Xp * min(max(yr, 0), Y - 1) + x : -1;
            }
        }
        auto issue = [&](int k) {  // slice k of the tile (z = zt0 - RZ + k, clamped) into the next slot
            const int z = min(max(zt0 - RZ + k, 0), Z - 1);
            if (TMA) {
                if (lane == 0) {
                    mbar_arrive_expect_tx(full + issue_slot, sizeof(float) * G::BOX);
                    tma_load_4d(ring[issue_slot], mg, x0 - G::HX, y0 - R, z, c, full + issue_slot);
                }
            } else {
                float* dst = ring[issue_slot] + 4 * lane;
                const float* src = gc + (long long)XY * z;
#pragma unroll
                for (int j = 0; j < NJ; ++j)
                    if (ADJ) {  // zeros outside the volume
                        const bool in = goff[j] >= 0 && zt0 - RZ + k >= 0 && zt0 - RZ + k < Z;
                        if (lane + 32 * j < NF) cp_async16_or_zero(dst + 128 * j, in ? src + goff[j] : src, in);
                    } else if (goff[j] >= 0) {
                        cp_async16(dst + 128 * j, src + goff[j]);
                    }
            }
            issue_slot = issue_slot + 1 == NS ? 0 : issue_slot + 1;
            ++pending;
        };
        for (int k = 0; k < NS; ++k) {
            if (k < nsl) issue(k);
            if (!TMA) cp_async_commit();
        }
        float2 part[NP][RZ > 0 ? 2 * RZ : 1];  // the z chains in flight of each row pair
#pragma unroll
        for (int p = 0; p < NP; ++p)
#pragma unroll
            for (int j = 0; j < (RZ > 0 ? 2 * RZ : 1); ++j) part[p][j] = make_float2(0.f, 0.f);
        const int x = x0 + lane, rows = x < X ? min(Y - y0, TY) : 0;  // rows that this lane stores
        const long long m0 = c * a.NT + P.off + (x + Xp * y0) + (long long)XY * (zt0 - 2 * RZ);
        float* mn = (kPlane ? a.mid : a.m_n) + m0;
        const float* ms = MODE == kOutOfPlace ? a.m + m0 : nullptr;
        for (int k = 0; k < nsl; ++k, mn += XY, ms += MODE == kOutOfPlace ? XY : 0) {
            const float* m = MODE == kOutOfPlace ? ms : mn;
            const bool store = k >= 2 * RZ;  // slice zt0 + k - 2RZ is complete with this one
            float mo[TY];
            if (store && kMomentum)
#pragma unroll
                for (int r = 0; r < TY; ++r)
                    if (r < rows) mo[r] = m[Xp * r];
            if (TMA) {
                const bool ok = mbar_wait_bounded(full + slot, (phase >> slot) & 1u);
                if (!__all_sync(0xffffffffu, ok)) {
                    failed = true;
                    break;
                }
                phase ^= 1u << slot;
                --pending;
            } else {
                cp_async_wait<NS - 1>();
                __syncwarp();
            }
            float* box = ring[slot];
            if (edge && !ADJ) fix_edges<R, TMA, TY>(box, x0, y0, X, Y);
            const float* col = box + lane + G::HX - R;
            float2 ev[G::H / 2], od[G::H / 2];  // x-filtered rows (2 r, 2 r + 1) and (2 r - 1, 2 r)
            // row pairs in groups of kILP, whose chains are independent
#pragma unroll
            for (int r0 = 0; r0 < G::H / 2; r0 += kILP) {
#pragma unroll
                for (int q = 0; q < K; ++q)
#pragma unroll
                    for (int rp = r0; rp < r0 + kILP && rp < G::H / 2; ++rp)
                        ev[rp] = __ffma2_rn(make_float2(a.taps[q], a.taps[q]),
                                            make_float2(col[2 * rp * WS + q], col[(2 * rp + 1) * WS + q]),
                                            q ? ev[rp] : make_float2(0.f, 0.f));
                if (ADJ && edge && (x == 0 || x == X - 1)) {  // the ends of the x axis
                    const int step = x == 0 ? 1 : -1;
#pragma unroll
                    for (int rp = r0; rp < r0 + kILP && rp < G::H / 2; ++rp)
#pragma unroll
                        for (int d = 0; d < R; ++d) {
                            ev[rp].x = fmaf(a.fold[d], col[2 * rp * WS + R + step * d], ev[rp].x);
                            ev[rp].y = fmaf(a.fold[d], col[(2 * rp + 1) * WS + R + step * d], ev[rp].y);
                        }
                }
#pragma unroll
                for (int rp = r0; rp < r0 + kILP && rp < G::H / 2; ++rp)
                    if (rp > 0) od[rp] = make_float2(ev[rp - 1].y, ev[rp].x);
                // output rows 2 p, 2 p + 1 of p = rp - R: staged rows 2 p .. 2 p + 1 + 2 R
                float2 v[kILP], o[kILP];
#pragma unroll
                for (int q = 0; q < K; ++q)
#pragma unroll
                    for (int rp = r0; rp < r0 + kILP && rp < G::H / 2; ++rp) {
                        if (rp < R) continue;
                        const int p = rp - R;
                        v[rp - r0] = __ffma2_rn(make_float2(a.taps[q], a.taps[q]), q & 1 ? od[p + (q + 1) / 2] : ev[p + q / 2],
                                                q ? v[rp - r0] : make_float2(0.f, 0.f));
                    }
                if (ADJ && edge)  // the ends of the y axis
#pragma unroll
                    for (int rp = r0; rp < r0 + kILP && rp < G::H / 2; ++rp) {
                        if (rp < R) continue;
                        auto row = [&](int i) { return i & 1 ? ev[i / 2].y : ev[i / 2].x; };
                        const int i0 = 2 * (rp - R), i1 = i0 + 1;  // output rows; their own staged rows are i + R
#pragma unroll
                        for (int d = 0; d < R; ++d) {
                            if (y0 + i0 == 0) v[rp - r0].x = fmaf(a.fold[d], row(i0 + R + d), v[rp - r0].x);
                            if (y0 + i0 == Y - 1) v[rp - r0].x = fmaf(a.fold[d], row(i0 + R - d), v[rp - r0].x);
                            if (y0 + i1 == Y - 1) v[rp - r0].y = fmaf(a.fold[d], row(i1 + R - d), v[rp - r0].y);
                        }
                    }
#pragma unroll
                for (int j = 2 * RZ; j >= 0; --j)
#pragma unroll
                    for (int rp = r0; rp < r0 + kILP && rp < G::H / 2; ++rp) {
                        if (rp < R) continue;
                        const int p = rp - R;
                        if (kPlane) {
                            o[rp - r0] = v[rp - r0];
                            continue;
                        }
                        const float2 n = __ffma2_rn(make_float2(a.taps[j], a.taps[j]), v[rp - r0],
                                                    j > 0 ? part[p][j > 0 ? j - 1 : 0] : make_float2(0.f, 0.f));
                        if (j == 2 * RZ)
                            o[rp - r0] = n;
                        else
                            part[p][j] = n;
                    }
                if (ADJ && !kPlane) {  // the ends of the z axis: this slice's extra share of output slices 0 and Z - 1
                    const int zc = zt0 - R + k;
#pragma unroll
                    for (int d = 0; d < R; ++d)
#pragma unroll
                        for (int rp = r0; rp < r0 + kILP && rp < G::H / 2; ++rp) {
                            if (rp < R) continue;
                            const float2 w = make_float2(a.fold[d], a.fold[d]);
                            if (zc == d) part[rp - R][R + d] = __ffma2_rn(w, v[rp - r0], part[rp - R][R + d]);
                            if (zc == Z - 1 - d) part[rp - R][R - d] = __ffma2_rn(w, v[rp - r0], part[rp - R][R - d]);
                        }
                }
                if (store)
#pragma unroll
                    for (int rp = r0; rp < r0 + kILP && rp < G::H / 2; ++rp) {
                        if (rp < R) continue;
                        const int p = rp - R;
                        if (2 * p < rows)
                            mn[Xp * (2 * p)] = !kMomentum ? o[rp - r0].x : a.damping * mo[2 * p] - a.step * o[rp - r0].x;
                        if (2 * p + 1 < rows)
                            mn[Xp * (2 * p + 1)] =
                                !kMomentum ? o[rp - r0].y : a.damping * mo[2 * p + 1] - a.step * o[rp - r0].y;
                    }
            }
            __syncwarp();  // every lane has read the slot
            if (k + NS < nsl) issue(k + NS);
            if (!TMA) cp_async_commit();
            slot = slot + 1 == NS ? 0 : slot + 1;
        }
    }
    if (TMA && failed && lane == 0) {
        // the copies that this warp has in flight end (bounded) before its shared memory goes
        for (; pending > 0; --pending) {
            mbar_wait_bounded(full + slot, (phase >> slot) & 1u);
            slot = slot + 1 == NS ? 0 : slot + 1;
        }
        atomicOr(a.err, kErrTmaTimeout);
    }
}

// The smoothing in two launches: the plane forms above filter every slice along x and y into
// `mid`, this kernel filters mid along z and feeds the momentum (or, transposed, m_n), tap for
// tap in the same order, so the bits are those of the one launch.  No slice is filtered along x
// and y twice (a march of d slices filters d + 2 R), no z chains are held across a slice (the plane
// kernel's 16 rows take 64 registers instead of 168), and every slice is a tile of its own, which
// is what small volumes and wide filters lack; large volumes at small radii pay 24 bytes per voxel
// more of traffic instead.  20 unrolled iterations: radius 3, 64^3 1.33 -> 1.10 ms, 96^3 2.46 -> 2.33,
// 128^3 4.83 -> 4.85; radius 5, 91x109x91 3.76 -> 2.98; radius 7, 128^3 9.04 -> 6.30; radius 1, 64^3
// 0.95 -> 1.03.  A thread takes kZBatch slices' loads together; bound by their latency.
constexpr int kZBatch = 4;
// In place at radius 6 the compiler settles on 40 registers and a load at a time (35 us on 41x195x75); held to five
// blocks per SM it takes 48 and the batch (31 us), as it does by itself at radius 7.
template <int R, SmoothMode MODE>
__global__ void __launch_bounds__(256, R == 6 && MODE == kInPlace ? 5 : 0) sob_smooth_z_kernel(SobIterArgs a) {
    pdl_wait();
    constexpr bool ADJ = MODE == kTranspose;
    constexpr int U = kZBatch;
    for (int t = blockIdx.x; t < 3 * a.ntiles_z; t += gridDim.x) {
        const int c = t % 3;
        Tile tl;
        Pair P;
        if (!take_tile(a, a.tiles_z, t / 3, kTileY, a.depth_z, tl, P)) continue;
        const int X = P.X, Y = P.Y, Z = P.Z, XY = P.Xp * P.Y;
        const int x = tl.y + (threadIdx.x & 31), y = tl.z + (threadIdx.x >> 5);
        if (x >= X || y >= Y) continue;
        const int zt0 = tl.w, zt1 = min(zt0 + a.depth_z, Z), nsl = zt1 - zt0 + 2 * R;
        const long long at = c * a.NT + P.off + x + P.Xp * y;
        const float* g = a.mid + at;
        const float* m = (MODE == kOutOfPlace ? a.m : a.m_n) + at;
        float* mn = a.m_n + at;
        float part[R > 0 ? 2 * R : 1];
#pragma unroll
        for (int j = 0; j < (R > 0 ? 2 * R : 1); ++j) part[j] = 0.f;
        for (int k0 = 0; k0 < nsl; k0 += U) {
            float v[U], mo[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = k0 + u, z = zt0 - R + k;
                const bool in = k < nsl && (!ADJ || (z >= 0 && z < Z));
                v[u] = in ? chain_load(g + XY * min(max(z, 0), Z - 1)) : 0.f;
                mo[u] = !ADJ && k >= 2 * R && k < nsl ? m[XY * (z - R)] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = k0 + u, z = zt0 - R + k;
                float o = 0.f;
#pragma unroll
                for (int j = 2 * R; j >= 0; --j) {
                    const float n = fmaf(a.taps[j], v[u], j > 0 ? part[j > 0 ? j - 1 : 0] : 0.f);
                    if (j == 2 * R)
                        o = n;
                    else
                        part[j] = n;
                }
                if (ADJ)
#pragma unroll
                    for (int d = 0; d < R; ++d) {
                        if (z == d) part[R + d] = fmaf(a.fold[d], v[u], part[R + d]);
                        if (z == Z - 1 - d) part[R - d] = fmaf(a.fold[d], v[u], part[R - d]);
                    }
                if (k >= 2 * R && k < nsl) mn[XY * (z - R)] = ADJ ? o : a.damping * mo[u] - a.step * o;
            }
        }
    }
}

template <int R>
const void* smooth_fn(int tma, bool tall) {
    constexpr int kShort = sob_smooth_tile_y(R, false), kTall = sob_smooth_tile_y(R, true);
    if (tall)
        return tma ? (const void*)sob_smooth3_kernel<R, true, kTall, kInPlace>
                   : (const void*)sob_smooth3_kernel<R, false, kTall, kInPlace>;
    return tma ? (const void*)sob_smooth3_kernel<R, true, kShort, kInPlace>
               : (const void*)sob_smooth3_kernel<R, false, kShort, kInPlace>;
}

// nullptr where sob_smooth_split never asks for the form
template <int R>
const void* smooth_unrolled_fn(bool transposed, bool tall) {
    if constexpr (sob_smooth_ever_one_unrolled(R)) {
        constexpr int kShort = sob_smooth_tile_y(R, false), kTall = sob_smooth_tile_y(R, true);
        if (transposed)
            return tall ? (const void*)sob_smooth3_kernel<R, false, kTall, kTranspose>
                        : (const void*)sob_smooth3_kernel<R, false, kShort, kTranspose>;
        return tall ? (const void*)sob_smooth3_kernel<R, false, kTall, kOutOfPlace>
                    : (const void*)sob_smooth3_kernel<R, false, kShort, kOutOfPlace>;
    }
    return nullptr;
}

template <int R>
void smooth_split_fns(SmoothForm form, bool tall, const void** planes, const void** z) {
    *planes = *z = nullptr;
    if constexpr (sob_smooth_ever_split(R)) {
        constexpr int kShort = sob_smooth_tile_y(R, false), kTall = sob_smooth_tile_y(R, true);
        if (form == kSmoothTransposed)
            *planes = tall ? (const void*)sob_smooth3_kernel<R, false, kTall, kPlanesTranspose>
                           : (const void*)sob_smooth3_kernel<R, false, kShort, kPlanesTranspose>;
        else
            *planes = tall ? (const void*)sob_smooth3_kernel<R, false, kTall, kPlanes>
                           : (const void*)sob_smooth3_kernel<R, false, kShort, kPlanes>;
        *z = form == kSmoothTransposed ? (const void*)sob_smooth_z_kernel<R, kTranspose>
             : form == kSmoothUnrolled ? (const void*)sob_smooth_z_kernel<R, kOutOfPlace>
                                       : (const void*)sob_smooth_z_kernel<R, kInPlace>;
    }
}

}  // namespace

void sob_smooth_split_fns(int radius, SmoothForm form, bool tall, const void** planes, const void** z) {
    switch (radius) {
        case 0: return smooth_split_fns<0>(form, tall, planes, z);
        case 1: return smooth_split_fns<1>(form, tall, planes, z);
        case 2: return smooth_split_fns<2>(form, tall, planes, z);
        case 3: return smooth_split_fns<3>(form, tall, planes, z);
        case 4: return smooth_split_fns<4>(form, tall, planes, z);
        case 5: return smooth_split_fns<5>(form, tall, planes, z);
        case 6: return smooth_split_fns<6>(form, tall, planes, z);
        default: return smooth_split_fns<7>(form, tall, planes, z);
    }
}

cudaError_t launch_smooth_split(const SobIterArgs& a, SmoothForm form, bool tall, int grid, cudaStream_t s, bool behind) {
    const void *planes, *z;
    sob_smooth_split_fns(a.radius, form, tall, &planes, &z);
    void* args[1] = {const_cast<SobIterArgs*>(&a)};
    const cudaError_t e = launch_kernel(planes, grid, kSmoothThreads, 0, args, s, behind);
    return e != cudaSuccess ? e : launch_kernel(z, 3 * a.ntiles_z, 256, 0, args, s, behind);
}

const void* sob_smooth3_fn(int radius, int tma, bool tall) {
    switch (radius) {
        case 0: return smooth_fn<0>(tma, tall);
        case 1: return smooth_fn<1>(tma, tall);
        case 2: return smooth_fn<2>(tma, tall);
        case 3: return smooth_fn<3>(tma, tall);
        case 4: return smooth_fn<4>(tma, tall);
        case 5: return smooth_fn<5>(tma, tall);
        case 6: return smooth_fn<6>(tma, tall);
        default: return smooth_fn<7>(tma, tall);
    }
}

const void* sob_smooth3_unrolled_fn(int radius, bool transposed, bool tall) {
    switch (radius) {
        case 0: return smooth_unrolled_fn<0>(transposed, tall);
        case 1: return smooth_unrolled_fn<1>(transposed, tall);
        case 2: return smooth_unrolled_fn<2>(transposed, tall);
        case 3: return smooth_unrolled_fn<3>(transposed, tall);
        case 4: return smooth_unrolled_fn<4>(transposed, tall);
        case 5: return smooth_unrolled_fn<5>(transposed, tall);
        case 6: return smooth_unrolled_fn<6>(transposed, tall);
        default: return smooth_unrolled_fn<7>(transposed, tall);
    }
}

}  // namespace frg
