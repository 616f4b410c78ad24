// nb_force_mixed.cuh -- the mixed-precision direct-sum force kernels for
// sm_103a, templated on the j-tile size TJ (128, 256, 512 sources) and the
// depth NST of the shared-memory ring; nb_force_mixed_t{128,256,512}.cu
// instantiate them per tile size and nb_force_mixed.cu dispatches.
//
// Replaces compute_force_gpu_kernel (src/directsumgpu/gravity.jl:22-34), which
// reads every source from global memory once per target thread, with:
//   * a pack kernel that writes sources as FP32 float4 (x-o, y-o, z-o, m) in
//     j-tiles of TJ particles, with an FP64 origin o per tile (the centre of
//     the tile's bounding box), kept as a float pair hi + lo;
//   * a force kernel whose CTA holds BLOCK*IPT targets in registers and streams
//     every j-tile through shared memory with bulk async copies
//     (cp.async.bulk ... mbarrier::complete_tx, per CTA, no multicast) in an
//     NST-deep ring.  Each target's position is re-expressed relative to the
//     tile origin with three FP32 operations per coordinate, then the pair
//     loop runs in FP32.  Per-tile FP32 partial sums are folded into
//     (sum, carry) pairs with TwoSum.
//
// Pair law (per target softening h, src/directsum/gravity.jl:8-28):
//   r >= h : a += m d / r^3                 (fast path, branch-free)
//   r <  h : Gadget-2 spline polynomial     (rare slow path; includes j == i)
// Potential (src/directsum/potential.jl:2-27): -m/r, spline inside h, 0 at r=0.
#pragma once

#include <cooperative_groups.h>

#include "nb_pairs.cuh"

namespace nb {

// ---------------------------------------------------------------------------
// Pack: one CTA of TJ threads per j-tile.  Slot i of the packed array holds
// particle perm[i] (identity when perm == nullptr), in pairs: slots 2p, 2p+1 of
// a tile are stored as float4 (x0, x1, y0, y1), float4 (z0, z1, m0, m1), so
// the packed-FP32x2 pair loop evaluates two sources per instruction.  The tile
// origin is the centre of the tile's FP64 bounding box, origin.w its half
// diagonal.
// ---------------------------------------------------------------------------
// Optional extras (PackExtra): with DRIFT each particle takes its step's drift
// first, in the operation order of k_drift (the step's own kernel for it read
// and wrote the same positions once more); the active particles are counted for
// the active list; the split positions go out by
// slot for the force kernel, which otherwise gathers and splits them anew in
// every CTA (12 FP64-pipe operations per target, 0.4 us of an SM's FP64 pipe
// per 128 targets).
template <int TJ, bool DRIFT>
__global__ void __launch_bounds__(TJ) k_pack(const double* __restrict__ x,
                                                 const double* __restrict__ y,
                                                 const double* __restrict__ z,
                                                 const double* __restrict__ m, int64_t n,
                                                 const int32_t* __restrict__ perm,
                                                 float4* __restrict__ pack,
                                                 TileOrigin* __restrict__ origin,
                                                 float4* __restrict__ ext, PackExtra e) {
    // Each particle is split once into a double-float pair (12 FP64-pipe
    // operations, the slow pipe on this GPU).  The tile's box is reduced in
    // FP32 from the pairs relative to the tile's first particle c, the
    // common-mass test compares bit patterns, and thread 0 alone forms the
    // FP64 tile origin c + float offset and shares it.
    __shared__ float red[6][TJ / 32];
    __shared__ double cref[4];
    __shared__ float2 csplit[3];
    __shared__ TileOrigin tile_o;
    const int64_t i = (int64_t)blockIdx.x * TJ + threadIdx.x;
    const bool valid = i < n;
    double px = 0.0, py = 0.0, pz = 0.0, pm = 0.0;
    float hs = 0.0f;
    if (e.done)
        for (int64_t k = i; k < e.ndone; k += (int64_t)gridDim.x * TJ) e.done[k] = 0;
    if (valid) {
        const int64_t p = perm ? (int64_t)perm[i] : i;
        if (DRIFT) {
            const double t = e.clk->t_float;
            const double dt = e.dt > 0.0 ? __dadd_rn(__dadd_rn(t, e.dt), -t) : e.clk->dt_drift;
            px = __dadd_rn(e.x[p], __dmul_rn(e.vx[p], dt));
            py = __dadd_rn(e.y[p], __dmul_rn(e.vy[p], dt));
            pz = __dadd_rn(e.z[p], __dmul_rn(e.vz[p], dt));
            e.x[p] = px;
            e.y[p] = py;
            e.z[p] = pz;
        } else {
            px = x[p];
            py = y[p];
            pz = z[p];
        }
        pm = m[p];
        if (e.split) hs = (float)(e.type ? e.soft[e.type[p] - 1] : e.h_const);
    }
    if (e.counts) {
        // active particles (Ti_endstep == t_int) per 128 slots
        __shared__ uint32_t wact[TJ / 32];
        const bool act = valid && e.ti_end[perm ? (int64_t)perm[i] : i] == e.clk->t_int;
        const unsigned mask = __ballot_sync(0xffffffffu, act);
        if ((threadIdx.x & 31) == 0) wact[threadIdx.x >> 5] = __popc(mask);
        __syncthreads();
        if ((threadIdx.x & 127) == 0) {
            const uint32_t* w = wact + (threadIdx.x >> 5);
            if (i < n) e.counts[i >> 7] = w[0] + w[1] + w[2] + w[3];
        }
    }
    const float2 sx = split_df(px), sy = split_df(py), sz = split_df(pz);
    if (e.split && valid) {
        e.split[2 * i] = make_float4(sx.x, sx.y, sy.x, sy.y);
        e.split[2 * i + 1] = make_float4(sz.x, sz.y, hs, 0.0f);
    }
    if (threadIdx.x == 0) {  // every tile holds at least one particle (tiles cover [0, n))
        cref[0] = px;
        cref[1] = py;
        cref[2] = pz;
        cref[3] = pm;
        csplit[0] = sx;
        csplit[1] = sy;
        csplit[2] = sz;
    }
    __syncthreads();
    const double m0 = cref[3];
    // offsets from c for the box (within a few FP32 ulp of the FP64 offsets;
    // the box is enlarged below to cover that)
    const float fx = rel_df(sx, csplit[0].x, csplit[0].y);
    const float fy = rel_df(sy, csplit[1].x, csplit[1].y);
    const float fz = rel_df(sz, csplit[2].x, csplit[2].y);
    const bool same_mass = !valid || __double_as_longlong(pm) == __double_as_longlong(m0);
    float v[6];
    v[0] = valid ? fx : 3e38f;
    v[1] = valid ? fy : 3e38f;
    v[2] = valid ? fz : 3e38f;
    v[3] = valid ? -fx : 3e38f;
    v[4] = valid ? -fy : 3e38f;
    v[5] = valid ? -fz : 3e38f;
#pragma unroll
    for (int k = 0; k < 6; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] = fminf(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < 6; ++k) red[k][warp] = v[k];
    }
    const bool uniform = __syncthreads_and(same_mass) && m0 > 0.0;
    float lo[3], hi[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float a = red[k][0], b = red[k + 3][0];
#pragma unroll
        for (int w = 1; w < TJ / 32; ++w) {
            a = fminf(a, red[k][w]);
            b = fminf(b, red[k + 3][w]);
        }
        lo[k] = a;
        hi[k] = -b;
    }
    const float ex = hi[0] - lo[0], ey = hi[1] - lo[1], ez = hi[2] - lo[2];
    const float amax = fmaxf(fmaxf(fabsf(lo[0]), fabsf(hi[0])),
                             fmaxf(fmaxf(fabsf(lo[1]), fabsf(hi[1])), fmaxf(fabsf(lo[2]), fabsf(hi[2]))));
    if (threadIdx.x == 0) {
        // origin at the box centre; the half diagonal is enlarged to cover the
        // rounding of the FP32 relative coordinates
        const float rr = 0.5f * sqrtf(ex * ex + ey * ey + ez * ez);
        tile_o = make_tile_origin(cref[0] + (double)(0.5f * (lo[0] + hi[0])),
                                  cref[1] + (double)(0.5f * (lo[1] + hi[1])),
                                  cref[2] + (double)(0.5f * (lo[2] + hi[2])),
                                  (double)rr * (1.0 + 1e-5) + 4.0e-7 * (double)amax);
    }
    __syncthreads();
    const TileOrigin to = tile_o;
    // ext.w: the common mass m of the tile's sources when all are equal (the
    // pair loops then apply it once per tile), else 0.  A partial tile stores
    // -m: its far padding adds exactly 0 to the acceleration in that form
    // (r^-3 underflows) but not to the potential, so the potential loops use
    // the per-pair masses there.
    const bool full = ((int64_t)blockIdx.x + 1) * TJ <= n;
    const float mu = uniform ? (full ? (float)m0 : -(float)m0) : 0.0f;
    // Sources relative to the origin by the same FP32 steps the force kernels
    // apply to targets (rel_df), so a particle's own source entry and its
    // target coordinates are bit-identical and the self pair has r = 0.
    float qx = 1e18f, qy = 1e18f, qz = 1e18f, qm = 0.0f;
    if (valid) {
        qx = rel_df(sx, to.hi.x, to.lo.x);
        qy = rel_df(sy, to.hi.y, to.lo.y);
        qz = rel_df(sz, to.hi.z, to.lo.z);
        qm = (float)pm;
    }
    // A full tile of one common mass keeps that mass in ext.w only; its mass
    // slots hold |q|^2 for the expanded far loop (pair_loop_expand).  Every
    // pair loop takes the mass of such a tile from ext.w.
    if (mu > 0.0f) qm = fmaf(qx, qx, fmaf(qy, qy, qz * qz));
    // (Zero-mass padding far away contributes exactly 0 and never takes the
    // r < h path.)  Paired layout: sources 2p and 2p+1 of the tile occupy
    // float4 (x0, x1, y0, y1) and float4 (z0, z1, m0, m1).
    float* base = reinterpret_cast<float*>(pack + (int64_t)blockIdx.x * TJ);
    const int pr = threadIdx.x >> 1, half = threadIdx.x & 1;
    base[8 * pr + half] = qx;
    base[8 * pr + 2 + half] = qy;
    base[8 * pr + 4 + half] = qz;
    base[8 * pr + 6 + half] = qm;
    if (threadIdx.x == 0) {
        origin[blockIdx.x] = to;
        // Half extents of the box for the near test, enlarged to cover the
        // rounding of the FP32 relative coordinates (the test must never
        // under-estimate them).
        const float slack = 4.0e-7f * amax;
        ext[blockIdx.x] = make_float4(0.5f * ex * (1.0f + 1e-5f) + slack, 0.5f * ey * (1.0f + 1e-5f) + slack,
                                      0.5f * ez * (1.0f + 1e-5f) + slack, mu);
    }
}


// ---------------------------------------------------------------------------
// Force kernel.
//
// CTA = BLOCK threads, IPT targets per thread (slot k*BLOCK + tid).  Targets'
// FP64 positions live in shared memory as float pairs hi + lo; per j-tile each
// thread re-expresses them relative to the tile origin (also hi + lo) with
// three FP32 operations per coordinate, so the tile loop issues no FP64
// instruction.
//
// j-tiles of TJ sources stream through an NST-stage ring.  full[s] (mbarrier, count 1 +
// transaction bytes) completes when the bulk copy of the tile has landed.
// There is no CTA-wide barrier per tile: every warp bumps done[s] after it has
// read stage s, and the last warp to do so re-arms full[s] and issues the copy
// of tile t + NST into it.  Warps may therefore run up to NST - 1
// tiles apart.  Every wait is bounded; a timed-out warp records
// DEVERR_TIMEOUT and stops, and the CTA drains its copies before exiting.
// ---------------------------------------------------------------------------
// CTAs per SM the register allocation is held to (acceleration-only launches
// of 128 threads); overridable at build time for launch-shape experiments.
#ifndef NB_MINB_IPT1
#define NB_MINB_IPT1 6
#endif
#ifndef NB_MINB_IPT2
#define NB_MINB_IPT2 5
#endif
#ifndef NB_MINB_IPT4
#define NB_MINB_IPT4 1
#endif
// With the potential: alone 7 and 6 CTAs (one, two targets per thread; N = 50021:
// 755 -> 720 us, N = 100003: 2483 -> 2402 us against the compiler's choice of 6
// and 4), beside the acceleration 5 and its choice (1090 -> 1078 us).
template <int BLOCK, int IPT, bool ACC, bool POT>
struct ForceOcc {
    static constexpr int value =
        BLOCK != 128 ? 1
        : !POT       ? (IPT == 1 ? NB_MINB_IPT1 : (IPT == 2 ? NB_MINB_IPT2 : NB_MINB_IPT4))
        : ACC        ? (IPT == 1 ? 5 : 1)
                     : (IPT == 1 ? 7 : (IPT == 2 ? 6 : 1));
};

// The clock update of a constant step whose drift ran in the pack (one thread).
__device__ __forceinline__ void end_constant_step(const Targets& tg) {
    Clock* c = tg.step_clk;
    const double t = c->t_float;
    c->t_float = __dadd_rn(t, tg.kick_dt);
    c->dt_drift = __dadd_rn(c->t_float, -t);
    c->last_t_float = c->t_float;  // src/run.jl:164
    c->interactions = __dadd_rn(c->interactions, __dmul_rn((double)tg.n, (double)tg.n));
    c->steps += 1;
}

// Join of a block whose parts are one cluster: every CTA leaves its compensated
// sums in its shared memory (sum: 6 x kPer floats) and joins a js-th of the
// block's targets from all of them, one (target, component) per thread, in part
// order.  Against the join by the last CTA through global memory this saves
// the sums' round trip through the L2, the count, and most of the time of the
// FP64 epilogue, which one CTA's threads otherwise share the FP64 pipe of one
// SM for: 5.7 of 19.5 us of a force launch at N = 4096, 3.7 of 7.4 at N = 1000.
// A part whose wait ran out (gave_up, CTA-uniform) leaves a mark in place of its
// sums, a NaN that no sum can be, and then no CTA of the block stores, kicks or
// advances the clock.
constexpr uint32_t kGaveUp = 0x7fe0dead;

template <int BLOCK, int IPT>
__device__ __forceinline__ void cluster_join(float* sum, bool gave_up, int js, int part, int64_t base, int64_t ntg,
                                             const float* sx, const float* cx, const float* sy,
                                             const float* cy, const float* sz, const float* cz,
                                             const Targets& tg, double G) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    constexpr int kPer = BLOCK * IPT;
    const int tid = threadIdx.x;
    __syncthreads();  // every warp is done with the tiles that sum overwrites
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        float* q = sum + k * BLOCK + tid;
        q[0 * kPer] = sx[k];
        q[1 * kPer] = cx[k];
        q[2 * kPer] = sy[k];
        q[3 * kPer] = cy[k];
        q[4 * kPer] = sz[k];
        q[5 * kPer] = cz[k];
    }
    if (gave_up)
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int k = 0; k < IPT; ++k) sum[2 * j * kPer + k * BLOCK + tid] = __uint_as_float(kGaveUp);
    const int seg = (kPer + js - 1) / js, lo = part * seg;
    bool whole = true;
    cluster.sync();
    for (int i = tid; i < 3 * seg; i += BLOCK) {
        const int comp = i / seg, slot = lo + i % seg;
        const int64_t t = base + slot;
        if (slot >= kPer || t >= ntg) continue;
        const int32_t p = tg.idx ? tg.idx[t] : (int32_t)t;
        double* a = comp == 0 ? tg.ax : comp == 1 ? tg.ay : tg.az;
        double* v = comp == 0 ? tg.vx : comp == 1 ? tg.vy : tg.vz;
        const double vp = v ? v[p] : 0.0;
        float s = 0.0f, c = 0.0f;
#pragma unroll 8
        for (int u = 0; u < js; ++u) {
            const float* q = cluster.map_shared_rank(sum + 2 * comp * kPer + slot, u);
            const float v = q[0];
            whole = whole && __float_as_uint(v) != kGaveUp;
            two_sum_acc(s, c, v);
            c += q[kPer];
        }
        if (!whole) break;
        const double acc = ((double)s + (double)c) * G;
        a[p] = acc;
        if (v) v[p] = __dadd_rn(vp, __dmul_rn(acc, tg.kick_dt));  // k_kick with constant steps
    }
    // (this thread has joined the block's first target)
    if (tg.step_clk && base == 0 && part == 0 && tid == 0 && whole) end_constant_step(tg);
    cluster.sync();  // the last read of another CTA's shared memory
}

// The shape that small systems run in.  The others do without: its mere
// presence changed the pair loop's schedule (N = 2^20: 344 -> 356 ms a step).
template <int BLOCK, int IPT, int TJ, bool ACC, bool POT>
constexpr bool kClusterJoin = BLOCK == 128 && IPT == 1 && TJ == 128 && ACC && !POT;

template <int LAW, bool ACC, bool POT, int BLOCK, int IPT, int TJ, int NST>
__global__ void __launch_bounds__(BLOCK, (ForceOcc<BLOCK, IPT, ACC, POT>::value)) k_force_mixed(Sources32 src, Targets tg, double G,
                                                       uint32_t* __restrict__ err) {
    static_assert(TJ == 128 || TJ == 256 || TJ == 512, "tile of 128, 256 or 512 sources");
    constexpr int kWarpsPerCta = BLOCK / 32;
    __shared__ __align__(128) float4 buf[NST * TJ];
    __shared__ __align__(8) uint64_t full[NST];
    __shared__ uint32_t done[NST];
    __shared__ uint32_t abort_flag;
    __shared__ float2 tpx[BLOCK * IPT], tpy[BLOCK * IPT], tpz[BLOCK * IPT];

    const int64_t ntg = tg.d_count ? (int64_t)(*tg.d_count) : tg.n;
    const int64_t nblk = (ntg + BLOCK * IPT - 1) / (BLOCK * IPT);
    const int js = !src.partial ? 1 : src.jsplit > 0 ? src.jsplit : split_parts(nblk, src.ntiles);
    const int64_t blk = (int64_t)blockIdx.x / js;
    const int part = (int)(blockIdx.x % js);
    const int64_t base = blk * (BLOCK * IPT);
    if (blk >= nblk) return;  // CTA-uniform
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int t_lo = (int)((int64_t)part * src.ntiles / js);
    const int ntiles = (int)((int64_t)(part + 1) * src.ntiles / js) - t_lo;  // tiles of this CTA

    if (tid == 0) {
#pragma unroll
        for (int s = 0; s < NST; ++s) {
            mbar_init(&full[s], 1);
            done[s] = 0;
        }
        abort_flag = 0;
        fence_mbar_init();
    }

    int32_t pidx[IPT];  // the particle index, or with split positions the slot; -1: none
    float hh[IPT], h2[IPT];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int64_t t = base + k * BLOCK + tid;
        pidx[k] = -1;
        if (tg.split) {
            float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), b = a;
            if (t < ntg) {
                pidx[k] = (int32_t)t;
                a = tg.split[2 * t];
                b = tg.split[2 * t + 1];
            }
            tpx[k * BLOCK + tid] = make_float2(a.x, a.y);
            tpy[k * BLOCK + tid] = make_float2(a.z, a.w);
            tpz[k * BLOCK + tid] = make_float2(b.x, b.y);
            hh[k] = b.z;
            h2[k] = hh[k] * hh[k];
            continue;
        }
        double x = 0.0, y = 0.0, z = 0.0, h = tg.h_const;
        if (t < ntg) {
            const int32_t p = tg.idx ? tg.idx[t] : (int32_t)t;
            pidx[k] = p;
            x = tg.x[p];
            y = tg.y[p];
            z = tg.z[p];
            if (tg.type) h = tg.soft[tg.type[p] - 1];
        }
        tpx[k * BLOCK + tid] = split_df(x);
        tpy[k * BLOCK + tid] = split_df(y);
        tpz[k * BLOCK + tid] = split_df(z);
        hh[k] = (float)h;
        h2[k] = hh[k] * hh[k];
    }
    __syncthreads();
    if (tid == 0) {
        for (int s = 0; s < NST && s < ntiles; ++s) {
            mbar_arrive_expect_tx(&full[s], TJ * sizeof(float4));
            bulk_g2s(&buf[s * TJ], src.pack + (int64_t)(t_lo + s) * TJ, TJ * sizeof(float4),
                     &full[s]);
        }
    }

    float sx[IPT], sy[IPT], sz[IPT], sp[IPT];
    float cx[IPT], cy[IPT], cz[IPT], cp[IPT];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        sx[k] = sy[k] = sz[k] = sp[k] = 0.0f;
        cx[k] = cy[k] = cz[k] = cp[k] = 0.0f;
    }

    bool timed_out = false;
    for (int t = 0; t < ntiles; ++t) {
        const int s = t % NST;
        const uint32_t par = (uint32_t)(t / NST) & 1u;
        const float4 oh = src.origin[t_lo + t].hi, ol = src.origin[t_lo + t].lo;
        float xr[IPT], yr[IPT], zr[IPT];
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            xr[k] = rel_df(tpx[k * BLOCK + tid], oh.x, ol.x);
            yr[k] = rel_df(tpy[k * BLOCK + tid], oh.y, ol.y);
            zr[k] = rel_df(tpz[k * BLOCK + tid], oh.z, ol.z);
        }
        float ax[IPT], ay[IPT], az[IPT], ap[IPT];
#pragma unroll
        for (int k = 0; k < IPT; ++k) ax[k] = ay[k] = az[k] = ap[k] = 0.0f;

        const bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(&full[s], par, kWaitTimeoutNs));
        if (!ok || abort_flag) {
            timed_out = true;
            if (lane == 0) {
                atomicOr(err, DEVERR_TIMEOUT);
                atomicExch(&abort_flag, 1u);
            }
            break;
        }
        const float4* b = &buf[s * TJ];
        // Warp-uniform choice of the pair loop: when every target of the warp
        // lies farther than (tile radius + h) from the tile origin, no pair of
        // this tile can have r < h and the branch-free loop runs.
        const float4 ex = src.ext[t_lo + t];
        bool near = false;
        if (LAW == NB_LAW_SPLINE_G2) near = warp_near<IPT>(ex, xr, yr, zr, hh, pidx);
        if (near)
            pair_loop_checked<LAW, ACC, POT, IPT, TJ>(b, xr, yr, zr, hh, h2, ax, ay, az, ap, ex.w);
        else if (ex.w > 0.0f && warp_expandable<IPT>(ex, oh.w, xr, yr, zr, pidx))
            pair_loop_expand<LAW, ACC, POT, IPT, TJ>(b, xr, yr, zr, h2, ax, ay, az, ap, ex.w);
        else
            pair_loop_far<LAW, ACC, POT, IPT, TJ>(b, xr, yr, zr, h2, ax, ay, az, ap, ex.w);

        // Release stage s; the last warp out refills it with tile t + NST.
        __syncwarp();
        if (lane == 0) {
            __threadfence_block();
            const uint32_t prev = atomicAdd(&done[s], 1u);
            if (prev == kWarpsPerCta - 1) {
                __threadfence_block();
                done[s] = 0;
                if (t + NST < ntiles) {
                    mbar_arrive_expect_tx(&full[s], TJ * sizeof(float4));
                    bulk_g2s(&buf[s * TJ], src.pack + (int64_t)(t_lo + t + NST) * TJ,
                             TJ * sizeof(float4), &full[s]);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            if (ACC) {
                two_sum_acc(sx[k], cx[k], ax[k]);
                two_sum_acc(sy[k], cy[k], ay[k]);
                two_sum_acc(sz[k], cz[k], az[k]);
            }
            if (POT) two_sum_acc(sp[k], cp[k], ap[k]);
        }
    }

    if (__syncthreads_or(timed_out)) {
        if (tid == 0) {
            // Drain every copy that may still be in flight before exiting.
            for (int u = 0; u < ntiles; ++u)
                (void)mbar_wait_bounded(&full[u % NST], (uint32_t)(u / NST) & 1u,
                                        kWaitTimeoutNs / 8);
        }
        // (a cluster's CTAs stay: the others read their shared memory)
        if (!(kClusterJoin<BLOCK, IPT, TJ, ACC, POT> && src.cluster)) return;
    }

    if constexpr (kClusterJoin<BLOCK, IPT, TJ, ACC, POT>) {
        if (src.cluster) {
            cluster_join<BLOCK, IPT>(reinterpret_cast<float*>(buf), abort_flag != 0u, js, part, base, ntg, sx, cx, sy, cy, sz,
                                     cz, tg, G);
            return;
        }
    }
    if (js > 1) {
        // Compensated partials of this CTA's tile range; the CTA that finishes
        // last adds its block's parts in part order as double-float numbers in
        // FP32 (TwoSum of the sums, carries added), about 48 bits.  Which CTA
        // that is does not change the result.
        constexpr int64_t kPer = BLOCK * IPT;
        float* q0 = src.partial + blk * js * 8 * kPer + tid;
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            float* q = q0 + part * 8 * kPer + k * BLOCK;
            const float v[8] = {sx[k], cx[k], sy[k], cy[k], sz[k], cz[k], sp[k], cp[k]};
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (j < 6 ? ACC : POT) __stcg(q + j * kPer, v[j]);
        }
        __threadfence();  // the sums before the count
        __syncthreads();
        if (tid == 0) abort_flag = atomicAdd(&src.done[blk], 1u) == (uint32_t)(js - 1);
        __syncthreads();
        if (!abort_flag) return;
        if (tg.vx) {  // the velocities that the kick will want
#pragma unroll
            for (int k = 0; k < IPT; ++k) {
                if (pidx[k] < 0) continue;
                const int32_t p = tg.split && tg.idx ? tg.idx[pidx[k]] : pidx[k];
                prefetch_l1(tg.vx + p);
                prefetch_l1(tg.vy + p);
                prefetch_l1(tg.vz + p);
            }
        }
        __threadfence();  // the count before the other parts' sums
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            sx[k] = sy[k] = sz[k] = sp[k] = 0.0f;
            cx[k] = cy[k] = cz[k] = cp[k] = 0.0f;
        }
        // kJU parts at a time, their loads in flight together (an L2 round trip
        // each batch, which the join of a small system mostly waits for)
        constexpr int kJU = IPT == 1 ? 8 : 4;
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            for (int u0 = 0; u0 < js; u0 += kJU) {
                float v[kJU][8];
#pragma unroll
                for (int u = 0; u < kJU; ++u)
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (j < 6 ? ACC : POT)
                            v[u][j] = u0 + u < js ? __ldcg(q0 + ((u0 + u) * 8 + j) * kPer + k * BLOCK) : 0.0f;
#pragma unroll
                for (int u = 0; u < kJU; ++u) {
                    if (ACC) {
                        two_sum_acc(sx[k], cx[k], v[u][0]);
                        cx[k] += v[u][1];
                        two_sum_acc(sy[k], cy[k], v[u][2]);
                        cy[k] += v[u][3];
                        two_sum_acc(sz[k], cz[k], v[u][4]);
                        cz[k] += v[u][5];
                    }
                    if (POT) {
                        two_sum_acc(sp[k], cp[k], v[u][6]);
                        cp[k] += v[u][7];
                    }
                }
            }
        }
    }
    if (tg.step_clk && blk == 0 && tid == 0) end_constant_step(tg);
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        if (pidx[k] < 0) continue;
        const int32_t p = tg.split && tg.idx ? tg.idx[pidx[k]] : pidx[k];
        if (ACC) {
            const double a0 = ((double)sx[k] + (double)cx[k]) * G;
            const double a1 = ((double)sy[k] + (double)cy[k]) * G;
            const double a2 = ((double)sz[k] + (double)cz[k]) * G;
            tg.ax[p] = a0;
            tg.ay[p] = a1;
            tg.az[p] = a2;
            if (tg.vx) {  // k_kick with constant steps, its operation order
                tg.vx[p] = __dadd_rn(tg.vx[p], __dmul_rn(a0, tg.kick_dt));
                tg.vy[p] = __dadd_rn(tg.vy[p], __dmul_rn(a1, tg.kick_dt));
                tg.vz[p] = __dadd_rn(tg.vz[p], __dmul_rn(a2, tg.kick_dt));
            }
        }
        if (POT) {
            // The loops accumulate +m/r; phi = -sum.
            double phi = -((double)sp[k] + (double)cp[k]);
            if (LAW == NB_LAW_PLUMMER && tg.self_mass) {
                // Remove the self pair, bit-identical to the term the loop added.
                const float mself = (float)tg.self_mass[p];
                phi += (double)(mself * rsqrt_approx(h2[k]));
            }
            tg.pot[p] = phi * G;
        }
    }
}

// Small systems: the parts of each block as one cluster of up to 8 CTAs, the
// portable size, while the clusters of all blocks run at once.  us a step with /
// without clusters: N = 1000 14.5 / 16.6, 2048 16.5 / 18.6, 4096 22.7 / 25.4,
// 8192 47.7 / 47.1, 16384 140 / 127.
constexpr int kClusterParts = 8;
constexpr int64_t kClusterBlocks = 48;
inline bool cluster_split(const Sources32& src, const Targets& tg, int64_t nblk) {
    return src.partial && src.jsplit == 0 && !tg.d_count && tg.split && src.ntiles > 1 &&
           nblk <= kClusterBlocks;
}

// Launch of one force evaluation with tiles of TJ sources (instantiated in
// nb_force_mixed_t<TJ>.cu).  Shapes: (128 | 256 threads) x (1 | 2 | 4 targets
// per thread) with the default 4-stage ring; the acceleration-only form of
// 128 x 1 and 128 x 2 also with 3 and 6 stages (6 only for tiles of up to 256
// sources: 6 x 8 KiB would pass the 48 KiB of static shared memory).  Other
// combinations use 4 stages.
template <int LAW, bool ACC, bool POT, int TJ>
cudaError_t launch_cfg_tile(const Sources32& src, const Targets& tg, double G, uint32_t* err,
                            int block, int ipt, int stages, cudaStream_t s) {
    const int64_t per = (int64_t)block * ipt, nblk = (tg.n + per - 1) / per;
    if (nblk <= 0) return cudaSuccess;
    // an active list may hold fewer blocks, split into more parts each: at most
    // kSplitItems items where that is more than 8 per block
    const int js = !src.partial ? 1 : src.jsplit > 0 ? src.jsplit : split_parts(nblk, src.ntiles);
    int64_t grid = nblk * js;
    if constexpr (kClusterJoin<128, 1, TJ, ACC, POT>) {
        if (block == 128 && ipt == 1 && stages == 4 && cluster_split(src, tg, nblk)) {
            Sources32 sc = src;
            sc.cluster = 1;
            sc.jsplit = src.ntiles < kClusterParts ? src.ntiles : kClusterParts;
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3((unsigned)(nblk * sc.jsplit));
            cfg.blockDim = dim3(128);
            cfg.stream = s;
            cudaLaunchAttribute at{};
            at.id = cudaLaunchAttributeClusterDimension;
            at.val.clusterDim.x = (unsigned)sc.jsplit;
            at.val.clusterDim.y = 1;
            at.val.clusterDim.z = 1;
            cfg.attrs = &at;
            cfg.numAttrs = 1;
            return cudaLaunchKernelEx(&cfg, k_force_mixed<LAW, ACC, POT, 128, 1, TJ, 4>, sc, tg, G, err);
        }
    }
    if (src.partial && src.jsplit == 0 && tg.d_count) {
        const int64_t most = nblk * src.ntiles < kSplitItems ? nblk * src.ntiles : kSplitItems;
        if (grid < most) grid = most;
    }
    bool launched = false;
#define NB_LAUNCH(B, I, S)                                                                  \
    if (!launched && block == B && ipt == I) {                                             \
        k_force_mixed<LAW, ACC, POT, B, I, TJ, S><<<(unsigned)grid, B, 0, s>>>(src, tg, G, err); \
        launched = true;                                                                   \
    }
    if constexpr (ACC && !POT) {
        if (stages == 3) {
            NB_LAUNCH(128, 1, 3)
            NB_LAUNCH(128, 2, 3)
        }
        if constexpr (TJ <= 256) {
            if (stages == 6) {
                NB_LAUNCH(128, 1, 6)
                NB_LAUNCH(128, 2, 6)
            }
        }
    }
    NB_LAUNCH(128, 1, 4)
    NB_LAUNCH(128, 2, 4)
    NB_LAUNCH(128, 4, 4)
    NB_LAUNCH(256, 1, 4)
    NB_LAUNCH(256, 2, 4)
    if constexpr (TJ <= 256) {
        // 1024 targets' positions (24 KiB) next to a ring of 512-source tiles
        // would pass the 48 KiB of static shared memory
        NB_LAUNCH(256, 4, 4)
    }
#undef NB_LAUNCH
    if (!launched) return cudaErrorInvalidValue;
    return cudaGetLastError();
}

template <int TJ>
cudaError_t launch_force_mixed_tile(int law, bool pot, const Sources32& src, const Targets& tg,
                                    double G, uint32_t* err, int block, int ipt, int stages,
                                    cudaStream_t s) {
    const bool acc = tg.ax != nullptr;
    if (!acc && !pot) return cudaSuccess;
    if (law == NB_LAW_PLUMMER) {
        if (!acc) return launch_cfg_tile<NB_LAW_PLUMMER, false, true, TJ>(src, tg, G, err, block, ipt, stages, s);
        return pot ? launch_cfg_tile<NB_LAW_PLUMMER, true, true, TJ>(src, tg, G, err, block, ipt, stages, s)
                   : launch_cfg_tile<NB_LAW_PLUMMER, true, false, TJ>(src, tg, G, err, block, ipt, stages, s);
    }
    if (!acc) return launch_cfg_tile<NB_LAW_SPLINE_G2, false, true, TJ>(src, tg, G, err, block, ipt, stages, s);
    return pot ? launch_cfg_tile<NB_LAW_SPLINE_G2, true, true, TJ>(src, tg, G, err, block, ipt, stages, s)
               : launch_cfg_tile<NB_LAW_SPLINE_G2, true, false, TJ>(src, tg, G, err, block, ipt, stages, s);
}

template <int TJ>
cudaError_t launch_pack_tile(const double* x, const double* y, const double* z, const double* m,
                             int64_t n, const int32_t* perm, float4* pack, TileOrigin* origin,
                             float4* ext, const PackExtra& px, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const int64_t ntiles = (n + TJ - 1) / TJ;
    if (px.vx)
        k_pack<TJ, true><<<(unsigned)ntiles, TJ, 0, s>>>(x, y, z, m, n, perm, pack, origin, ext, px);
    else
        k_pack<TJ, false><<<(unsigned)ntiles, TJ, 0, s>>>(x, y, z, m, n, perm, pack, origin, ext, px);
    return cudaGetLastError();
}

}  // namespace nb
