// nb_force_fp64.cu -- plain FP64 direct-sum force (the reference's Float64 form).
//
// Built with -fmad=false so every a*b+c rounds twice, as Julia evaluates the
// pair expressions of src/directsum/gravity.jl:8-28 and
// src/directsum/potential.jl:2-27; sqrt and division are IEEE-rounded.  Each
// pair term is therefore the same double the CPU computes; the per-target sum
// is compensated (TwoSum), so the result differs from the CPU's pairwise sum
// (src/directsum/gravity.jl:45) only by that sum's own rounding.
//
// Sources are staged through shared memory in tiles of kTile (x, y, z, m);
// one target per thread.
//
// What bounds it: the FP64 pipe (2 lanes per clock and SM on this GPU), about
// 60 FP64-pipe operations per pair, so the time is pairs / (busy SMs).  One
// block of targets per CTA leaves most SMs idle below 152 x 8 blocks (N =
// 4096: 32 CTAs on 152 SMs, 8.0 ms a force), so each block's sources are
// split over js CTAs (fp64_split) whose compensated partial sums are joined
// in part order by k_force_fp64_join: 1.76 ms a step at N = 4096, the rate
// of a full GPU (9.6 G interactions/s).
#include "nb_internal.cuh"

namespace nb {

constexpr int kTile = 128;
constexpr int kFp64Items = 8 * 152;   // (block, part) items a split evaluation aims at
constexpr int64_t kFp64MinPart = 32;  // fewest sources in a part

// Parts that each block of targets is split into.  Up to kFp64Items items in
// all: 8 CTAs of 128 threads fill an SM (60 registers), the items of one wave
// differ by at most 1 in 8 between SMs, and the partials stay within a fixed
// scratch (fp64_partial_bytes).  From kFp64Items / 2 blocks of targets on
// there is nothing to split.  Depends on the counts only, so the sums do not
// depend on scheduling; with an active list the count is the device's.
__host__ __device__ __forceinline__ int fp64_split(int64_t nblocks, int64_t nsrc) {
    int64_t js = nblocks > 0 ? kFp64Items / nblocks : 1;
    const int64_t most = nsrc / kFp64MinPart;
    if (js > most) js = most;
    return js < 1 ? 1 : (int)js;
}

size_t fp64_partial_bytes() { return sizeof(double) * 8 * (size_t)kFp64Items * kTile; }

template <int LAW>
__device__ __forceinline__ void pair_force64(double px, double py, double pz, dvec4 q, double G,
                                             double h, double h_inv, double h3_inv, double& fx,
                                             double& fy, double& fz) {
    const double dx = q.x - px, dy = q.y - py, dz = q.z - pz;
    const double r2 = dx * dx + dy * dy + dz * dz;
    double fac;
    if (LAW == NB_LAW_PLUMMER) {
        const double r2e = r2 + h * h;
        fac = q.w / (r2e * sqrt(r2e));
    } else {
        const double r = sqrt(r2);
        if (r >= h) {
            fac = q.w / (r2 * r);
        } else {
            const double u = r * h_inv;
            if (u < 0.5)
                fac = q.w * h3_inv * (10.666666666667 + u * u * (32.0 * u - 38.4));
            else
                fac = q.w * h3_inv *
                      (21.333333333333 - 48.0 * u + 38.4 * (u * u) - 10.666666666667 * (u * u * u) -
                       0.066666666667 / (u * u * u));
        }
    }
    fx = dx * fac * G;
    fy = dy * fac * G;
    fz = dz * fac * G;
}

template <int LAW>
__device__ __forceinline__ double pair_pot64(double px, double py, double pz, dvec4 q, double G,
                                             double h, double h_inv) {
    const double dx = q.x - px, dy = q.y - py, dz = q.z - pz;
    const double r2 = dx * dx + dy * dy + dz * dz;
    const double r = sqrt(r2);
    double pot;
    if (LAW == NB_LAW_PLUMMER) {
        pot = -q.w / sqrt(r2 + h * h) * G;
    } else if (r >= h) {
        pot = -q.w / r * G;
    } else {
        const double u = r * h_inv;
        double wp;
        if (u < 0.5)
            wp = -2.8 + u * u * (5.333333333333 + u * u * (6.4 * u - 9.6));
        else
            wp = -3.2 + 0.066666666667 / u +
                 u * u * (10.666666666667 + u * (-16.0 + u * (9.6 - 2.133333333333 * u)));
        pot = q.w * h_inv * wp * G;
    }
    if (r == 0.0) pot = pot * 0.0;
    return pot;
}

template <int LAW, bool ACC, bool POT>
__global__ void __launch_bounds__(kTile)
    k_force_fp64(Sources64 src, Targets tg, double G, double* __restrict__ partial) {
    __shared__ dvec4 sj[kTile];
    const int64_t ntg = tg.d_count ? (int64_t)(*tg.d_count) : tg.n;
    const int64_t nblocks = (ntg + kTile - 1) / kTile;
    const int js = fp64_split(nblocks, src.n);
    const int64_t blk = (int64_t)blockIdx.x / js;
    const int part = (int)((int64_t)blockIdx.x % js);
    if (blk >= nblocks) return;  // CTA-uniform
    const int64_t t = blk * kTile + threadIdx.x;
    int32_t p = -1;
    double px = 0.0, py = 0.0, pz = 0.0, h = tg.h_const;
    if (t < ntg) {
        p = tg.idx ? tg.idx[t] : (int32_t)t;
        px = tg.x[p];
        py = tg.y[p];
        pz = tg.z[p];
        if (tg.type) h = tg.soft[tg.type[p] - 1];
    }
    const double h_inv = 1.0 / h;
    const double h3_inv = h_inv * h_inv * h_inv;
    double sx = 0.0, sy = 0.0, sz = 0.0, sp = 0.0;
    double cx = 0.0, cy = 0.0, cz = 0.0, cp = 0.0;
    const int64_t jlo = src.n * part / js, jhi = src.n * (part + 1) / js;
    for (int64_t j0 = jlo; j0 < jhi; j0 += kTile) {
        __syncthreads();
        const int64_t jj = j0 + threadIdx.x;
        if (jj < jhi) sj[threadIdx.x] = make_dvec4(src.x[jj], src.y[jj], src.z[jj], src.m[jj]);
        __syncthreads();
        const int cnt = (int)((jhi - j0) < kTile ? (jhi - j0) : kTile);
        for (int j = 0; j < cnt; ++j) {
            const dvec4 q = sj[j];
            if (ACC) {
                double fx, fy, fz;
                pair_force64<LAW>(px, py, pz, q, G, h, h_inv, h3_inv, fx, fy, fz);
                two_sum_acc(sx, cx, fx);
                two_sum_acc(sy, cy, fy);
                two_sum_acc(sz, cz, fz);
            }
            if (POT) two_sum_acc(sp, cp, pair_pot64<LAW>(px, py, pz, q, G, h, h_inv));
        }
    }
    if (js > 1) {
        // compensated sums of this part, one row of kTile per quantity
        double* q = partial + (blk * js + part) * (8 * kTile) + threadIdx.x;
        if (ACC) {
            q[0 * kTile] = sx;
            q[1 * kTile] = cx;
            q[2 * kTile] = sy;
            q[3 * kTile] = cy;
            q[4 * kTile] = sz;
            q[5 * kTile] = cz;
        }
        if (POT) {
            q[6 * kTile] = sp;
            q[7 * kTile] = cp;
        }
        return;
    }
    if (p < 0) return;
    if (ACC) {
        tg.ax[p] = sx + cx;
        tg.ay[p] = sy + cy;
        tg.az[p] = sz + cz;
    }
    if (POT) tg.pot[p] = sp + cp;
}

// Adds the parts of every target in part order, sums with TwoSum and carries
// beside them, so a split evaluation keeps the accuracy of an unsplit one.
template <bool ACC, bool POT>
__global__ void __launch_bounds__(kTile)
    k_force_fp64_join(int64_t nsrc, Targets tg, const double* __restrict__ partial) {
    const int64_t ntg = tg.d_count ? (int64_t)(*tg.d_count) : tg.n;
    const int64_t nblocks = (ntg + kTile - 1) / kTile;
    const int js = fp64_split(nblocks, nsrc);
    const int64_t t = (int64_t)blockIdx.x * kTile + threadIdx.x;
    if (js == 1 || t >= ntg) return;
    const int32_t p = tg.idx ? tg.idx[t] : (int32_t)t;
    double s[4] = {0.0, 0.0, 0.0, 0.0}, c[4] = {0.0, 0.0, 0.0, 0.0};
    for (int part = 0; part < js; ++part) {
        const double* q = partial + ((int64_t)blockIdx.x * js + part) * (8 * kTile) + threadIdx.x;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (k < 3 ? !ACC : !POT) continue;
            two_sum_acc(s[k], c[k], q[(2 * k) * kTile]);
            c[k] += q[(2 * k + 1) * kTile];
        }
    }
    if (ACC) {
        tg.ax[p] = s[0] + c[0];
        tg.ay[p] = s[1] + c[1];
        tg.az[p] = s[2] + c[2];
    }
    if (POT) tg.pot[p] = s[3] + c[3];
}

template <int LAW>
static cudaError_t launch_law(bool acc, bool pot, const Sources64& src, const Targets& tg,
                              double G, double* partial, cudaStream_t s) {
    const int64_t nblocks = (tg.n + kTile - 1) / kTile;
    if (nblocks <= 0) return cudaSuccess;
    // an active list may leave any number of blocks up to nblocks, split further the fewer they are
    const int js = fp64_split(nblocks, src.n);
    const bool split = js > 1 || (tg.d_count && fp64_split(1, src.n) > 1);
    int64_t grid = nblocks * js;
    if (tg.d_count && split && grid < kFp64Items) grid = kFp64Items;
    if (acc && pot)
        k_force_fp64<LAW, true, true><<<(unsigned)grid, kTile, 0, s>>>(src, tg, G, partial);
    else if (acc)
        k_force_fp64<LAW, true, false><<<(unsigned)grid, kTile, 0, s>>>(src, tg, G, partial);
    else if (pot)
        k_force_fp64<LAW, false, true><<<(unsigned)grid, kTile, 0, s>>>(src, tg, G, partial);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || !split) return e;
    // blocks that can be split: at most kFp64Items / 2
    const int64_t jb = nblocks < kFp64Items / 2 ? nblocks : kFp64Items / 2;
    if (acc && pot)
        k_force_fp64_join<true, true><<<(unsigned)jb, kTile, 0, s>>>(src.n, tg, partial);
    else if (acc)
        k_force_fp64_join<true, false><<<(unsigned)jb, kTile, 0, s>>>(src.n, tg, partial);
    else if (pot)
        k_force_fp64_join<false, true><<<(unsigned)jb, kTile, 0, s>>>(src.n, tg, partial);
    return cudaGetLastError();
}

cudaError_t launch_force_fp64(int law, bool pot, const Sources64& src, const Targets& tg,
                              double G, double* partial, cudaStream_t s) {
    const bool acc = tg.ax != nullptr;
    if (law == NB_LAW_PLUMMER) return launch_law<NB_LAW_PLUMMER>(acc, pot, src, tg, G, partial, s);
    return launch_law<NB_LAW_SPLINE_G2>(acc, pot, src, tg, G, partial, s);
}

}  // namespace nb
