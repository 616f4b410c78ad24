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
// What bounds it: the FP64 pipe (2 lanes per clock and SM on this GPU), so the
// time is FP64 operations / busy SMs.  A pair takes 40 (counted by
// inst_executed_pipe_fp64; 43 unless G = 1): the separation and its square (8),
// the products with it (3), the three sums, ordered on the integer pipe
// (ordered_sum_acc, 12 instead of TwoSum's 21), and one square root and one
// quotient, shared by force and potential (17).  One
// block of targets per CTA leaves most SMs idle below 152 x 8 blocks (N =
// 4096: 32 CTAs on 152 SMs, 8.0 ms a force), so each block's sources are split
// over js CTAs (fp64_split) whose compensated partial sums are joined in part
// order by k_force_fp64_join: 1.31 ms a step at N = 4096, 12.5 G interactions/s
// at N = 12000.
// An own root and quotient from one reciprocal root took 1.24 ms there; their
// terms were other doubles for subnormal masses (28 % of them at 2^-1060) and
// the same elsewhere only as far as tried, so both are the compiler's.
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

// (s, c) += v as two_sum_acc, with the operands ordered by exponent on the
// integer pipe so that three additions give the rounding error (Dekker 1971)
// instead of five; the same error, being exact either way.
__device__ __forceinline__ void ordered_sum_acc(double& s, double& c, double v) {
    const bool swap = (__double2hiint(v) & 0x7fffffff) > (__double2hiint(s) & 0x7fffffff);
    const double a = swap ? v : s, b = swap ? s : v;
    const double t = __dadd_rn(a, b);
    c = __dadd_rn(c, __dadd_rn(b, -__dadd_rn(t, -a)));
    s = t;
}

// Pair at separation (dx, dy, dz): acceleration factor fac (times the
// separation and G) and potential pot (with G).
template <int LAW, bool ACC, bool POT>
__device__ __forceinline__ void pair64(double dx, double dy, double dz, double m, double G, double h,
                                       double h_inv, double h3_inv, double& fac, double& pot) {
    const double r2 = dx * dx + dy * dy + dz * dz;
    const double x = LAW == NB_LAW_PLUMMER ? r2 + h * h : r2;
    const double r = sqrt(x);
    // r >= h on the bit patterns: both are non-negative
    if (LAW == NB_LAW_PLUMMER || __double_as_longlong(r) >= __double_as_longlong(h)) {
        if (ACC) fac = m / (x * r);
        if (POT) pot = -m / r * G;
        if (LAW == NB_LAW_PLUMMER && POT && r2 == 0.0) pot = pot * 0.0;
        return;
    }
    const double u = r * h_inv;
    if (u < 0.5) {
        if (ACC) fac = m * h3_inv * (10.666666666667 + u * u * (32.0 * u - 38.4));
        if (POT) pot = m * h_inv * (-2.8 + u * u * (5.333333333333 + u * u * (6.4 * u - 9.6))) * G;
        if (POT && r == 0.0) pot = pot * 0.0;
    } else {
        if (ACC)
            fac = m * h3_inv *
                  (21.333333333333 - 48.0 * u + 38.4 * (u * u) - 10.666666666667 * (u * u * u) -
                   0.066666666667 / (u * u * u));
        if (POT)
            pot = m * h_inv *
                  (-3.2 + 0.066666666667 / u +
                   u * u * (10.666666666667 + u * (-16.0 + u * (9.6 - 2.133333333333 * u)))) *
                  G;
    }
}

// UNIT_G: G is exactly 1 (the default unit system), so the three products by it,
// which change no bit, are left out.
template <int LAW, bool ACC, bool POT, bool UNIT_G>
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
            const double dx = q.x - px, dy = q.y - py, dz = q.z - pz;
            double fac = 0.0, pot = 0.0;
            pair64<LAW, ACC, POT>(dx, dy, dz, q.w, G, h, h_inv, h3_inv, fac, pot);
            if (ACC) {
                ordered_sum_acc(sx, cx, UNIT_G ? dx * fac : dx * fac * G);
                ordered_sum_acc(sy, cy, UNIT_G ? dy * fac : dy * fac * G);
                ordered_sum_acc(sz, cz, UNIT_G ? dz * fac : dz * fac * G);
            }
            if (POT) ordered_sum_acc(sp, cp, pot);
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
// beside them, so a split evaluation keeps the accuracy of an unsplit one.  One
// thread per target over all parts, a serial chain on the FP64 pipe: at N = 2048
// (64 parts) 69 us beside a force of 331, with the potential 94 beside 407 (cold
// caches).
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
    const bool unit = G == 1.0;
#define NB_FP64(A, P)                                                                             \
    (unit ? k_force_fp64<LAW, A, P, true><<<(unsigned)grid, kTile, 0, s>>>(src, tg, G, partial)    \
          : k_force_fp64<LAW, A, P, false><<<(unsigned)grid, kTile, 0, s>>>(src, tg, G, partial))
    if (acc && pot)
        NB_FP64(true, true);
    else if (acc)
        NB_FP64(true, false);
    else if (pot)
        NB_FP64(false, true);
#undef NB_FP64
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
