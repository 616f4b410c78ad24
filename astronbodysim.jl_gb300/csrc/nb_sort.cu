// nb_sort.cu -- spatial ordering of the sources for the mixed-precision force.
//
// The FP32 pair arithmetic works on coordinates relative to an FP64 origin per
// j-tile; its rounding error scales with the size of the tile.  Sorting the
// particles along a Morton (Z-order) curve makes every tile spatially compact,
// so close pairs are evaluated on small relative coordinates.
//
//   1. FP64 bounding box of all particles (two-stage min/max, deterministic);
//   2. 63-bit Morton key per particle (21 bits per axis over the box);
//   3. stable LSD radix sort of (key, index), 8-bit digits, 8 passes.
// The result is a deterministic permutation for given positions.
//
// The sort of up to kClusterSortMax keys is bound by latency: as a chain of
// kernels (histogram, scan, scatter per pass, 27 launches with the keys) it took
// 125 us at N = 4096 and 200 us at N = 65536.  It runs instead as one cluster
// of up to 16 CTAs whose shared memory holds all keys, passes separated by
// hardware cluster barriers, digit counts and keys exchanged through
// distributed shared memory (k_sort_cluster): 35 us at N = 4096, 86 us at
// N = 65536, 143 us (277 as a chain) at N = 131072.  Larger sorts, bound by their
// passes over memory, and GPUs without room for the cluster keep the chain:
// per-block digit histograms -> one exclusive scan -> stable scatter that ranks
// equal digits by (round, warp, lane) order.
#include <cooperative_groups.h>

#include "nb_internal.cuh"

namespace nb {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;  // per thread
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;
constexpr int kWarps = kSortThreads / 32;
constexpr int kBboxBlocks = 64;
constexpr int kBboxThreads = 512;
constexpr int kMortonThreads = 64;  // small CTAs: the FP64 divisions of a small system over many SMs

int64_t sort_blocks(int64_t n) { return (n + kSortTile - 1) / kSortTile; }
int64_t scan_tmp_words(int64_t len);
cudaError_t launch_exclusive_scan2(uint32_t* counts, int64_t len, uint32_t* tmp, cudaStream_t s);

// Scratch layout (bytes) for n particles.
size_t sort_scratch_bytes(int64_t n) {
    const int64_t nb = sort_blocks(n);
    auto al = [](size_t v) { return (v + 255) / 256 * 256; };
    return al(sizeof(uint64_t) * n) * 2 + al(sizeof(int32_t) * n) +
           al(sizeof(uint32_t) * (size_t)kRadix * nb) +
           al(sizeof(unsigned long long) * 6 * kBboxBlocks) + al(sizeof(uint32_t) * (size_t)scan_tmp_words(kRadix * nb));
}

struct SortScratch {
    uint64_t* keys_a;
    uint64_t* keys_b;
    int32_t* vals_b;
    uint32_t* counts;
    unsigned long long* bbox_part;
    uint32_t* scan_tmp;
};

static SortScratch carve(void* base, int64_t n) {
    auto al = [](size_t v) { return (v + 255) / 256 * 256; };
    char* p = static_cast<char*>(base);
    SortScratch s;
    s.keys_a = (uint64_t*)p;
    p += al(sizeof(uint64_t) * n);
    s.keys_b = (uint64_t*)p;
    p += al(sizeof(uint64_t) * n);
    s.vals_b = (int32_t*)p;
    p += al(sizeof(int32_t) * n);
    s.counts = (uint32_t*)p;
    p += al(sizeof(uint32_t) * (size_t)kRadix * sort_blocks(n));
    s.bbox_part = (unsigned long long*)p;
    p += al(sizeof(unsigned long long) * 6 * kBboxBlocks);
    s.scan_tmp = (uint32_t*)p;
    return s;
}

// Order-preserving unsigned image of a double; a NaN never wins the minimum.
// The box is reduced on these images, off the slow FP64 pipe.
__device__ __forceinline__ unsigned long long ord_image(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return v != v ? ~0ull : (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double ord_double(unsigned long long k) {
    return __longlong_as_double((long long)((k >> 63) ? (k & 0x7fffffffffffffffull) : ~k));
}
// The warp's minima of v[0..5].
__device__ __forceinline__ void warp_min6(unsigned long long* v) {
#pragma unroll
    for (int k = 0; k < 6; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] = min(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
}

// Minima of x, y, z, -x, -y, -z over each block's particles, as images.
__global__ void __launch_bounds__(kBboxThreads)
    k_bbox_partial(const double* __restrict__ x, const double* __restrict__ y,
                   const double* __restrict__ z, int64_t n, unsigned long long* __restrict__ part) {
    __shared__ unsigned long long red[6][kBboxThreads / 32];
    const unsigned long long big = ord_image(1e300);
    unsigned long long v[6] = {big, big, big, big, big, big};
    for (int64_t i = (int64_t)blockIdx.x * kBboxThreads + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * kBboxThreads) {
        const double a = x[i], b = y[i], c = z[i];
        v[0] = min(v[0], ord_image(a));
        v[1] = min(v[1], ord_image(b));
        v[2] = min(v[2], ord_image(c));
        v[3] = min(v[3], ord_image(-a));
        v[4] = min(v[4], ord_image(-b));
        v[5] = min(v[5], ord_image(-c));
    }
    warp_min6(v);
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int k = 0; k < 6; ++k) red[k][threadIdx.x >> 5] = v[k];
    __syncthreads();
    if (threadIdx.x < 6) {
        unsigned long long r = red[threadIdx.x][0];
        for (int w = 1; w < kBboxThreads / 32; ++w) r = min(r, red[threadIdx.x][w]);
        part[blockIdx.x * 6 + threadIdx.x] = r;
    }
}

__device__ __forceinline__ uint64_t spread3_21(uint64_t v) {
    v &= 0x1fffffull;
    v = (v | (v << 32)) & 0x1f00000000ffffull;
    v = (v | (v << 16)) & 0x1f0000ff0000ffull;
    v = (v | (v << 8)) & 0x100f00f00f00f00full;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}

// Keys of all particles; every block joins the nblocks partial boxes for itself.
__global__ void __launch_bounds__(kMortonThreads)
    k_morton(const double* __restrict__ x, const double* __restrict__ y,
             const double* __restrict__ z, int64_t n, const unsigned long long* __restrict__ part,
             int nblocks, uint64_t* __restrict__ keys, int32_t* __restrict__ vals) {
    __shared__ unsigned long long red[6][kMortonThreads / 32];
    const unsigned long long big = ord_image(1e300);
    unsigned long long v[6] = {big, big, big, big, big, big};
    for (int b = threadIdx.x; b < nblocks; b += kMortonThreads)
#pragma unroll
        for (int k = 0; k < 6; ++k) v[k] = min(v[k], part[b * 6 + k]);
    warp_min6(v);
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int k = 0; k < 6; ++k) red[k][threadIdx.x >> 5] = v[k];
    __syncthreads();
    const int64_t i = (int64_t)blockIdx.x * kMortonThreads + threadIdx.x;
    if (i >= n) return;
    double lo[3], hi[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        lo[k] = ord_double(min(red[k][0], red[k][1]));
        hi[k] = -ord_double(min(red[k + 3][0], red[k + 3][1]));
    }
    static_assert(kMortonThreads == 64, "two warps' minima");
    const double p[3] = {x[i], y[i], z[i]};
    uint64_t q[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double ext = hi[k] - lo[k];
        double f = ext > 0.0 ? (p[k] - lo[k]) / ext : 0.0;
        f = fmin(fmax(f, 0.0), 1.0);
        q[k] = (uint64_t)(f * 2097151.0);
    }
    keys[i] = spread3_21(q[0]) | (spread3_21(q[1]) << 1) | (spread3_21(q[2]) << 2);
    vals[i] = (int32_t)i;
}

__global__ void __launch_bounds__(kSortThreads)
    k_radix_hist(const uint64_t* __restrict__ keys, int64_t n, int shift, int nblocks,
                 uint32_t* __restrict__ counts) {
    __shared__ uint32_t h[kRadix];
    h[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kSortTile;
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const int64_t i = base + r * kSortThreads + threadIdx.x;
        if (i < n) atomicAdd(&h[(keys[i] >> shift) & (kRadix - 1)], 1u);
    }
    __syncthreads();
    counts[(int64_t)threadIdx.x * nblocks + blockIdx.x] = h[threadIdx.x];
}

// Exclusive scan of len counts with one block of 1024 threads.
__global__ void __launch_bounds__(1024) k_scan(uint32_t* __restrict__ c, int64_t len) {
    __shared__ uint32_t part[1024];
    const int64_t per = (len + 1023) / 1024;
    const int64_t b = threadIdx.x * per;
    const int64_t e = min(len, b + per);
    uint32_t s = 0;
    for (int64_t i = b; i < e; ++i) s += c[i];
    part[threadIdx.x] = s;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        uint32_t v = threadIdx.x >= o ? part[threadIdx.x - o] : 0u;
        __syncthreads();
        part[threadIdx.x] += v;
        __syncthreads();
    }
    uint32_t run = part[threadIdx.x] - s;  // exclusive
    for (int64_t i = b; i < e; ++i) {
        const uint32_t v = c[i];
        c[i] = run;
        run += v;
    }
}

__global__ void __launch_bounds__(kSortThreads)
    k_radix_scatter(const uint64_t* __restrict__ kin, const int32_t* __restrict__ vin,
                    uint64_t* __restrict__ kout, int32_t* __restrict__ vout, int64_t n, int shift,
                    int nblocks, const uint32_t* __restrict__ offs) {
    __shared__ uint32_t wcnt[kWarps][kRadix + 1];
    __shared__ uint32_t wbase[kWarps][kRadix + 1];
    __shared__ uint32_t run[kRadix];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    run[tid] = offs[(int64_t)tid * nblocks + blockIdx.x];
    for (int w = 0; w < kWarps; ++w) wcnt[w][tid] = 0;
    if (tid < kWarps) wcnt[tid][kRadix] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kSortTile;
    const uint32_t lt = (1u << lane) - 1u;
    for (int r = 0; r < kSortItems; ++r) {
        const int64_t i = base + r * kSortThreads + tid;
        const bool valid = i < n;
        uint64_t key = 0;
        int32_t val = 0;
        uint32_t d = kRadix;  // sentinel bin for lanes past the end
        if (valid) {
            key = kin[i];
            val = vin ? vin[i] : (int32_t)i;
            d = (uint32_t)((key >> shift) & (kRadix - 1));
        }
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        const uint32_t rank = __popc(peers & lt);
        if (lane == __ffs(peers) - 1) wcnt[warp][d] = __popc(peers);
        __syncthreads();
        {
            uint32_t acc = run[tid];
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                const uint32_t c = wcnt[w][tid];
                wbase[w][tid] = acc;
                acc += c;
                wcnt[w][tid] = 0;
            }
            run[tid] = acc;
        }
        __syncthreads();
        if (valid) {
            const uint32_t pos = wbase[warp][d] + rank;
            kout[pos] = key;
            vout[pos] = val;
        }
        if (tid < kWarps) wcnt[tid][kRadix] = 0;
        __syncthreads();
    }
}

// Multi-CTA exclusive scan for long arrays: each CTA sums a chunk of
// kScanChunk counts, one CTA scans the chunk sums, each CTA rescans its chunk
// from its offset.
constexpr int kScanThreads = 256;
constexpr int kScanPer = 16;
constexpr int kScanChunk = kScanThreads * kScanPer;
constexpr int64_t kScanMaxChunks = 1024;  // chunk sums scanned by one k_scan CTA

__global__ void __launch_bounds__(kScanThreads)
    k_scan_chunk_sums(const uint32_t* __restrict__ c, int64_t len, uint32_t* __restrict__ sums) {
    const int64_t b = (int64_t)blockIdx.x * kScanChunk;
    uint32_t s = 0;
    for (int i = threadIdx.x; i < kScanChunk; i += kScanThreads) {
        const int64_t j = b + i;
        if (j < len) s += c[j];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __shared__ uint32_t w[kScanThreads / 32];
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int k = 0; k < kScanThreads / 32; ++k) t += w[k];
        sums[blockIdx.x] = t;
    }
}

__global__ void __launch_bounds__(kScanThreads)
    k_scan_chunk_apply(uint32_t* __restrict__ c, int64_t len, const uint32_t* __restrict__ offs) {
    __shared__ uint32_t part[kScanThreads];
    const int64_t b = (int64_t)blockIdx.x * kScanChunk + (int64_t)threadIdx.x * kScanPer;
    uint32_t v[kScanPer];
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
        const int64_t j = b + k;
        v[k] = j < len ? c[j] : 0u;
        s += v[k];
    }
    part[threadIdx.x] = s;
    __syncthreads();
    for (int o = 1; o < kScanThreads; o <<= 1) {
        const uint32_t t = threadIdx.x >= o ? part[threadIdx.x - o] : 0u;
        __syncthreads();
        part[threadIdx.x] += t;
        __syncthreads();
    }
    uint32_t run = offs[blockIdx.x] + part[threadIdx.x] - s;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
        const int64_t j = b + k;
        if (j < len) c[j] = run;
        run += v[k];
    }
}

// Exclusive prefix sum of len 32-bit counts in place.  `tmp` (may be null for
// len <= kScanChunk * 4) holds scan_tmp_words(len) words.
int64_t scan_tmp_words(int64_t len) { return (len + kScanChunk - 1) / kScanChunk + 1; }

cudaError_t launch_exclusive_scan2(uint32_t* counts, int64_t len, uint32_t* tmp, cudaStream_t s) {
    if (len <= 0) return cudaSuccess;
    const int64_t nchunks = (len + kScanChunk - 1) / kScanChunk;
    if (!tmp || nchunks <= 4 || nchunks > kScanMaxChunks * kScanChunk) {
        k_scan<<<1, 1024, 0, s>>>(counts, len);
        return cudaGetLastError();
    }
    k_scan_chunk_sums<<<(unsigned)nchunks, kScanThreads, 0, s>>>(counts, len, tmp);
    k_scan<<<1, 1024, 0, s>>>(tmp, nchunks);
    k_scan_chunk_apply<<<(unsigned)nchunks, kScanThreads, 0, s>>>(counts, len, tmp);
    return cudaGetLastError();
}

// Exclusive prefix sum of len 32-bit counts in place (one CTA of 1024 threads).
cudaError_t launch_exclusive_scan(uint32_t* counts, int64_t len, cudaStream_t s) {
    if (len <= 0) return cudaSuccess;
    k_scan<<<1, 1024, 0, s>>>(counts, len);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Radix sort in one cluster.  CTA c of C holds positions [c M, (c + 1) M) of
// the current order, M = THREADS * ITEMS, in shared memory (keys and values,
// double-buffered).  A pass:
//   * every warp ranks its 32 * ITEMS consecutive keys by digit, in order
//     (votes per round, running counts per warp and digit), and the CTA
//     turns the warps' counts into offsets and publishes its digit counts;
//   * after a cluster barrier each CTA reads all CTAs' counts, which gives
//     the first position of each of its digits in the whole order;
//   * keys and values are put in digit order within the CTA, so that a warp
//     then writes a few runs and not 32 scattered words to their positions in
//     the other buffers of the CTAs that own them (distributed shared memory);
//     cluster barrier.
// Stable, so the permutation is the same as that of the chain of kernels.
// Positions past n are not stored; only the last CTAs have such.
// ---------------------------------------------------------------------------
constexpr int kCsMaxCluster = 16;
constexpr int64_t kClusterSortMax = (int64_t)kCsMaxCluster * 1024 * 8;

template <int THREADS, int ITEMS>
struct CsShared {
    uint64_t key[2][THREADS * ITEMS];
    int32_t val[2][THREADS * ITEMS];
    uint16_t cnt[THREADS / 32][kRadix];  // per warp: counts, then offsets within the CTA (< 2^16)
    uint32_t total[kRadix];          // this CTA's digit counts, read by the others
    uint32_t base[kRadix];           // first position of each of its digits
    uint32_t start[kRadix];          // first of each digit among this CTA's own keys in digit order
    uint32_t wsum[2][kRadix / 32];
};

// The lanes with this lane's digit, among the valid ones.  A vote per bit beats
// match_any here; with the runs above it took a sort of 65536 from 106 to 86 us,
// of 131072 from 172 to 143 us, of 30000 from 69 to 61 us.
__device__ __forceinline__ uint32_t same_digit(uint32_t d, bool valid) {
    uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (int b = 0; b < kRadixBits; ++b) {
        const bool bit = (d >> b) & 1u;
        const uint32_t v = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? v : ~v;
    }
    return peers;
}

template <int THREADS, int ITEMS>
__global__ void __launch_bounds__(THREADS)
    k_sort_cluster(const uint64_t* __restrict__ keys, int32_t* __restrict__ vals, int n, int passes) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char cs_raw[];
    using Shared = CsShared<THREADS, ITEMS>;
    Shared& sh = *reinterpret_cast<Shared*>(cs_raw);
    cg::cluster_group cluster = cg::this_cluster();
    constexpr int M = THREADS * ITEMS, kWarpsOf = THREADS / 32;
    const int C = (int)cluster.num_blocks(), c = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int first = c * M, count = min(M, max(0, n - first));  // keys this CTA holds
    for (int i = tid; i < count; i += THREADS) {
        sh.key[0][i] = keys[first + i];
        sh.val[0][i] = vals[first + i];
    }
    // every CTA of the cluster runs before any of them writes into another
    cluster.sync();
    for (int pass = 0; pass < passes; ++pass) {
        const int src = pass & 1, shift = pass * kRadixBits;
        for (int d = lane; d < kRadix; d += 32) sh.cnt[warp][d] = 0;
        __syncwarp();
        uint64_t key[ITEMS];
        int32_t val[ITEMS];
        uint32_t rank[ITEMS];
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) {
            const int i = warp * 32 * ITEMS + r * 32 + lane;
            const bool valid = i < count;
            key[r] = valid ? sh.key[src][i] : 0ull;
            val[r] = valid ? sh.val[src][i] : 0;
            const uint32_t d = (uint32_t)(key[r] >> shift) & (kRadix - 1);
            const uint32_t peers = same_digit(d, valid);
            const uint32_t before = __popc(peers & ((1u << lane) - 1u));
            rank[r] = valid ? sh.cnt[warp][d] + before : 0u;
            __syncwarp();
            if (valid && before == 0u) sh.cnt[warp][d] += (uint16_t)__popc(peers);
            __syncwarp();
        }
        __syncthreads();
        if (tid < kRadix) {
            uint32_t run = 0;
#pragma unroll
            for (int w = 0; w < kWarpsOf; ++w) {
                const uint32_t v = sh.cnt[w][tid];
                sh.cnt[w][tid] = (uint16_t)run;
                run += v;
            }
            sh.total[tid] = run;
        }
        cluster.sync();
        uint32_t all = 0, prev = 0, own = 0, incl = 0, iown = 0;
        if (tid < kRadix) {
            own = sh.total[tid];
#pragma unroll 8
            for (int k = 0; k < C; ++k) {
                const uint32_t v = *cluster.map_shared_rank(&sh.total[tid], k);
                all += v;
                prev += k < c ? v : 0u;
            }
            incl = all;
            iown = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                const uint32_t u = __shfl_up_sync(0xffffffffu, iown, o);
                if (lane >= o) {
                    incl += v;
                    iown += u;
                }
            }
            if (lane == 31) {
                sh.wsum[0][warp] = incl;
                sh.wsum[1][warp] = iown;
            }
        }
        __syncthreads();
        if (tid < kRadix) {
            uint32_t b = incl - all + prev, l = iown - own;
            for (int w = 0; w < warp; ++w) {
                b += sh.wsum[0][w];
                l += sh.wsum[1][w];
            }
            sh.base[tid] = b;
            sh.start[tid] = l;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) {
            const int i = warp * 32 * ITEMS + r * 32 + lane;
            if (i < count) {
                const uint32_t d = (uint32_t)(key[r] >> shift) & (kRadix - 1);
                const uint32_t at = sh.start[d] + sh.cnt[warp][d] + rank[r];
                sh.key[src][at] = key[r];
                sh.val[src][at] = val[r];
            }
        }
        __syncthreads();
        for (int i = tid; i < count; i += THREADS) {
            const uint64_t k = sh.key[src][i];
            const uint32_t d = (uint32_t)(k >> shift) & (kRadix - 1);
            const uint32_t pos = sh.base[d] + ((uint32_t)i - sh.start[d]);
            const int to = (int)(pos / M), at = (int)(pos % M);
            *cluster.map_shared_rank(&sh.key[src ^ 1][at], to) = k;
            *cluster.map_shared_rank(&sh.val[src ^ 1][at], to) = sh.val[src][i];
        }
        // all keys have arrived; also the last read of total, and of a CTA's
        // shared memory by another, before it is written again or given up
        cluster.sync();
    }
    for (int i = tid; i < count; i += THREADS) vals[first + i] = sh.val[passes & 1][i];
}

// Launches the cluster sort of n <= C * THREADS * ITEMS keys; *done false:
// this GPU cannot hold the cluster (nothing was launched).
template <int THREADS, int ITEMS>
static cudaError_t launch_cluster(const uint64_t* keys, int32_t* vals, int64_t n, int passes, bool* done,
                                  cudaStream_t s) {
    auto kern = k_sort_cluster<THREADS, ITEMS>;
    constexpr size_t smem = sizeof(CsShared<THREADS, ITEMS>);
    static_assert(smem <= 232448, "227 KB of shared memory per CTA");
    int C = 1;
    while ((int64_t)C * THREADS * ITEMS < n) C *= 2;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && C > 8)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)C);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)C;
    at.val.clusterDim.y = 1;
    at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg);
    if (e != cudaSuccess || clusters < 1) {
        (void)cudaGetLastError();
        *done = false;
        return cudaSuccess;
    }
    *done = true;
    return cudaLaunchKernelEx(&cfg, kern, keys, vals, (int)n, passes);
}

// As many CTAs as give each at least 512 keys, up to the 16 of a cluster, then
// more threads, then more keys per thread.
static cudaError_t launch_cluster_sort(const uint64_t* keys, int32_t* vals, int64_t n, int passes,
                                       bool* done, cudaStream_t s) {
    *done = false;
    if (n > kClusterSortMax) return cudaSuccess;
    const int64_t per = (n + kCsMaxCluster - 1) / kCsMaxCluster;  // keys per CTA of the largest cluster
    if (per <= 512) return launch_cluster<512, 1>(keys, vals, n, passes, done, s);
    if (per <= 1024) return launch_cluster<1024, 1>(keys, vals, n, passes, done, s);
    if (per <= 2048) return launch_cluster<1024, 2>(keys, vals, n, passes, done, s);
    if (per <= 4096) return launch_cluster<1024, 4>(keys, vals, n, passes, done, s);
    return launch_cluster<1024, 8>(keys, vals, n, passes, done, s);
}

// Key buffer inside a sort scratch of sort_scratch_bytes(n) bytes.
uint64_t* sort_keys_buffer(void* scratch, int64_t n) { return carve(scratch, n).keys_a; }

// Stable LSD radix sort of (keys, vals): keys in sort_keys_buffer(scratch, n),
// vals (n int32) in place; `passes` 8-bit digits from the bottom (even).  chain:
// without the cluster sort.
cudaError_t launch_sort_keys(void* scratch, int64_t n, int32_t* vals, int passes, cudaStream_t s, bool chain) {
    if (n <= 0) return cudaSuccess;
    SortScratch sc = carve(scratch, n);
    bool done = false;
    cudaError_t e = chain ? cudaSuccess : launch_cluster_sort(sc.keys_a, vals, n, passes, &done, s);
    if (e != cudaSuccess || done) return e;
    const int nblocks = (int)sort_blocks(n);
    uint64_t* kin = sc.keys_a;
    uint64_t* kout = sc.keys_b;
    int32_t* vin = vals;
    int32_t* vout = sc.vals_b;
    for (int pass = 0; pass < passes; ++pass) {
        const int shift = pass * kRadixBits;
        k_radix_hist<<<nblocks, kSortThreads, 0, s>>>(kin, n, shift, nblocks, sc.counts);
        e = launch_exclusive_scan2(sc.counts, (int64_t)kRadix * nblocks, sc.scan_tmp, s);
        if (e != cudaSuccess) return e;
        k_radix_scatter<<<nblocks, kSortThreads, 0, s>>>(kin, vin, kout, vout, n, shift, nblocks,
                                                         sc.counts);
        uint64_t* tk = kin;
        kin = kout;
        kout = tk;
        int32_t* tv = vin;
        vin = vout;
        vout = tv;
    }
    // After an even number of passes the sorted values are back in vals.
    return cudaGetLastError();
}

// Computes perm[0..n) = particle indices in Morton order of (x, y, z).
cudaError_t launch_morton_sort(const double* x, const double* y, const double* z, int64_t n,
                               void* scratch, int32_t* perm, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    SortScratch sc = carve(scratch, n);
    const int64_t gb = (n + kBboxThreads - 1) / kBboxThreads;
    const int bb = (int)(gb < kBboxBlocks ? gb : kBboxBlocks);
    k_bbox_partial<<<bb, kBboxThreads, 0, s>>>(x, y, z, n, sc.bbox_part);
    k_morton<<<(unsigned)((n + kMortonThreads - 1) / kMortonThreads), kMortonThreads, 0, s>>>(
        x, y, z, n, sc.bbox_part, bb, sc.keys_a, perm);
    return launch_sort_keys(scratch, n, perm, 8, s);
}

}  // namespace nb
