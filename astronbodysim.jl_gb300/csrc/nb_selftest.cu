// nb_selftest.cu -- exercises the bounded-wait path that every mbarrier wait
// of the force kernels takes, without any fault: one warp waits on an
// mbarrier that nothing arrives on, gives up after the limit, records
// DEVERR_TIMEOUT in a device error word and returns.  The host reads the word;
// the context stays usable.
#include <cstdio>

#include "nb_force_mixed.cuh"

namespace {

__global__ void k_wait_nothing(uint64_t timeout_ns, uint32_t* err, unsigned long long* waited_ns) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        nb::mbar_init(&bar, 1);  // expects one arrival that never comes
        nb::fence_mbar_init();
    }
    __syncthreads();
    const uint64_t t0 = nb::globaltimer_ns();
    const bool ok = __all_sync(0xffffffffu, nb::mbar_wait_bounded(&bar, 0u, timeout_ns));
    if (threadIdx.x == 0) {
        *waited_ns = (unsigned long long)(nb::globaltimer_ns() - t0);
        if (!ok) atomicOr(err, nb::DEVERR_TIMEOUT);
    }
}

}  // namespace

extern "C" int nb_selftest_wait_timeout(int device, int64_t timeout_ns, double* waited_ms) {
    if (timeout_ns <= 0 || timeout_ns > 2000000000LL) return NB_ERR_INVALID_ARG;
    if (cudaSetDevice(device) != cudaSuccess) return NB_ERR_CUDA;
    void* mem = nullptr;
    if (cudaMalloc(&mem, 64) != cudaSuccess) return NB_ERR_OOM;
    uint32_t* err = static_cast<uint32_t*>(mem);
    unsigned long long* waited = reinterpret_cast<unsigned long long*>(static_cast<char*>(mem) + 8);
    cudaMemset(mem, 0, 64);
    k_wait_nothing<<<1, 32>>>((uint64_t)timeout_ns, err, waited);
    cudaError_t e = cudaDeviceSynchronize();
    uint32_t bits = 0;
    unsigned long long ns = 0;
    if (e == cudaSuccess) e = cudaMemcpy(&bits, err, sizeof bits, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&ns, waited, sizeof ns, cudaMemcpyDeviceToHost);
    cudaFree(mem);
    if (e != cudaSuccess) return NB_ERR_CUDA;
    if (waited_ms) *waited_ms = (double)ns * 1e-6;
    return (bits & nb::DEVERR_TIMEOUT) ? NB_ERR_TIMEOUT : NB_OK;
}

// ---------------------------------------------------------------------------
// FP32 throughput probe: the denominator of the force kernel's roofline,
// measured instead of assumed.  Every thread runs 8 independent dependency
// chains a = a * b + c (scalar fma.rn.f32, or packed fma.rn.f32x2 on float2),
// so the FMA pipe, not latency, bounds the rate.  Grid: 4 CTAs of 256 threads
// per SM.  The chains stay finite (|b| < 1); one thread stores a value that
// depends on every chain so nothing is dead code.
// ---------------------------------------------------------------------------
namespace {

constexpr int kPeakThreads = 256;
constexpr int kPeakChains = 8;

__global__ void __launch_bounds__(kPeakThreads) k_fma_scalar(int iters, float b, float c,
                                                              float* sink) {
    float a[kPeakChains];
#pragma unroll
    for (int k = 0; k < kPeakChains; ++k) a[k] = (float)(threadIdx.x + k) * 1e-3f;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int r = 0; r < 16; ++r) {
#pragma unroll
            for (int k = 0; k < kPeakChains; ++k) a[k] = __fmaf_rn(a[k], b, c);
        }
    }
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < kPeakChains; ++k) s += a[k];
    if (s == 12345.0f) *sink = s;  // never true for these inputs; keeps the chains live
}

__global__ void __launch_bounds__(kPeakThreads) k_fma_packed(int iters, float b, float c,
                                                              float* sink) {
    float2 a[kPeakChains];
    const float2 b2 = make_float2(b, b), c2 = make_float2(c, c);
#pragma unroll
    for (int k = 0; k < kPeakChains; ++k)
        a[k] = make_float2((float)(threadIdx.x + k) * 1e-3f, (float)(threadIdx.x - k) * 1e-3f);
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int r = 0; r < 16; ++r) {
#pragma unroll
            for (int k = 0; k < kPeakChains; ++k) a[k] = __ffma2_rn(a[k], b2, c2);
        }
    }
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < kPeakChains; ++k) s += a[k].x + a[k].y;
    if (s == 12345.0f) *sink = s;
}

}  // namespace

extern "C" int nb_selftest_fp32_peak(int device, int packed, double* tflops, double* ms) {
    if (cudaSetDevice(device) != cudaSuccess) return NB_ERR_CUDA;
    int nsm = 0;
    if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
        return NB_ERR_CUDA;
    float* sink = nullptr;
    if (cudaMalloc(&sink, sizeof(float)) != cudaSuccess) return NB_ERR_OOM;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int grid = 4 * nsm;
    const int iters = 4096;  // x 16 x 8 chains per thread
    const double lanes_per_op = packed ? 2.0 : 1.0;
    const double flop = 2.0 * lanes_per_op * (double)grid * kPeakThreads * iters * 16.0 * kPeakChains;
    float best = 1e30f;
    cudaError_t e = cudaSuccess;
    for (int rep = 0; rep < 6 && e == cudaSuccess; ++rep) {
        cudaEventRecord(e0);
        if (packed)
            k_fma_packed<<<grid, kPeakThreads>>>(iters, 0.9999f, 1e-4f, sink);
        else
            k_fma_scalar<<<grid, kPeakThreads>>>(iters, 0.9999f, 1e-4f, sink);
        cudaEventRecord(e1);
        e = cudaEventSynchronize(e1);
        float t = 0.0f;
        if (e == cudaSuccess) e = cudaEventElapsedTime(&t, e0, e1);
        if (rep > 0 && t < best) best = t;  // first launch is the warm-up
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(sink);
    if (e != cudaSuccess) return NB_ERR_CUDA;
    if (ms) *ms = best;
    if (tflops) *tflops = flop / (best * 1e-3) / 1e12;
    return NB_OK;
}

// ---------------------------------------------------------------------------
// Join of a block of 128 targets whose parts are one cluster, with sums that
// the host can add up, and one part that gives up (gave_up; none: -1).
// ---------------------------------------------------------------------------
namespace {

__global__ void __launch_bounds__(128) k_join_cluster(nb::Targets tg, int js, int gave_up) {
    __shared__ float sum[6 * 128];
    const int part = (int)blockIdx.x, t = (int)threadIdx.x;
    // (sum, carry) of this part per component: 2^part + t and (component + 1) 2^-40
    const float s[1] = {exp2f((float)part) + (float)t};
    const float c0[1] = {exp2f(-40.0f)}, c1[1] = {2.0f * c0[0]}, c2[1] = {3.0f * c0[0]};
    nb::cluster_join<128, 1>(sum, part == gave_up, js, part, 0, tg.n, s, c0, s, c1, s, c2, tg, 1.0);
}

}  // namespace

extern "C" int nb_selftest_cluster_join(int device, int parts, int gave_up, int n, double* acc, double* vel,
                                        double* t_float) {
    if (parts < 1 || parts > nb::kClusterParts || gave_up >= parts || n < 1 || n > 128 || !acc || !vel || !t_float)
        return NB_ERR_INVALID_ARG;
    if (cudaSetDevice(device) != cudaSuccess) return NB_ERR_CUDA;
    const size_t rows = sizeof(double) * 6 * 128;  // ax, ay, az, vx, vy, vz
    char* mem = nullptr;
    if (cudaMalloc(&mem, rows + sizeof(nb::Clock)) != cudaSuccess) return NB_ERR_OOM;
    double* row = reinterpret_cast<double*>(mem);
    nb::Targets tg{};
    tg.n = n;
    tg.ax = row;
    tg.ay = row + 128;
    tg.az = row + 2 * 128;
    tg.vx = row + 3 * 128;
    tg.vy = row + 4 * 128;
    tg.vz = row + 5 * 128;
    tg.kick_dt = 0.5;
    tg.step_clk = reinterpret_cast<nb::Clock*>(mem + rows);
    cudaMemset(mem, 0, rows + sizeof(nb::Clock));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)parts);
    cfg.blockDim = dim3(128);
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)parts;
    at.val.clusterDim.y = 1;
    at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, k_join_cluster, tg, parts, gave_up);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    nb::Clock c{};
    if (e == cudaSuccess) e = cudaMemcpy(acc, row, rows / 2, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(vel, row + 3 * 128, rows / 2, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&c, tg.step_clk, sizeof c, cudaMemcpyDeviceToHost);
    cudaFree(mem);
    if (e != cudaSuccess) return NB_ERR_CUDA;
    *t_float = c.t_float;
    return NB_OK;
}

extern "C" int nb_selftest_sort(int device, int64_t n, const uint64_t* keys, int passes, int chain, int32_t* perm) {
    if (n < 1 || n > (int64_t)1 << 24 || !keys || !perm || passes < 2 || passes > 8 || passes % 2)
        return NB_ERR_INVALID_ARG;
    if (cudaSetDevice(device) != cudaSuccess) return NB_ERR_CUDA;
    const size_t scratch = nb::sort_scratch_bytes(n);  // a multiple of 256
    char* mem = nullptr;
    if (cudaMalloc(&mem, scratch + sizeof(int32_t) * (size_t)n) != cudaSuccess) return NB_ERR_OOM;
    int32_t* vals = reinterpret_cast<int32_t*>(mem + scratch);
    for (int64_t i = 0; i < n; ++i) perm[i] = (int32_t)i;
    cudaError_t e = cudaMemcpy(vals, perm, sizeof(int32_t) * (size_t)n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(nb::sort_keys_buffer(mem, n), keys, sizeof(uint64_t) * (size_t)n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = nb::launch_sort_keys(mem, n, vals, passes, nullptr, chain != 0);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(perm, vals, sizeof(int32_t) * (size_t)n, cudaMemcpyDeviceToHost);
    cudaFree(mem);
    return e == cudaSuccess ? NB_OK : NB_ERR_CUDA;
}
