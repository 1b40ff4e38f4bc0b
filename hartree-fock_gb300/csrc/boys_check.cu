// hfg_boys_eval: the device Boys function of the ERI kernels (boys.cuh), evaluated on an array of T values,
// for known-answer tests against the reference's Boys::calculateBoys (src/Boys.cpp:14-71) and the
// convergent series: the slice of the requested top order is staged in shared memory and boys_eval<L, Real> fills
// F_0 .. F_L, as in the FP32, warp, lane-group and store kernels.  hfg_boys_scaled does the same with scaled_boys<L>
// and the BoysFast slice, as in the FP64 thread, chunk and gradient kernels.
#include "boys.cuh"
#include "hfgpu.h"

#include <cuda_runtime.h>

#include <vector>

namespace
{
template <int L, typename Real>
__global__ void boys_eval_kernel(const double* __restrict__ T, long long n, const Real* __restrict__ slice_g,
                                 double* __restrict__ F)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Real* slice = reinterpret_cast<Real*>(smem_raw);
    constexpr int kVals = hfg::BoysGrid<Real>::kPoints * hfg::BoysGrid<Real>::kRow;
    for (int i = threadIdx.x; i < kVals; i += blockDim.x) slice[i] = slice_g[i];
    __syncthreads();
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x)
    {
        Real f[L + 1];
        hfg::boys_eval<L, Real>(static_cast<Real>(T[i]), slice, f);
#pragma unroll
        for (int m = 0; m <= L; ++m) F[i * (L + 1) + m] = static_cast<double>(f[m]);
    }
}

template <typename Real> cudaError_t launch_boys(int L, const double* T, long long n, const Real* slice, double* F)
{
    const size_t smem = sizeof(Real) * hfg::BoysGrid<Real>::kPoints * hfg::BoysGrid<Real>::kRow;
    const int blocks  = static_cast<int>(n / 256 + 1 < 1024 ? n / 256 + 1 : 1024);
    switch (L)
    {
#define HFG_BOYS_CASE(LL)                                                                                              \
    case LL: boys_eval_kernel<LL, Real><<<blocks, 256, smem>>>(T, n, slice, F); break;
        HFG_BOYS_CASE(0) HFG_BOYS_CASE(1) HFG_BOYS_CASE(2) HFG_BOYS_CASE(3) HFG_BOYS_CASE(4)
        HFG_BOYS_CASE(5) HFG_BOYS_CASE(6) HFG_BOYS_CASE(7) HFG_BOYS_CASE(8) HFG_BOYS_CASE(9)
#undef HFG_BOYS_CASE
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

template <int L>
__global__ void scaled_boys_kernel(const double* __restrict__ in, long long n, const double* __restrict__ slice_g,
                                   double* __restrict__ F)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* slice       = reinterpret_cast<double*>(smem_raw);
    constexpr int kVals = hfg::BoysFast::kPoints * hfg::BoysFast::kRow;
    for (int i = threadIdx.x; i < kVals; i += blockDim.x) slice[i] = slice_g[i];
    __syncthreads();
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x)
    {
        double f[L + 1];
        hfg::scaled_boys<L>(in[3 * i], in[3 * i + 1], in[3 * i + 2], slice, f);
#pragma unroll
        for (int m = 0; m <= L; ++m) F[i * (L + 1) + m] = f[m];
    }
}

cudaError_t launch_scaled_boys(int L, const double* in, long long n, const double* slice, double* F)
{
    const int smem   = static_cast<int>(sizeof(double)) * hfg::BoysFast::kPoints * hfg::BoysFast::kRow;
    const int blocks = static_cast<int>(n / 256 + 1 < 1024 ? n / 256 + 1 : 1024);
    auto go          = [&](auto kern) {
        const cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (err != cudaSuccess)
            return err;
        kern<<<blocks, 256, smem>>>(in, n, slice, F);
        return cudaGetLastError();
    };
    switch (L)
    {
#define HFG_BOYS_CASE(LL)                                                                                              \
    case LL: return go(scaled_boys_kernel<LL>);
        HFG_BOYS_CASE(0) HFG_BOYS_CASE(1) HFG_BOYS_CASE(2) HFG_BOYS_CASE(3) HFG_BOYS_CASE(4)
        HFG_BOYS_CASE(5) HFG_BOYS_CASE(6) HFG_BOYS_CASE(7) HFG_BOYS_CASE(8) HFG_BOYS_CASE(9)
#undef HFG_BOYS_CASE
    default: return cudaErrorInvalidValue;
    }
}

template <typename Real> int run(int device, int L, long long n, const double* T, double* F)
{
    if (cudaSetDevice(device) != cudaSuccess)
        return HFG_ERR_CUDA;
    const std::vector<Real> slice = hfg::boys_slice_host<Real>(L);
    double *dT = nullptr, *dF = nullptr;
    Real* dS   = nullptr;
    int rc     = HFG_OK;
    const size_t nF = static_cast<size_t>(n) * (L + 1);
    if (cudaMalloc(&dT, sizeof(double) * n) != cudaSuccess || cudaMalloc(&dF, sizeof(double) * nF) != cudaSuccess ||
        cudaMalloc(&dS, sizeof(Real) * slice.size()) != cudaSuccess)
        rc = HFG_ERR_NOMEM;
    if (rc == HFG_OK && (cudaMemcpy(dT, T, sizeof(double) * n, cudaMemcpyHostToDevice) != cudaSuccess ||
                         cudaMemcpy(dS, slice.data(), sizeof(Real) * slice.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
                         launch_boys<Real>(L, dT, n, dS, dF) != cudaSuccess ||
                         cudaMemcpy(F, dF, sizeof(double) * nF, cudaMemcpyDeviceToHost) != cudaSuccess))
        rc = HFG_ERR_CUDA;
    cudaFree(dT);
    cudaFree(dF);
    cudaFree(dS);
    return rc;
}
} // namespace

extern "C" int hfg_boys_eval(int device, int m_max, int fp32, long long n, const double* T, double* F)
{
    if (m_max < 0 || m_max > hfg::kMaxLt + 1 || n <= 0 || !T || !F)
        return HFG_ERR_INVALID;
    for (long long i = 0; i < n; ++i)
        if (!(T[i] >= 0.0) || !(T[i] < 1e300))
            return HFG_ERR_INVALID;
    return fp32 ? run<float>(device, m_max, n, T, F) : run<double>(device, m_max, n, T, F);
}

extern "C" int hfg_boys_scaled(int device, int m_max, long long n, const double* c_s_R2, double* F)
{
    if (m_max < 0 || m_max > hfg::kMaxLt + 1 || n <= 0 || !c_s_R2 || !F)
        return HFG_ERR_INVALID;
    for (long long i = 0; i < n; ++i)
    {
        const double c = c_s_R2[3 * i], s = c_s_R2[3 * i + 1], R2 = c_s_R2[3 * i + 2];
        if (!(c > -1e300 && c < 1e300) || !(s <= 0.0 && s > -1e30) || !(R2 >= 0.0 && R2 < 1e30))
            return HFG_ERR_INVALID;
    }
    if (cudaSetDevice(device) != cudaSuccess)
        return HFG_ERR_CUDA;
    const std::vector<double> slice = hfg::boys_fast_slices_host(m_max).back();
    const size_t nF = static_cast<size_t>(n) * (m_max + 1);
    double *dIn = nullptr, *dF = nullptr, *dS = nullptr;
    int rc = HFG_OK;
    if (cudaMalloc(&dIn, sizeof(double) * 3 * n) != cudaSuccess || cudaMalloc(&dF, sizeof(double) * nF) != cudaSuccess ||
        cudaMalloc(&dS, sizeof(double) * slice.size()) != cudaSuccess)
        rc = HFG_ERR_NOMEM;
    if (rc == HFG_OK && (cudaMemcpy(dIn, c_s_R2, sizeof(double) * 3 * n, cudaMemcpyHostToDevice) != cudaSuccess ||
                         cudaMemcpy(dS, slice.data(), sizeof(double) * slice.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
                         launch_scaled_boys(m_max, dIn, n, dS, dF) != cudaSuccess ||
                         cudaMemcpy(F, dF, sizeof(double) * nF, cudaMemcpyDeviceToHost) != cudaSuccess))
        rc = HFG_ERR_CUDA;
    cudaFree(dIn);
    cudaFree(dF);
    cudaFree(dS);
    return rc;
}
