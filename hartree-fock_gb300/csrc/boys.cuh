// Boys function F_m(T) for the ERI kernels.
//
// Same scheme as the reference (src/Boys.cpp:14-71, after Weiss & Ochsenfeld, J. Comput. Chem. 36,
// 1390 (2015)): tabulate F_m on a uniform T grid, obtain F at an off-grid T by a Taylor expansion
// about a grid point using dF_m/dT = -F_{m+1}, then fill the lower orders by recursion; for T > 30 the
// asymptotic form F_0 = sqrt(pi/T)/2, F_{m+1} = (m+1/2) F_m / T.
//
// GB300 adaptation: the reference's grid (600,001 points x 34 orders of FP64 = 163 MB, 3 Taylor
// terms) cannot live in shared memory.  Here each kernel stages a class-specific slice in shared
// memory: only the K orders F_L .. F_{L+K-1} that the Taylor expansion of the top order needs (lower
// orders come from the downward recursion F_{m-1} = (2T F_m + e^{-T}) / (2m-1), stable for all T), each
// pre-divided by k!, plus e^{-T_i} so that e^{-T} = e^{-T_i} e^{-d} needs only a short series:
//
//            step h   Taylor terms K   points        slice size (L fixed)
//   FP64     0.05     7                601 (+1)      602 x 8 doubles = 38.5 KB
//   FP32     0.10     5                301 (+1)      302 x 6 floats  =  7.2 KB
//
// Nearest-point expansion keeps |d| <= h/2, so the truncation error is below (h/2)^K / K! relative:
// 1.2e-15 (FP64) and 2.6e-9 (FP32).
//
// The FP64 kernels that compute these scalars once per lane (the thread and chunk forms, the gradient) are
// bound by the FP64 pipe, where a warp instruction takes 16 cycles of the SM, and use a third slice with
// shorter polynomials (BoysFast below): Taylor polynomials of degree 13 economised by taking off their leading
// Chebyshev polynomials one by one (Lanczos 1938), six coefficients for F_L and seven for e^d:
//
//   FP64     1/32     6         962 points    962 x 7 doubles = 53.9 KB    (h/2)^6 / (2^5 6!) = 6.3e-16
//
// F_L and e^{-T} together take 11 DFMA instead of 13, the grid point is found in FP32, and the downward
// recursion runs on values that carry the prefactor already (scaled_boys); over T in [0, 30] its largest
// relative error against a long-double series is 4.0e-16 / 1.2e-15 / 1.8e-15 for L = 1 / 4 / 9, that of
// boys_eval times the prefactor powers 4.7e-16 / 1.2e-15 / 2.1e-15.  The other forms keep the smaller slice.
#pragma once

#include "hfg_common.cuh"

#include <cmath>
#include <vector>

namespace hfg
{
template <typename Real> struct BoysGrid;
template <> struct BoysGrid<double>
{
    static constexpr double kStep    = 0.05;
    static constexpr double kInvStep = 20.0;
    static constexpr int kTerms      = 7;
    static constexpr int kPoints     = 602;
    static constexpr int kRow        = kTerms + 1; // K scaled orders + e^{-T_i}
};
template <> struct BoysGrid<float>
{
    static constexpr double kStep    = 0.1;
    static constexpr double kInvStep = 10.0;
    static constexpr int kTerms      = 5;
    static constexpr int kPoints     = 302;
    static constexpr int kRow        = kTerms + 1;
};
constexpr double kBoysAsymptotic = 30.0;
constexpr double kSqrtPiBy2      = 0.88622692545275801365; // sqrt(pi)/2

// Host: F_m(T) from the convergent series F_m(T) = e^{-T}/2 * sum_i T^i / ((m+1/2)(m+3/2)...(m+i+1/2)),
// summed in long double until the terms stop changing the sum.
inline long double boys_series_host(int m, long double T)
{
    long double term = 1.0L / (m + 0.5L), sum = term;
    for (int i = 1; i < 2000; ++i)
    {
        term *= T / (m + i + 0.5L);
        const long double s2 = sum + term;
        if (s2 == sum)
            break;
        sum = s2;
    }
    return sum * std::exp(-T) / 2.0L;
}

// Host: the slice a class of total angular momentum L needs, row-major [point][kRow].
template <typename Real> std::vector<Real> boys_slice_host(int L)
{
    using G = BoysGrid<Real>;
    std::vector<Real> out(static_cast<size_t>(G::kPoints) * G::kRow);
    for (int i = 0; i < G::kPoints; ++i)
    {
        const long double Ti = i * static_cast<long double>(G::kStep);
        long double kfact    = 1.0L;
        for (int k = 0; k < G::kTerms; ++k)
        {
            if (k > 0)
                kfact *= k;
            out[static_cast<size_t>(i) * G::kRow + k] = static_cast<Real>(boys_series_host(L + k, Ti) / kfact);
        }
        out[static_cast<size_t>(i) * G::kRow + G::kTerms] = static_cast<Real>(std::exp(-Ti));
    }
    return out;
}

// 1/k! for the e^x series.
__host__ __device__ constexpr double inv_fact(int k)
{
    double f = 1.0;
    for (int i = 2; i <= k; ++i) f *= i;
    return 1.0 / f;
}
// y = t + magic rounds t to an integer held in the low bits of y: 1.5 * 2^52 (double), 1.5 * 2^23 (float).
template <typename Real> constexpr double kRoundMagic = 0.0;
template <> constexpr double kRoundMagic<double> = 6755399441055744.0;
template <> constexpr double kRoundMagic<float>  = 12582912.0;
template <typename Real> constexpr int kRoundMagicLow = 0;
template <> constexpr int kRoundMagicLow<double> = 0;          // low 32 bits of 1.5*2^52 are zero
template <> constexpr int kRoundMagicLow<float>  = 0x400000;   // mantissa of 1.5*2^23

// The grid of scaled_boys.
struct BoysFast
{
    static constexpr double kStep    = 0.03125;
    static constexpr double kInvStep = 32.0;
    static constexpr int kTerms      = 6;
    static constexpr int kPoints     = 962;
    static constexpr int kRow        = kTerms + 1; // coefficients + e^{-T_i}; odd, so rows spread over the banks
};

// Economises a polynomial c[0..n) in x on |x| <= r to its first `keep` coefficients (constexpr: also the
// coefficients of e^x below).  T_k(x/r) / 2^{k-1} scaled to leading coefficient 1 is subtracted from the top.
constexpr void economise(double* c, int n, int keep, double r)
{
    using F = double;
    for (int k = n - 1; k >= keep; --k)
    {
        // Chebyshev coefficients of T_k by T_{j+1} = 2 x T_j - T_{j-1}.
        F a[24] {}, b[24] {};
        a[0] = F(1);
        b[1] = F(1);
        for (int j = 1; j < k; ++j)
        {
            F t[24] {};
            for (int i = 0; i <= j; ++i) t[i + 1] = F(2) * b[i];
            for (int i = 0; i <= j; ++i) t[i] -= a[i];
            for (int i = 0; i <= j + 1; ++i)
            {
                a[i] = b[i];
                b[i] = t[i];
            }
        }
        const F top = c[k];
        F rk        = F(1); // r^(k - i)
        for (int i = k; i >= 0; --i, rk *= r) c[i] -= top * rk * b[i] / b[k];
    }
}

// Coefficient k of the economised e^x on |x| <= h/2; one more than F_L has, because e^x has
// nothing like F_{L+6}/F_L <= 1/13 in its error term (6.3e-16 with six, 1e-18 with seven).
constexpr int kExpTerms = BoysFast::kTerms + 1;
constexpr double exp_coefficient(int k)
{
    double c[14] {};
    for (int i = 0; i < 14; ++i) c[i] = inv_fact(i);
    economise(c, 14, kExpTerms, BoysFast::kStep / 2);
    return c[k];
}
template <int K> constexpr double kExpCoefficient = exp_coefficient(K);

// Host: the BoysFast slices of total angular momentum 0 .. l_max, each row-major [point][kRow].
inline std::vector<std::vector<double>> boys_fast_slices_host(int l_max)
{
    using G               = BoysFast;
    constexpr int kTaylor = 14;
    std::vector<std::vector<double>> out(l_max + 1, std::vector<double>(static_cast<size_t>(G::kPoints) * G::kRow));
    double eco[kTaylor][kTaylor] {}; // what economising moves from coefficient k to the lower ones
    for (int k = G::kTerms; k < kTaylor; ++k)
    {
        eco[k][k] = 1.0;
        economise(eco[k], kTaylor, G::kTerms, G::kStep / 2);
    }
    std::vector<long double> F(l_max + kTaylor);
    for (int i = 0; i < G::kPoints; ++i)
    {
        // All orders from the highest by the downward recursion (one series per point: long double is slow software
        // on some hosts), then per slice the Taylor coefficients F_{L+k} / k!.
        const long double Ti = i * static_cast<long double>(G::kStep), e = std::exp(-Ti);
        const int top = l_max + kTaylor - 1;
        F[top]        = boys_series_host(top, Ti);
        for (int m = top; m > 0; --m) F[m - 1] = (2 * Ti * F[m] + e) / (2 * m - 1);
        for (int L = 0; L <= l_max; ++L)
        {
            double* row = &out[L][static_cast<size_t>(i) * G::kRow];
            double moved[G::kTerms] {};
            for (int k = kTaylor - 1; k >= G::kTerms; --k)
                for (int j = 0; j < G::kTerms; ++j) moved[j] += static_cast<double>(F[L + k]) * inv_fact(k) * eco[k][j];
            long double kfact = 1.0L;
            for (int j = 0; j < G::kTerms; ++j)
            {
                if (j > 1)
                    kfact *= j;
                row[j] = static_cast<double>(F[L + j] / kfact + moved[j]);
            }
            row[G::kTerms] = static_cast<double>(e);
        }
    }
    return out;
}

#ifdef __CUDACC__
__device__ __forceinline__ int bits_low(double y) { return __double2loint(y); }
__device__ __forceinline__ int bits_low(float y) { return __float_as_int(y) & 0x7fffff; }
__device__ __forceinline__ double hfg_rsqrt(double x) { return rsqrt(x); }
__device__ __forceinline__ float hfg_rsqrt(float x) { return rsqrtf(x); }

// F[0..L] at T from the staged slice (shared memory) of this class.
template <int L, typename Real> __device__ __forceinline__ void boys_eval(Real T, const Real* __restrict__ slice, Real* F)
{
    using G = BoysGrid<Real>;
    if (T > Real(kBoysAsymptotic))
    {
        const Real r    = hfg_rsqrt(T);
        const Real invT = r * r;
        F[0]            = Real(kSqrtPiBy2) * r;
#pragma unroll
        for (int m = 0; m < L; ++m) F[m + 1] = (Real(m) + Real(0.5)) * invT * F[m];
        return;
    }
    // Nearest grid point without a float->int conversion: adding 1.5*2^52 leaves round(T/h) in the low
    // mantissa bits (T is finite and >= 0 here; the clamp keeps a corrupt T inside the slice).
    const Real y  = T * Real(G::kInvStep) + Real(kRoundMagic<Real>);
    const int pt  = max(0, min(static_cast<int>(bits_low(y) - kRoundMagicLow<Real>), G::kPoints - 1));
    const Real x  = (y - Real(kRoundMagic<Real>)) * Real(G::kStep) - T; // T_i - T
    const Real* g = slice + pt * G::kRow;
    Real f        = g[G::kTerms - 1];
#pragma unroll
    for (int k = G::kTerms - 2; k >= 0; --k) f = f * x + g[k];
    F[L] = f;
    if constexpr (L > 0)
    {
        // e^{-T} = e^{-T_i} * e^{x}, x = T_i - T, |x| <= h/2: series to the same order as the Taylor part.
        Real ex = Real(inv_fact(G::kTerms));
#pragma unroll
        for (int k = G::kTerms - 1; k >= 0; --k) ex = ex * x + Real(inv_fact(k));
        const Real e    = g[G::kTerms] * ex;
        const Real twoT = T + T;
#pragma unroll
        for (int m = L; m >= 1; --m) F[m - 1] = (twoT * F[m] + e) * Real(1.0 / (2 * m - 1));
    }
}

// Widening to double for the FP64 accumulators without the FP64 pipe (GB300 runs float -> double
// conversions there, at 1/64 of the FP32 rate): the IEEE-754 fields are moved with integer operations.
// Exact for normal numbers and zero; float subnormals (< 1.2e-38) become zero; infinities and NaNs keep
// their class.
__device__ __forceinline__ double widen(float x)
{
    const unsigned u                 = __float_as_uint(x);
    const unsigned e                 = (u >> 23) & 0xffu;
    const unsigned long long sign    = static_cast<unsigned long long>(u & 0x80000000u) << 32;
    const unsigned long long de      = e == 0xffu ? 0x7ffull : static_cast<unsigned long long>(e + 896u);
    const unsigned long long normal  = sign | (de << 52) | (static_cast<unsigned long long>(u & 0x7fffffu) << 29);
    return __longlong_as_double(static_cast<long long>(e == 0u ? sign : normal));
}
__device__ __forceinline__ double widen(double x) { return x; }

// |x| as a float by integer operations, truncated (below FP32's normal range 0, above it +inf).
__device__ __forceinline__ float narrow_abs(double x)
{
    const unsigned hi = static_cast<unsigned>(__double2hiint(x)) & 0x7fffffffu, lo = static_cast<unsigned>(__double2loint(x));
    if (hi < 0x38100000u)
        return 0.0f;
    if (hi >= 0x47f00000u)
        return __uint_as_float(0x7f800000u);
    return __uint_as_float(((hi - 0x38000000u) << 3) | (lo >> 29));
}

// s^N.
template <int N> __device__ __forceinline__ double power(double s)
{
    if constexpr (N == 1)
        return s;
    else if constexpr (N % 2 == 0)
    {
        const double h = power<N / 2>(s);
        return h * h;
    }
    else
        return s * power<N - 1>(s);
}

// f[m] = c s^m F_m(T), m = 0..L, with s = -2 rho and T = rho R2: what the R recursion starts from.  The
// recursion runs on the scaled values, f_{m-1} = (c s^{m-1} e^{-T} - R2 f_m) / (2m - 1) (2T = -s R2), which
// saves scaling each order, and the grid point is found in FP32 (an index off by one at a cell's edge only
// lets |d| exceed h/2 by an ulp of FP32).
template <int L> __device__ __forceinline__ void scaled_boys(double c, double s, double R2, const double* __restrict__ slice, double* f)
{
    using G          = BoysFast;
    const double m2T = s * R2; // -2T
    const float t2   = narrow_abs(m2T);
    if (t2 > static_cast<float>(2.0 * kBoysAsymptotic))
    {
        const double r = hfg_rsqrt(-0.5 * m2T);
        f[0]           = (c * kSqrtPiBy2) * r;
        if constexpr (L > 0)
        {
            const double g = s * (r * r); // f_{m+1} = s (m + 1/2) f_m / T
#pragma unroll
            for (int m = 0; m < L; ++m) f[m + 1] = ((m + 0.5) * g) * f[m];
        }
        return;
    }
    const float y   = fmaf(t2, static_cast<float>(0.5 * G::kInvStep), static_cast<float>(kRoundMagic<float>));
    const int pt    = max(0, min(__float_as_int(y) - __float_as_int(static_cast<float>(kRoundMagic<float>)), G::kPoints - 1));
    const float ti  = (y - static_cast<float>(kRoundMagic<float>)) * static_cast<float>(G::kStep); // exact
    const double x  = fma(0.5, m2T, widen(ti));                                                    // T_i - T
    const double* g = slice + pt * G::kRow;
    double F        = g[G::kTerms - 1];
#pragma unroll
    for (int k = G::kTerms - 2; k >= 0; --k) F = F * x + g[k];
    if constexpr (L == 0)
        f[0] = c * F;
    else
    {
        double ex = kExpCoefficient<kExpTerms - 1>;
        static_for<0, kExpTerms - 1>([&](auto K) { ex = ex * x + kExpCoefficient<kExpTerms - 2 - decltype(K)::value>; });
        double u[L];
        u[0] = c * (g[G::kTerms] * ex);
#pragma unroll
        for (int k = 1; k < L; ++k) u[k] = u[k - 1] * s;
        f[L] = (c * power<L>(s)) * F;
#pragma unroll
        for (int m = L; m >= 1; --m)
        {
            const double t = fma(-R2, f[m], u[m - 1]);
            f[m - 1]       = m == 1 ? t : t * (1.0 / (2 * m - 1));
        }
    }
}
#endif
} // namespace hfg
