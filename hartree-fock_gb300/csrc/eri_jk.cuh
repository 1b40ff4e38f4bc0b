// Fused McMurchie-Davidson ERI evaluation + J/K digestion for one shell-quartet class.
//
// Reference counterpart: IntegralEngine::electronRepulsion (src/IntegralEngine.cpp:731-992) fused with
// the digestion loop of SCF::buildFockMatrixDirect (src/SCF.cpp:630-711).
//
// One thread evaluates one surviving shell quartet (ab|cd) of class (LA LB | LC LD), LA >= LB,
// LC >= LD, with every loop over Cartesian components, Hermite indices and expansion coefficients
// unrolled at compile time (static_for), so the R, G and ERI arrays are register arrays.  The
// contraction order per quartet:
//
//   for each bra primitive pair:   G[tuv][kl] = sum_{ket prims} sum_{tau nu phi} (-1)^{tau+nu+phi}
//                                               E^{kl}_{tau nu phi} R_{t+tau, u+nu, v+phi}
//                                  ERI[ij][kl] += sum_{tuv} E^{ij}_{tuv} G[tuv][kl]
//
// with R^n_{000} = pref * (-2 rho)^n F_n (the Boys values carry the whole primitive prefactor
// 2 pi^{5/2} / (p q sqrt(p+q)) * K_ab K_cd * coefficients * radial norms).  The 3-D Hermite tables
// E^{ij}_{tuv} of each primitive pair are precomputed once per engine (they depend only on the pair),
// which removes the per-quartet E recursion of the reference (IntegralEngine.cpp:805-820).
//
// Digestion: with s = (a==b ? 1/2 : 1)(c==d ? 1/2 : 1)(ab==cd ? 1/2 : 1) and v = s*(ij|kl),
//   X[i,j] += 2 v dDt[k,l]    X[k,l] += 2 v dDt[i,j]
//   Y[i,k] += v dDs[j,l]      Y[i,l] += v dDs[j,k]    Y[j,k] += v dDs[i,l]    Y[j,l] += v dDs[i,k]
// and afterwards J = X + X^T, K = Y + Y^T.  This covers every permutation of every unique integral once,
// which is what the reference's AO-level symmetry factors (SCF.cpp:665-707) achieve; the reference's
// AO-level skip |(ij|kl)| < SCHWARTZ_THRESH (SCF.cpp:669-671) is applied to the same contracted values.
// Per-quartet partial sums are formed in registers and added to X/Y once per quartet.
#pragma once

#include "boys.cuh"
#include "hfg_common.cuh"

namespace hfg
{
constexpr double kTwoPi25 = 34.98683665524972497; // 2 pi^{5/2}

// 1/sqrt(p+q) and -2 pq/(p+q) for every two primitive-pair exponents of the basis: they depend on the
// exponents alone, of which a molecule's pairs have few distinct ones (136 for water in 6-31G**), and cost ten
// FP64 instructions per primitive quartet to compute against one 16-byte load.  Null where the basis has
// more than kMaxExponents of them (16.8 MB); the kernels compute the two numbers then.  FP64 builds with and
// without the table: 52.3 / 57.5 ms at 136 sums ((H2O)_16/6-31G**), and for 16 H2X with several X 16.8 / 20.6 at 595
// (C N O, 6-31G), 107 / 118 at 903 (C N O, 6-311G**), 14.9 / 18.2 at 990 (C N O F, 6-31G).
constexpr int kMaxExponents = 1024;
struct ExponentTable
{
    const double2* t; // [n][n]
    int n;
};

// Device view of everything a class kernel needs.
struct FockView
{
    const PairRec* pairs;
    const void* pptab[kNumPairClasses]; // per pair class: primitive-pair records (Real of the kernel)
    // Per pair class: the same records field-major, value f of primitive slot s at [f * kfs + s].  Slots
    // follow the sorted class lists, so consecutive kets of a list read consecutive addresses.
    const void* ksoa[kNumPairClasses];
    long long kfs[kNumPairClasses];
    const void* Dt;                     // dD_tot   (double for FP64 kernels, float for FP32 kernels)
    // The exchange matrices are transposed, element (r, c) at c + r * n: the exchange terms pair an AO of the
    // bra, which the lanes of a warp share, with one of the ket, which differs; along the ket index the
    // components of a shell and neighbouring shells now share sectors and lines.
    const void* Da;                     // dD_alpha, transposed
    const void* Db;                     // dD_beta (UHF), transposed
    double* X;                          // J accumulator (J = X + X^T)
    double* Ya;                         // K_alpha accumulator, transposed or not (K = Y + Y^T)
    double* Yb;                         // K_beta accumulator (UHF)
    const long long* mat_off;           // per molecule: offset of its n x n block in the packed matrices
    const int* mat_ld;                  // per molecule: n
    double ao_thr;                      // AO-level skip threshold (SCHWARTZ_THRESH)
    float ao_thr_f;                     // the same threshold for the FP32 kernels
    double* store;                      // if set: write the quartets' integrals here instead of digesting
    ExponentTable et;
};

__device__ constexpr double ang_norm(int l, int c)
{
    const int i = cart_exp(l, c, 0), j = cart_exp(l, c, 1), k = cart_exp(l, c, 2);
    const int d = dfact_odd(2 * i - 1) * dfact_odd(2 * j - 1) * dfact_odd(2 * k - 1);
    return d == 1 ? 1.0 : (d == 3 ? 0.57735026918962576451 : (d == 9 ? 1.0 / 3.0 : (d == 15 ? 0.25819888974716112568 : 1.0)));
}

// Enumerates Hermite triples of total degree <= L by descending degree: k-th entry's hidx(., ., ., L).
__host__ __device__ constexpr int herm_desc(int k, int L)
{
    int n = 0;
    for (int d = L; d >= 0; --d)
        for (int v = 0; v <= d; ++v)
            for (int u = 0; u <= d - v; ++u)
            {
                if (n == k)
                    return hidx(d - u - v, u, v, L);
                ++n;
            }
    return 0;
}

// R^0_{tuv} for t+u+v <= L into R[hidx(t,u,v,L)], from Fs[n] = pref (-2 rho)^n F_n, in place,
// level by level (IntegralEngine.cpp:1082-1162 computes the same recursion in a dense 4-D buffer).
template <int L, typename Real>
__device__ __forceinline__ void hermite_R(const Real* Fs, Real X, Real Y, Real Z, Real* R)
{
    R[0] = Fs[L];
    static_for<0, L>(
        [&](auto NN)
        {
            constexpr int n = L - 1 - decltype(NN)::value;
            static_for<0, nherm(L)>(
                [&](auto KK)
                {
                    constexpr int h = herm_desc(decltype(KK)::value, L);
                    constexpr int t = htuv(h, L, 0), u = htuv(h, L, 1), v = htuv(h, L, 2);
                    constexpr int d = t + u + v;
                    if constexpr (d >= 1 && d <= L - n)
                    {
                        if constexpr (t > 0)
                        {
                            if constexpr (t >= 2)
                                R[h] = X * R[hidx(t - 1, u, v, L)] + Real(t - 1) * R[hidx(t - 2, u, v, L)];
                            else
                                R[h] = X * R[hidx(t - 1, u, v, L)];
                        }
                        else if constexpr (u > 0)
                        {
                            if constexpr (u >= 2)
                                R[h] = Y * R[hidx(t, u - 1, v, L)] + Real(u - 1) * R[hidx(t, u - 2, v, L)];
                            else
                                R[h] = Y * R[hidx(t, u - 1, v, L)];
                        }
                        else
                        {
                            if constexpr (v >= 2)
                                R[h] = Z * R[hidx(t, u, v - 1, L)] + Real(v - 1) * R[hidx(t, u, v - 2, L)];
                            else
                                R[h] = Z * R[hidx(t, u, v - 1, L)];
                        }
                    }
                });
            R[0] = Fs[n];
        });
}

// Field f of one primitive-pair record: records stored whole (AoS) or field-major (SoA, stride fs).
template <typename Real, bool SoA> struct RecRef
{
    const Real* __restrict__ p;
    long long fs;
    __device__ __forceinline__ Real operator[](int f) const
    {
        if constexpr (SoA)
            return p[f * fs];
        else
            return p[f];
    }
};

// The scalar part of one primitive quartet: P - Q and Fs[n] = pref (-2 rho)^n F_n, n = 0..L.  Fast (FP64
// only): from a BoysFast slice and the exponent table; else from a BoysGrid<Real> slice.
template <int L, typename Real, bool Fast, typename Bra, typename Ket>
__device__ __forceinline__ void prim_scalars(const Bra& rb, const Ket& rk, const ExponentTable& et,
                                             const Real* __restrict__ slice, Real& X, Real& Y, Real& Z, Real* Fs)
{
    if constexpr (Fast)
    {
        X = rb[1] - rk[1];
        Y = rb[2] - rk[2];
        Z = rb[3] - rk[3];
        double rs, s;
        if (et.t != nullptr)
        {
            const double2 v = __ldg(et.t + (__double2loint(rb[5]) * et.n + __double2loint(rk[5])));
            rs              = v.x;
            s               = v.y;
        }
        else
        {
            rs = rsqrt(rb[0] + rk[0]);
            s  = (-2.0 * (rb[0] * rk[0])) * (rs * rs);
        }
        scaled_boys<L>((rb[4] * rk[4]) * rs, s, X * X + Y * Y + Z * Z, slice, Fs);
    }
    else
    {
        const Real p = rb[0], q = rk[0];
        X = rb[1] - rk[1];
        Y = rb[2] - rk[2];
        Z = rb[3] - rk[3];
        const Real rs   = hfg_rsqrt(p + q);
        const Real rho  = (p * q) * (rs * rs);
        const Real pref = (rb[4] * rk[4]) * rs;
        const Real T    = rho * (X * X + Y * Y + Z * Z);
        Real F[L + 1];
        boys_eval<L, Real>(T, slice, F);
        const Real m2r = Real(-2) * rho;
        Real w         = pref;
#pragma unroll
        for (int n = 0; n <= L; ++n)
        {
            Fs[n] = w * F[n];
            w *= m2r;
        }
    }
}

// The primitive quartets one lane of a group evaluates: bra primitives ib0, ib0 + ibs, ... and, for each,
// ket primitives ik0, ik0 + iks, ... (all of them by default).
struct PrimRange
{
    int ib0 = 0, ibs = 1, ik0 = 0, iks = 1;
};

// Contracted Cartesian integrals of one quartet (without the angular normalisation factors), for the ket
// components kl in [KL0, KL1) (all of them by default): acc[ij * (KL1 - KL0) + kl - KL0].  KSoA: the ket
// table tk is field-major with field stride kfs.  Fast (FP64, bound by the FP64 pipe): the scalars of
// scaled_boys, and every Hermite term is one DFMA straight into its accumulator; a local sum added
// afterwards costs HAB * NCD more FP64 instructions per primitive quartet.
template <int LA, int LB, int LC, int LD, typename Real, bool KSoA = false, int KL0 = 0,
          int KL1 = ncart(LC) * ncart(LD), bool Fast = false>
__device__ __forceinline__ void eval_quartet(const PairRec& bra, const PairRec& ket, const Real* __restrict__ tb,
                                             const Real* __restrict__ tk, const Real* __restrict__ slice,
                                             Real* acc, long long kfs = 0, const ExponentTable et = ExponentTable {},
                                             const PrimRange pr = PrimRange {})
{
    constexpr int LAB = LA + LB, LCD = LC + LD, L = LAB + LCD;
    constexpr int NAB = ncart(LA) * ncart(LB), NCD = KL1 - KL0;
    constexpr int HAB = nherm(LAB), HL = nherm(L);
    constexpr int SB = pp_stride(LA, LB), SK = pp_stride(LC, LD);
#pragma unroll
    for (int x = 0; x < NAB * NCD; ++x) acc[x] = Real(0);

    for (int ib = pr.ib0; ib < bra.npp; ib += pr.ibs)
    {
        const Real* __restrict__ rb = tb + static_cast<size_t>(bra.pp_off + ib) * SB;
        Real G[HAB * NCD];
#pragma unroll
        for (int x = 0; x < HAB * NCD; ++x) G[x] = Real(0);

        for (int ik = pr.ik0; ik < ket.npp; ik += pr.iks)
        {
            const RecRef<Real, KSoA> rk {KSoA ? tk + (ket.kslot + static_cast<long long>(ik) * ket.kstep)
                                              : tk + static_cast<size_t>(ket.pp_off + ik) * SK,
                                         kfs};
            Real X, Y, Z, Fs[L + 1];
            prim_scalars<L, Real, Fast>(rb, rk, et, slice, X, Y, Z, Fs);
            Real R[HL];
            hermite_R<L, Real>(Fs, X, Y, Z, R);

            static_for<KL0, KL1>(
                [&](auto KL)
                {
                    constexpr int kl   = decltype(KL)::value;
                    constexpr int lx   = e3_len(LC, LD, kl, 0), ly = e3_len(LC, LD, kl, 1), lz = e3_len(LC, LD, kl, 2);
                    constexpr int eoff = kPairHeader + e3_offset(LC, LD, kl);
                    static_for<0, HAB>(
                        [&](auto TUV)
                        {
                            constexpr int h = decltype(TUV)::value;
                            constexpr int t = htuv(h, LAB, 0), u = htuv(h, LAB, 1), v = htuv(h, LAB, 2);
                            Real s          = Fast ? G[h * NCD + (kl - KL0)] : Real(0);
                            static_for<0, lx * ly * lz>(
                                [&](auto EE)
                                {
                                    constexpr int e   = decltype(EE)::value;
                                    constexpr int tau = e % lx, nu = (e / lx) % ly, phi = e / (lx * ly);
                                    const Real rr     = R[hidx(t + tau, u + nu, v + phi, L)];
                                    const Real term   = (LC + LD == 0) ? rr : rk[eoff + e] * rr;
                                    if constexpr (((tau + nu + phi) & 1) != 0)
                                        s -= term;
                                    else
                                        s += term;
                                });
                            if constexpr (Fast)
                                G[h * NCD + (kl - KL0)] = s;
                            else
                                G[h * NCD + (kl - KL0)] += s;
                        });
                });
        }

        static_for<0, NAB>(
            [&](auto IJ)
            {
                constexpr int ij   = decltype(IJ)::value;
                constexpr int lx   = e3_len(LA, LB, ij, 0), ly = e3_len(LA, LB, ij, 1), lz = e3_len(LA, LB, ij, 2);
                constexpr int eoff = kPairHeader + e3_offset(LA, LB, ij);
#pragma unroll
                for (int kl = 0; kl < NCD; ++kl)
                {
                    Real s = Fast ? acc[ij * NCD + kl] : Real(0);
                    static_for<0, lx * ly * lz>(
                        [&](auto EE)
                        {
                            constexpr int e = decltype(EE)::value;
                            constexpr int t = e % lx, u = (e / lx) % ly, v = e / (lx * ly);
                            const Real gg = G[hidx(t, u, v, LAB) * NCD + kl];
                            s += (LA + LB == 0) ? gg : rb[eoff + e] * gg;
                        });
                    if constexpr (Fast)
                        acc[ij * NCD + kl] = s;
                    else
                        acc[ij * NCD + kl] += s;
                }
            });
    }
}

template <typename Real> __device__ __forceinline__ Real ao_threshold(const FockView& v)
{
    if constexpr (sizeof(Real) == 4)
        return v.ao_thr_f;
    else
        return v.ao_thr;
}

template <typename Real> __device__ __forceinline__ Real ldD(const void* p, long long i)
{
    return static_cast<const Real*>(p)[i];
}

// Density values one quartet's digestion reads: dD_tot over (cd) and (ab); per spin, the exchange
// partners (bd), (bc), (ad), (ac).
template <int LA, int LB, int LC, int LD, typename Real, bool UHF> struct DigestD
{
    static constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
    static constexpr int NS = UHF ? 2 : 1;
    static constexpr int kCount = NA * NB + NC * ND + NS * (NB * ND + NB * NC + NA * ND + NA * NC);
    // FP32 kernels (memory-latency bound) load them before the primitive loop, so the loads overlap the
    // integral evaluation, when they fit in about 40 registers; FP64 kernels (FP64-pipe bound) right
    // before the digestion.
    static constexpr bool kEarly = sizeof(Real) == 4 && kCount <= 40;
    Real Dcd[NC * ND], Dab[NA * NB];
    Real Dbd[NS][NB * ND], Dbc[NS][NB * NC], Dad[NS][NA * ND], Dac[NS][NA * NC];
};

template <int LA, int LB, int LC, int LD, typename Real, bool UHF>
__device__ __forceinline__ void load_digest_d(const PairRec& bra, const PairRec& ket, const FockView& v,
                                              DigestD<LA, LB, LC, LD, Real, UHF>& d)
{
    constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
    const long long off = v.mat_off[bra.mol];
    const int n         = v.mat_ld[bra.mol];
    const int a0 = bra.ao1, b0 = bra.ao2, c0 = ket.ao1, d0 = ket.ao2;
    auto at = [&](int r, int c) -> long long { return off + r + static_cast<long long>(c) * n; };
    auto tr = [&](int r, int c) -> long long { return off + c + static_cast<long long>(r) * n; };
#pragma unroll
    for (int k = 0; k < NC; ++k)
#pragma unroll
        for (int l = 0; l < ND; ++l) d.Dcd[k * ND + l] = ldD<Real>(v.Dt, at(c0 + k, d0 + l));
#pragma unroll
    for (int i = 0; i < NA; ++i)
#pragma unroll
        for (int j = 0; j < NB; ++j) d.Dab[i * NB + j] = ldD<Real>(v.Dt, at(a0 + i, b0 + j));
#pragma unroll
    for (int spin = 0; spin < (UHF ? 2 : 1); ++spin)
    {
        const void* Ds = spin == 0 ? v.Da : v.Db;
#pragma unroll
        for (int j = 0; j < NB; ++j)
        {
#pragma unroll
            for (int l = 0; l < ND; ++l) d.Dbd[spin][j * ND + l] = ldD<Real>(Ds, tr(b0 + j, d0 + l));
#pragma unroll
            for (int k = 0; k < NC; ++k) d.Dbc[spin][j * NC + k] = ldD<Real>(Ds, tr(b0 + j, c0 + k));
        }
#pragma unroll
        for (int i = 0; i < NA; ++i)
        {
#pragma unroll
            for (int l = 0; l < ND; ++l) d.Dad[spin][i * ND + l] = ldD<Real>(Ds, tr(a0 + i, d0 + l));
#pragma unroll
            for (int k = 0; k < NC; ++k) d.Dac[spin][i * NC + k] = ldD<Real>(Ds, tr(a0 + i, c0 + k));
        }
    }
}

// Ket components kl in [KL0, KL1) that touch ket Cartesian index k (of shell c) or l (of shell d).
template <int ND, int KL0, int KL1> __host__ __device__ constexpr bool chunk_has_k(int k)
{
    for (int kl = KL0; kl < KL1; ++kl)
        if (kl / ND == k)
            return true;
    return false;
}
template <int ND, int KL0, int KL1> __host__ __device__ constexpr bool chunk_has_l(int l)
{
    for (int kl = KL0; kl < KL1; ++kl)
        if (kl % ND == l)
            return true;
    return false;
}

// 2x and |x| < thr without the FP64 pipe in FP64 (thr >= 0; IEEE bit patterns of non-negative numbers order
// like the numbers, a NaN is above any thr).  Doubling drops subnormals, keeps infinities and NaN, and the
// largest binade becomes an infinity.
__device__ __forceinline__ double twice(double x)
{
    const int hi = __double2hiint(x), e = hi & 0x7ff00000;
    const bool top = e >= 0x7fe00000, sub = e == 0;
    const int h2   = e == 0x7ff00000 ? hi : top ? (hi & 0x80000000) | 0x7ff00000 : hi + 0x00100000;
    const int l2   = e == 0x7fe00000 ? 0 : __double2loint(x);
    return __hiloint2double(sub ? 0 : h2, sub ? 0 : l2);
}
__device__ __forceinline__ float twice(float x) { return 2.0f * x; }
__device__ __forceinline__ bool below(double x, double thr)
{
    return (__double_as_longlong(x) & 0x7fffffffffffffffll) < __double_as_longlong(thr);
}
__device__ __forceinline__ bool below(float x, float thr) { return fabsf(x) < thr; }

// Sums x[0..N) over the warp, handing half of the values to the other half of the lanes at every step: some
// N + 5 additions a lane in the place of 5 N.  Returns this lane's value and its index (-1: another lane
// adds it).  N <= 64; values beyond 32 leave two per lane, in `second`.
template <int N> __device__ __forceinline__ void warp_sum_spread(double* x, int lane, double& first, int& at1, double& second, int& at2)
{
    int base = 0, len = N; // this lane's values are base .. base + len of the original
    bool mine = true;
    static_for<0, 5>(
        [&](auto S)
        {
            constexpr int o = 16 >> decltype(S)::value;
            // Values held at this step: ceil(N / 2^S).
            constexpr int M = (N + (1 << decltype(S)::value) - 1) >> decltype(S)::value, H = (M + 1) / 2;
            const bool up = (lane & o) != 0;
            if constexpr (M == 1)
            {
                x[0] += __shfl_xor_sync(0xffffffffu, x[0], o);
                mine = mine && !up;
            }
            else
            {
#pragma unroll
                for (int k = 0; k < H; ++k)
                {
                    const double lo = x[k], hi = H + k < M ? x[H + k] : 0.0;
                    const double other = __shfl_xor_sync(0xffffffffu, up ? lo : hi, o);
                    x[k]               = (up ? hi : lo) + other;
                }
                base += up ? H : 0;
                len = up ? max(0, len - H) : min(len, H);
            }
        });
    constexpr int last = (N + 31) >> 5;
    first  = x[0];
    at1    = mine && len > 0 ? base : -1;
    second = last > 1 ? x[1] : 0.0;
    at2    = mine && len > 1 ? base + 1 : -1;
}

// Digestion of one evaluated quartet into X, Ya (, Yb), with its density values already loaded; acc holds
// the integrals of the ket components kl in [KL0, KL1) (all of them by default), and only the output
// elements those components reach are added.
// Normalised: acc carries the angular factors already.  The skip and the degeneracy factor (a power of two,
// 1 for most quartets) are applied before the contraction, without the FP64 pipe where nothing is to scale.
// bra_warp: every lane of the warp calls this together and all active lanes hold the same bra pair;
// the bra's Coulomb block X_ab is then summed over the warp and added once (inactive lanes pass
// active = false and acc = 0, and add nothing).  Otherwise each active lane adds its own.
template <int LA, int LB, int LC, int LD, typename Real, bool UHF, int KL0 = 0, int KL1 = ncart(LC) * ncart(LD),
          bool Normalised = false>
__device__ __forceinline__ void digest_loaded(const PairRec& bra, const PairRec& ket, bool same_pair, const Real* acc,
                                              const FockView& v, const DigestD<LA, LB, LC, LD, Real, UHF>& d,
                                              bool active, bool bra_warp)
{
    constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
    constexpr int NAB = NA * NB, CH = KL1 - KL0;
    const long long off = v.mat_off[bra.mol];
    const int n         = v.mat_ld[bra.mol];
    const Real s   = (bra.same ? Real(0.5) : Real(1)) * (ket.same ? Real(0.5) : Real(1)) * (same_pair ? Real(0.5) : Real(1));
    const Real thr = ao_threshold<Real>(v);
    const int a0 = bra.ao1, b0 = bra.ao2, c0 = ket.ao1, d0 = ket.ao2;
    auto at = [&](int r, int c) -> long long { return off + r + static_cast<long long>(c) * n; };
    auto tr = [&](int r, int c) -> long long { return off + c + static_cast<long long>(r) * n; };

    Real w[NAB * CH];
    static_for<0, NAB * CH>(
        [&](auto E)
        {
            constexpr int x   = decltype(E)::value;
            constexpr Real an = Real(ang_norm(LA, x / CH / NB) * ang_norm(LB, (x / CH) % NB) *
                                     ang_norm(LC, (KL0 + x % CH) / ND) * ang_norm(LD, (KL0 + x % CH) % ND));
            const Real eri = Normalised ? acc[x] : acc[x] * an;
            w[x]           = below(eri, thr) ? Real(0) : eri;
        });
    if (__any_sync(__activemask(), s != Real(1)))
#pragma unroll
        for (int x = 0; x < NAB * CH; ++x) w[x] *= s;

    Real Jab[NAB], Jcd[CH];
#pragma unroll
    for (int x = 0; x < NAB; ++x) Jab[x] = Real(0);
#pragma unroll
    for (int x = 0; x < CH; ++x) Jcd[x] = Real(0);

    constexpr int nspin = UHF ? 2 : 1;
#pragma unroll
    for (int spin = 0; spin < nspin; ++spin)
    {
        Real Kac[NA * NC], Kad[NA * ND], Kbc[NB * NC], Kbd[NB * ND];
#pragma unroll
        for (int x = 0; x < NA * NC; ++x) Kac[x] = Real(0);
#pragma unroll
        for (int x = 0; x < NA * ND; ++x) Kad[x] = Real(0);
#pragma unroll
        for (int x = 0; x < NB * NC; ++x) Kbc[x] = Real(0);
#pragma unroll
        for (int x = 0; x < NB * ND; ++x) Kbd[x] = Real(0);

        static_for<0, NA>(
            [&](auto I)
            {
                constexpr int i = decltype(I)::value;
                static_for<0, NB>(
                    [&](auto Jx)
                    {
                        constexpr int j = decltype(Jx)::value;
                        static_for<KL0, KL1>(
                            [&](auto KLx)
                            {
                                constexpr int kl = decltype(KLx)::value;
                                constexpr int k = kl / ND, l = kl % ND;
                                const Real g = w[(i * NB + j) * CH + (kl - KL0)];
                                if (spin == 0)
                                {
                                    Jab[i * NB + j] += g * d.Dcd[k * ND + l];
                                    Jcd[kl - KL0] += g * d.Dab[i * NB + j];
                                }
                                Kac[i * NC + k] += g * d.Dbd[spin][j * ND + l];
                                Kad[i * ND + l] += g * d.Dbc[spin][j * NC + k];
                                Kbc[j * NC + k] += g * d.Dad[spin][i * ND + l];
                                Kbd[j * ND + l] += g * d.Dac[spin][i * NC + k];
                            });
                    });
            });
        if (active)
        {
            double* Y = spin == 0 ? v.Ya : v.Yb;
            static_for<0, NA>(
                [&](auto I)
                {
                    constexpr int i = decltype(I)::value;
                    static_for<0, NC>(
                        [&](auto Kx)
                        {
                            constexpr int k = decltype(Kx)::value;
                            if constexpr (chunk_has_k<ND, KL0, KL1>(k))
                                atomicAdd(Y + tr(a0 + i, c0 + k), widen(Kac[i * NC + k]));
                        });
                    static_for<0, ND>(
                        [&](auto Lx)
                        {
                            constexpr int l = decltype(Lx)::value;
                            if constexpr (chunk_has_l<ND, KL0, KL1>(l))
                                atomicAdd(Y + tr(a0 + i, d0 + l), widen(Kad[i * ND + l]));
                        });
                });
            static_for<0, NB>(
                [&](auto Jx)
                {
                    constexpr int j = decltype(Jx)::value;
                    static_for<0, NC>(
                        [&](auto Kx)
                        {
                            constexpr int k = decltype(Kx)::value;
                            if constexpr (chunk_has_k<ND, KL0, KL1>(k))
                                atomicAdd(Y + tr(b0 + j, c0 + k), widen(Kbc[j * NC + k]));
                        });
                    static_for<0, ND>(
                        [&](auto Lx)
                        {
                            constexpr int l = decltype(Lx)::value;
                            if constexpr (chunk_has_l<ND, KL0, KL1>(l))
                                atomicAdd(Y + tr(b0 + j, d0 + l), widen(Kbd[j * ND + l]));
                        });
                });
        }
    }
    if (bra_warp)
    {
        // Warp sum of the bra block, then one atomic per element from lane 0.  A lane without integrals of its own
        // has loaded a quartet's densities all the same, and 0 times an infinite one is a NaN.
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int x = 0; x < NAB; ++x) Jab[x] = active ? Jab[x] : Real(0);
        if constexpr (sizeof(Real) == 8)
        {
            double t1, t2;
            int x1, x2;
            warp_sum_spread<NAB>(Jab, lane, t1, x1, t2, x2);
            if (x1 >= 0)
                atomicAdd(v.X + at(a0 + x1 / NB, b0 + x1 % NB), twice(t1));
            if (NAB > 32 && x2 >= 0)
                atomicAdd(v.X + at(a0 + x2 / NB, b0 + x2 % NB), twice(t2));
        }
        else
        {
#pragma unroll
            for (int x = 0; x < NAB; ++x)
            {
                Real t = Jab[x];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                if (lane == 0)
                    atomicAdd(v.X + at(a0 + x / NB, b0 + x % NB), widen(twice(t)));
            }
        }
    }
    else if (active)
    {
#pragma unroll
        for (int i = 0; i < NA; ++i)
#pragma unroll
            for (int j = 0; j < NB; ++j) atomicAdd(v.X + at(a0 + i, b0 + j), widen(twice(Jab[i * NB + j])));
    }
    if (active)
    {
#pragma unroll
        for (int x = 0; x < CH; ++x)
            atomicAdd(v.X + at(c0 + (KL0 + x) / ND, d0 + (KL0 + x) % ND), widen(twice(Jcd[x])));
    }
}

// Digestion of one evaluated quartet by one lane on its own.
template <int LA, int LB, int LC, int LD, typename Real, bool UHF>
__device__ __forceinline__ void digest_quartet(const PairRec& bra, const PairRec& ket, bool same_pair, const Real* acc,
                                               const FockView& v)
{
    DigestD<LA, LB, LC, LD, Real, UHF> d;
    load_digest_d<LA, LB, LC, LD, Real, UHF>(bra, ket, v, d);
    digest_loaded<LA, LB, LC, LD, Real, UHF>(bra, ket, same_pair, acc, v, d, true, false);
}

// Values of the Boys slice the thread, chunk and gradient kernels stage: BoysFast in FP64.
template <typename Real> __host__ __device__ constexpr int boys_slice_size()
{
    return sizeof(Real) == 8 ? BoysFast::kPoints * BoysFast::kRow : BoysGrid<Real>::kPoints * BoysGrid<Real>::kRow;
}

// Stage this class's Boys slice in shared memory.
template <typename Real, int n = BoysGrid<Real>::kPoints * BoysGrid<Real>::kRow>
__device__ __forceinline__ void stage_boys(const Real* __restrict__ g, Real* s)
{
    for (int i = threadIdx.x; i < n; i += blockDim.x) s[i] = g[i];
    __syncthreads();
}

// How a launch splits its quartets' primitive quartets over lanes.  A quartet's primitive quartets are one
// dependent FP64 chain per thread, and the contracted shells have hundreds to thousands of them ((8 8|8 8)
// primitives in cc-pVDZ): a list too short to fill the GPU then takes as long as its longest quartet.  So
// a window of 32 list entries is worked on by G warps, G a power of two up to `smax` (1 to 128): every
// quartet gets G lanes, each with a strided share of the bra and ket primitives, and the lanes' integrals
// are summed before one of them digests.  G grows with the window's primitive count P until each lane
// has at most m = max(1, prims / lanes) primitive quartets, `prims` being the whole list's primitive
// quartets and `lanes` what fills the GPU: a long list (m above any P) runs one lane per quartet, as
// before, and pays nothing.  A list of many waves, whose items go to whoever is free (`next`), splits eight
// times finer, down to 32 primitive quartets a lane (every lane repeats the transform of its bra primitives and
// joins the sum over lanes), so that its last items are an eighth of a lane's share and not all of it.
struct SplitArgs
{
    int smax = 1;                             // warps per window at most, a power of two; 1: no split
    int run  = 1;                             // consecutive items taken at a time
    // Items taken so far by the whole launch (zeroed before it), or null: items go round robin.  The windows of a
    // list differ a hundredfold in primitive quartets, and with some hundred windows a warp round robin left
    // the SMs idle for a fifth of the FP64 (ps|ss) kernel of (H2O)_16 (ncu: 16.4 M of 21.2 M cycles active).
    unsigned long long* next = nullptr;
    unsigned lanes = 1;                       // lanes that fill the GPU
    unsigned long long prims = 0;             // the list's primitive quartets,
    const unsigned long long* prims_dev = nullptr; // or where they stand (a captured graph's lists)
};

// Primitive quartets a lane of a split list has at most.
__host__ __device__ inline unsigned long long split_share(unsigned long long prims, unsigned lanes, bool queued)
{
    unsigned long long m = prims / lanes;
    if (queued && m > 32)
        m = m / 8 > 32 ? m / 8 : 32;
    return m > 1 ? m : 1;
}

// Lanes per quartet for P primitive quartets at m a lane.
__device__ __forceinline__ int split_lanes(int P, unsigned long long m, int smax)
{
    int g = 1;
    while (g < smax && static_cast<unsigned long long>(g) * m < static_cast<unsigned long long>(P)) g <<= 1;
    return g;
}

// Takes the next run of items [at, end) of `units`; false at the end of the list.  `who`: this taker's number
// of `takers` (round robin); `lead`: the lane that asks the counter, whose answer the mask's lanes share.
__device__ __forceinline__ bool take_items(const SplitArgs& sp, unsigned long long units, unsigned long long who,
                                           unsigned long long takers, unsigned mask, int lead, unsigned long long& round,
                                           unsigned long long& at, unsigned long long& end)
{
    if (sp.next == nullptr)
        at = (round++ * takers + who) * sp.run;
    else
    {
        if ((threadIdx.x & 31) == lead)
            at = atomicAdd(sp.next, static_cast<unsigned long long>(sp.run));
        at = __shfl_sync(mask, at, lead);
    }
    end = at + sp.run < units ? at + sp.run : units;
    return at < units;
}

// Share of lane r of g: the g lanes as a gb x gk grid over the bra and ket primitives, powers of two with
// the fewest rounds.
__device__ __forceinline__ PrimRange split_range(int npb, int npk, int r, int g)
{
    int best = 1 << 30, bk = 1;
    for (int gk = 1; gk <= g; gk <<= 1)
    {
        const int gb = g / gk, rounds = ((npb + gb - 1) / gb) * ((npk + gk - 1) / gk);
        if (rounds < best)
        {
            best = rounds;
            bk   = gk;
        }
    }
    return PrimRange {r / bk, g / bk, r % bk, bk};
}

// Digestion of one quartet by a whole warp: w[ij * (KL1 - KL0) + kl - KL0] in shared memory holds the
// contracted integrals with their angular factors; each lane owns output elements of J and K.  (One lane
// digesting for the warp would run NAB * NCD * 6 dependent FP64 instructions on its own.)
template <int LA, int LB, int LC, int LD, typename Real, bool UHF, int KL0, int KL1>
__device__ __forceinline__ void digest_shared(const PairRec& bra, const PairRec& ket, bool same_pair, Real* w,
                                              const FockView& v)
{
    constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
    constexpr int NAB = NA * NB, CH = KL1 - KL0;
    const int lane = threadIdx.x & 31;
    const long long off = v.mat_off[bra.mol];
    const int n         = v.mat_ld[bra.mol];
    const int a0 = bra.ao1, b0 = bra.ao2, c0 = ket.ao1, d0 = ket.ao2;
    auto at = [&](int r, int c) -> long long { return off + r + static_cast<long long>(c) * n; };
    auto tr = [&](int r, int c) -> long long { return off + c + static_cast<long long>(r) * n; };
    const Real s   = (bra.same ? Real(0.5) : Real(1)) * (ket.same ? Real(0.5) : Real(1)) * (same_pair ? Real(0.5) : Real(1));
    const Real thr = ao_threshold<Real>(v);
    for (int x = lane; x < NAB * CH; x += 32) w[x] = below(w[x], thr) ? Real(0) : s * w[x];
    __syncwarp();
    constexpr int nJ = NAB + CH, nK = (NA + NB) * (NC + ND), nspin = UHF ? 2 : 1;
    for (int o = lane; o < nJ + nspin * nK; o += 32)
    {
        Real sum = Real(0);
        if (o < NAB)
        {
            for (int x = 0; x < CH; ++x) sum += w[o * CH + x] * ldD<Real>(v.Dt, at(c0 + (KL0 + x) / ND, d0 + (KL0 + x) % ND));
            atomicAdd(v.X + at(a0 + o / NB, b0 + o % NB), widen(twice(sum)));
        }
        else if (o < nJ)
        {
            const int x = o - NAB;
            for (int ij = 0; ij < NAB; ++ij) sum += w[ij * CH + x] * ldD<Real>(v.Dt, at(a0 + ij / NB, b0 + ij % NB));
            atomicAdd(v.X + at(c0 + (KL0 + x) / ND, d0 + (KL0 + x) % ND), widen(twice(sum)));
        }
        else
        {
            // K(row AO of a or b, column AO of c or d), contracted with D(the other bra AO, the other ket AO).
            const int k = (o - nJ) % nK, spin = (o - nJ) / nK;
            const int row = k / (NC + ND), col = k % (NC + ND);
            const bool ra = row < NA, cc = col < NC;
            const int i0 = ra ? row : row - NA, k0 = cc ? col : col - NC;
            const void* Ds = spin == 0 ? v.Da : v.Db;
            for (int x = 0; x < CH; ++x)
            {
                const int kk = (KL0 + x) / ND, ll = (KL0 + x) % ND;
                if ((cc ? kk : ll) != k0)
                    continue;
                const int dcol = cc ? d0 + ll : c0 + kk;
                if (ra)
                    for (int j = 0; j < NB; ++j) sum += w[(i0 * NB + j) * CH + x] * ldD<Real>(Ds, tr(b0 + j, dcol));
                else
                    for (int i = 0; i < NA; ++i) sum += w[(i * NB + i0) * CH + x] * ldD<Real>(Ds, tr(a0 + i, dcol));
            }
            bool reached = false;
            for (int x = 0; x < CH; ++x) reached = reached || (cc ? (KL0 + x) / ND : (KL0 + x) % ND) == k0;
            if (reached)
                atomicAdd((spin == 0 ? v.Ya : v.Yb) + tr((ra ? a0 : b0) + i0, (cc ? c0 : d0) + k0), widen(sum));
        }
    }
    __syncwarp(); // the next quartet reuses w
}

// Values of the block's shared scratch of a split launch (per warp one quartet's integrals).
template <int LA, int LB, int KL0, int KL1> __host__ __device__ constexpr int split_scratch()
{
    return 4 * ncart(LA) * ncart(LB) * (KL1 - KL0);
}

// The quartets of one list for the ket components [KL0, KL1): thread per quartet, or G lanes per quartet
// (SplitArgs).  `scratch`: split_scratch() values of shared memory, used by split launches only.
template <int LA, int LB, int LC, int LD, typename Real, bool UHF, int KL0, int KL1>
__device__ __forceinline__ void class_body(const Quartet* __restrict__ list, unsigned long long n, const FockView& v,
                                           const Real* __restrict__ slice, Real* scratch, const SplitArgs& sp)
{
    constexpr int NB = ncart(LB), ND = ncart(LD);
    constexpr int NAB = ncart(LA) * NB, NCD = ncart(LC) * ND, CH = KL1 - KL0, N = NAB * CH;
    const Real* tb      = static_cast<const Real*>(v.pptab[pair_class(LA, LB)]);
    const Real* tk      = static_cast<const Real*>(v.ksoa[pair_class(LC, LD)]);
    const long long kfs = v.kfs[pair_class(LC, LD)];
    using DD            = DigestD<LA, LB, LC, LD, Real, UHF>;
    constexpr bool kEarly = DD::kEarly && CH == NCD;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    // FP32 lists are never split: their chains are short, and their integrals keep one order of summation.
    constexpr bool kFP64 = sizeof(Real) == 8, kSplit = kFP64;
    const int S          = kSplit ? sp.smax : 1;
    const unsigned long long items = ((n + 31) >> 5) * static_cast<unsigned long long>(S);
    unsigned long long m = 0;
    if (kSplit && S > 1)
        m = split_share(sp.prims_dev ? *sp.prims_dev : sp.prims, sp.lanes, sp.next != nullptr);
    // Warp-uniform iteration (every lane runs the same trip count, inactive lanes past the end), so that
    // the digestion may sum the bra block over the warp.  With S >= 64 the four warps of a block take slices of
    // one window, so that they may share a quartet (G = 64, 128): their branches on G are block-uniform.
    // Runs keep the windows of one bra pair together, whose rows of D and records are then found in L1.
    // The four warps of a block may share a quartet (G = 64, 128) and so walk together; lists that long in windows
    // split to at most 32 (plan_items), so these go round robin.
    const bool by_block = S >= 64;
    unsigned long long round = 0, at = 0, end = 0;
    while (take_items(sp, by_block ? items / 4 : items, by_block ? blockIdx.x : blockIdx.x * 4ull + wib,
                      by_block ? gridDim.x : gridDim.x * 4ull, 0xffffffffu, 0, round, at, end))
    for (; at < end; ++at)
    {
        const unsigned long long it = by_block ? at * 4 + wib : at;
        unsigned long long base = it * 32, q = base + lane;
        int g = 1, r = 0;
        PrimRange pr;
        if (kSplit && S > 1)
        {
            const int ls    = __ffs(S) - 1;
            base            = (it >> ls) * 32;
            const int slc   = static_cast<int>(it) & (S - 1);
            q               = base + lane;
            const Quartet w = list[q < n ? q : base];
            g = split_lanes(__reduce_max_sync(0xffffffffu, v.pairs[w.bra].npp * v.pairs[w.ket].npp), m, S);
            if (slc >= g)
            {
                if (!by_block)
                    at |= S - 1; // on to the next window of the run
                continue;
            }
            q = base + (g <= 32 ? slc * (32 / g) + lane / g : slc / (g / 32));
            r = g <= 32 ? lane % g : (slc % (g / 32)) * 32 + lane;
        }
        const bool active = q < n;
        const Quartet qt  = list[active ? q : base];
        const PairRec bra = v.pairs[qt.bra];
        const PairRec ket = v.pairs[qt.ket];
        if (g > 1)
            pr = split_range(bra.npp, ket.npp, r, g);
        DD d;
        if (kEarly)
            load_digest_d<LA, LB, LC, LD, Real, UHF>(bra, ket, v, d);
        Real acc[N];
        if (active)
            eval_quartet<LA, LB, LC, LD, Real, true, KL0, KL1, kFP64>(bra, ket, tb, tk, slice, acc, kfs, v.et, pr);
        else
        {
#pragma unroll
            for (int x = 0; x < N; ++x) acc[x] = Real(0);
        }
        bool leader = active;
        if (kSplit && g > 1)
        {
            for (int o = min(g, 32) >> 1; o > 0; o >>= 1)
#pragma unroll
                for (int x = 0; x < N; ++x) acc[x] += __shfl_xor_sync(0xffffffffu, acc[x], o);
            if (g >= 32)
            {
                // One quartet per warp or group of warps: its integrals through shared memory.
                Real* w = scratch + wib * N;
                if (lane == 0)
                    static_for<0, N>(
                        [&](auto E)
                        {
                            constexpr int e = decltype(E)::value;
                            constexpr Real an = Real(ang_norm(LA, e / CH / NB) * ang_norm(LB, (e / CH) % NB) *
                                                     ang_norm(LC, (KL0 + e % CH) / ND) * ang_norm(LD, (KL0 + e % CH) % ND));
                            w[e] = acc[e] * an;
                        });
                const int nw = g / 32;
                if (nw > 1)
                    __syncthreads();
                else
                    __syncwarp();
                if (wib % nw == 0 && active)
                {
                    for (int k = 1; k < nw; ++k)
                        for (int x = lane; x < N; x += 32) w[x] += w[k * N + x];
                    __syncwarp();
                    digest_shared<LA, LB, LC, LD, Real, UHF, KL0, KL1>(bra, ket, qt.bra == qt.ket, w, v);
                }
                if (nw > 1)
                    __syncthreads(); // the leading warp has read the others' integrals
                continue;
            }
            leader = active && r == 0;
            if (!leader)
            {
#pragma unroll
                for (int x = 0; x < N; ++x) acc[x] = Real(0);
            }
        }
        if (!kEarly)
            load_digest_d<LA, LB, LC, LD, Real, UHF>(bra, ket, v, d); // values the chunk does not read are never loaded
        const unsigned bra0 = __shfl_sync(0xffffffffu, qt.bra, 0);
        const bool bra_warp = __all_sync(0xffffffffu, qt.bra == bra0);
        digest_loaded<LA, LB, LC, LD, Real, UHF, KL0, KL1>(bra, ket, qt.bra == qt.ket, acc, v, d, leader, bra_warp);
    }
}

// Thread form: one launch processes the whole surviving list of one class; the list length is read on
// the device (written by the list builder), so a build needs no host round trip between kernels.
template <int LA, int LB, int LC, int LD, typename Real, bool UHF>
__global__ void __launch_bounds__(128) jk_class_kernel(const Quartet* __restrict__ list,
                                                       const unsigned long long* __restrict__ count, FockView v,
                                                       const Real* __restrict__ boys_slice, SplitArgs sp)
{
    constexpr int NCD = ncart(LC) * ncart(LD);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Real* slice                = reinterpret_cast<Real*>(smem_raw);
    const unsigned long long n = *count;
    if (static_cast<unsigned long long>(blockIdx.x) * 4 >= ((n + 31) >> 5) * static_cast<unsigned long long>(sp.smax))
        return;
    stage_boys<Real, boys_slice_size<Real>()>(boys_slice, slice);
    class_body<LA, LB, LC, LD, Real, UHF, 0, NCD>(list, n, v, slice, slice + boys_slice_size<Real>(), sp);
}

// Store mode of the thread classes: one thread per quartet writes its contracted integrals (the Schwartz
// bounds, stored integrals and single blocks).  It stays on the BoysGrid slice and one lane per quartet: the
// kets of a list are sorted by Q, copies of one molecule have Q equal up to the last bits, and which of
// them share a warp decides the rounding of the FP32 sums of a mixed build; the Q of one basis and
// geometry is therefore kept bit for bit.
template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(128) jk_store_kernel(const Quartet* __restrict__ list,
                                                       const unsigned long long* __restrict__ count, FockView v,
                                                       const double* __restrict__ boys_slice)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* slice              = reinterpret_cast<double*>(smem_raw);
    const unsigned long long n = *count;
    if (static_cast<unsigned long long>(blockIdx.x) * blockDim.x >= n)
        return;
    stage_boys<double>(boys_slice, slice);
    constexpr int N = ncart(LA) * ncart(LB) * ncart(LC) * ncart(LD);
    const double* tb = static_cast<const double*>(v.pptab[pair_class(LA, LB)]);
    const double* tk = static_cast<const double*>(v.ksoa[pair_class(LC, LD)]);
    for (unsigned long long q = static_cast<unsigned long long>(blockIdx.x) * blockDim.x + threadIdx.x; q < n;
         q += static_cast<unsigned long long>(gridDim.x) * blockDim.x)
    {
        const Quartet qt = list[q];
        double acc[N];
        eval_quartet<LA, LB, LC, LD, double, true>(v.pairs[qt.bra], v.pairs[qt.ket], tb, tk, slice, acc,
                                                   v.kfs[pair_class(LC, LD)]);
        static_for<0, N>(
            [&](auto E)
            {
                constexpr int e  = decltype(E)::value;
                constexpr int NB = ncart(LB), NC = ncart(LC), ND = ncart(LD), NCD = NC * ND;
                constexpr double an = ang_norm(LA, e / NCD / NB) * ang_norm(LB, (e / NCD) % NB)
                                    * ang_norm(LC, (e % NCD) / ND) * ang_norm(LD, e % ND);
                v.store[q * N + e] = acc[e] * an;
            });
    }
}

// Ket-chunked thread form: one thread per (shell quartet, chunk of CH ket Cartesian components).  For the
// d-containing classes a thread cannot hold a whole quartet's G[HAB][NCD] and ERI[NAB][NCD] in registers;
// restricted to CH ket components the thread keeps R, G[HAB][CH] and ERI[NAB][CH] in registers, with every
// loop unrolled at compile time, and digests the integrals of its chunk (the bra Coulomb block summed over
// the warp as in the thread form; the exchange and ket Coulomb elements its chunk reaches).  Each chunk
// is its own launch over the whole list (jk_class_chunk_kernel<..., KL0, KL1>), so that every SM runs one
// chunk's unrolled code at a time: with the chunks of a quartet in neighbouring blocks of one launch the
// resident blocks of an SM ran different chunk bodies and stalled on instruction fetch (ncu: 30 cycles
// per issued instruction).  Each chunk recomputes the Boys values and R of its quartet, which buys full
// lanes and no shared-memory round trips; the list and the records are re-read per chunk from L2.

// Chunks of CH ket components of a (LC LD) ket.
template <int LC, int LD, int CH> __host__ __device__ constexpr int num_chunks()
{
    return (ncart(LC) * ncart(LD) + CH - 1) / CH;
}

// One chunk, ket components [KL0, KL1), of every quartet of the list.
template <int LA, int LB, int LC, int LD, typename Real, bool UHF, int KL0, int KL1>
__global__ void __launch_bounds__(128) jk_class_chunk_kernel(const Quartet* __restrict__ list,
                                                             const unsigned long long* __restrict__ count, FockView v,
                                                             const Real* __restrict__ boys_slice, SplitArgs sp)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Real* slice                = reinterpret_cast<Real*>(smem_raw);
    const unsigned long long n = *count;
    if (static_cast<unsigned long long>(blockIdx.x) * 4 >= ((n + 31) >> 5) * static_cast<unsigned long long>(sp.smax))
        return;
    stage_boys<Real, boys_slice_size<Real>()>(boys_slice, slice);
    class_body<LA, LB, LC, LD, Real, UHF, KL0, KL1>(list, n, v, slice, slice + boys_slice_size<Real>(), sp);
}

// Digestion of stored integrals (the stored-integral SCF): integral blocks written once in store mode
// (row-major [ij][kl] per quartet, angular factors included) are digested with full densities every
// build.  Ket-chunked like jk_class_chunk_kernel so that the integrals and partial sums of a thread stay
// in registers: a thread digests ket components [KL0, KL1) of one quartet.
template <int LA, int LB, int LC, int LD, bool UHF, int KL0, int KL1>
__device__ __forceinline__ void stored_body(const Quartet* __restrict__ list, unsigned long long n, const FockView& v,
                                            const double* __restrict__ store, unsigned qb, unsigned nqb)
{
    constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
    constexpr int NAB = NA * NB, NCD = NC * ND, CH = KL1 - KL0;
    using DD       = DigestD<LA, LB, LC, LD, double, UHF>;
    const int lane = threadIdx.x & 31;
    for (unsigned long long base = static_cast<unsigned long long>(qb) * blockDim.x + (threadIdx.x & ~31u); base < n;
         base += static_cast<unsigned long long>(nqb) * blockDim.x)
    {
        const unsigned long long q = base + lane;
        const bool active          = q < n;
        const Quartet qt           = list[active ? q : base];
        const PairRec bra          = v.pairs[qt.bra];
        const PairRec ket          = v.pairs[qt.ket];
        double acc[NAB * CH];
        const double* __restrict__ blk = store + (active ? q : base) * static_cast<unsigned long long>(NAB * NCD);
        static_for<0, NAB>(
            [&](auto IJ)
            {
                constexpr int ij = decltype(IJ)::value;
                static_for<KL0, KL1>(
                    [&](auto KLx)
                    {
                        constexpr int kl = decltype(KLx)::value;
                        acc[ij * CH + (kl - KL0)] = active ? blk[ij * NCD + kl] : 0.0;
                    });
            });
        DD d;
        load_digest_d<LA, LB, LC, LD, double, UHF>(bra, ket, v, d);
        const unsigned bra0 = __shfl_sync(0xffffffffu, qt.bra, 0);
        const bool bra_warp = __all_sync(0xffffffffu, qt.bra == bra0);
        digest_loaded<LA, LB, LC, LD, double, UHF, KL0, KL1, true>(bra, ket, qt.bra == qt.ket, acc, v, d, active, bra_warp);
    }
}

// Ket components per thread of the stored digestion: at most 36 integrals per thread.
template <int LA, int LB, int LC, int LD> __host__ __device__ constexpr int stored_chunk()
{
    constexpr int NAB = ncart(LA) * ncart(LB), NCD = ncart(LC) * ncart(LD);
    constexpr int c   = 36 / NAB > 0 ? 36 / NAB : 1;
    return c < NCD ? c : NCD;
}

template <int LA, int LB, int LC, int LD, bool UHF>
__global__ void __launch_bounds__(128) jk_stored_kernel(const Quartet* __restrict__ list, unsigned long long n,
                                                        FockView v, const double* __restrict__ store)
{
    constexpr int NCD = ncart(LC) * ncart(LD), CH = stored_chunk<LA, LB, LC, LD>(), NCH = num_chunks<LC, LD, CH>();
    const unsigned qb = blockIdx.x / NCH, nqb = gridDim.x / NCH;
    const int chunk   = static_cast<int>(blockIdx.x % NCH);
    if (qb >= nqb || static_cast<unsigned long long>(qb) * blockDim.x >= n)
        return;
    static_for<0, NCH>(
        [&](auto C)
        {
            constexpr int c = decltype(C)::value;
            if (chunk == c)
                stored_body<LA, LB, LC, LD, UHF, c * CH, (c * CH + CH < NCD ? c * CH + CH : NCD)>(list, n, v, store, qb,
                                                                                                nqb);
        });
}

} // namespace hfg
