// Kernel instantiations and launchers of ONE shell-quartet class.  The build compiles this file four
// times per class, -DHFG_QCLASS=<0..20> -DHFG_PART=<0..3>: part 0 the RHF FP64 Fock kernels (with the store and
// stored-integral kernels and the form mask), part 1 the FP32 Fock kernels, part 2 the gradient kernels, part 3
// the UHF FP64 Fock kernels, so that the 84 units compile in parallel and the largest class does not
// serialise the build.
#include "engine.h"
#include "eri_grad.cuh"
#include "eri_group.cuh"

#ifndef HFG_QCLASS
#error "compile with -DHFG_QCLASS=<quartet class>"
#endif
#ifndef HFG_PART
#error "compile with -DHFG_PART=<0: RHF FP64, 1: FP32, 2: gradient, 3: UHF FP64 kernels>"
#endif

namespace hfg
{
namespace
{
constexpr int QC = HFG_QCLASS;
constexpr int bra_class()
{
    int p = 0;
    while ((p + 1) * (p + 2) / 2 <= QC) ++p;
    return p;
}
constexpr int P1 = bra_class();
constexpr int P2 = QC - P1 * (P1 + 1) / 2;
constexpr int LA = pair_class_l1(P1), LB = pair_class_l2(P1), LC = pair_class_l1(P2), LD = pair_class_l2(P2);
constexpr int NAB = ncart(LA) * ncart(LB), NCD = ncart(LC) * ncart(LD);
constexpr int L   = LA + LB + LC + LD;
// Classes with the warp-cooperative form instead of the thread form (whose ptxas stack frame would exceed ~1.2 KB in
// sm_103a code at -O3):
//   FP64: (dp|pp) (dp|ds) (dp|dp) (dd|ps) (dd|pp) (dd|ds) (dd|dp) (dd|dd)   = classes 12-14, 16-20
//   FP32: (dp|dp) (dd|pp) (dd|ds) (dd|dp) (dd|dd)                           = classes 14, 17-20
// In FP64 all but (dd|dd) run the chunk form below; the warp form evaluates their stored integrals.
constexpr bool warp_form(bool fp32)
{
    return fp32 ? (QC == 14 || QC >= 17) : (QC == 12 || QC == 13 || QC == 14 || QC >= 16);
}
// The primitive-parallel group form exists for the small, contracted classes (L <= 3, <= 27 integrals).
constexpr bool kGroup = (L <= 3) && (NAB * NCD <= 27);
// FP32 classes whose thread form sits at the 255-register limit ((dp|ps), (dp|pp), (dp|ds), (dd|ps): one or
// two blocks per SM) also compile the warp form, and the autotuner times both.
constexpr bool dual_form(bool fp32) { return fp32 && (QC == 11 || QC == 12 || QC == 13 || QC == 16); }
// Ket-chunked thread form (FP32 d classes): ket components per thread, chosen so that R, G[HAB][CH] and
// ERI[NAB][CH] stay in registers (HL + (HAB + NAB) * CH floats well below 255); 0 = not compiled.
//   (dp|pp) (dp|ds): 3   (dp|dp): 2   (dd|ps) (dd|pp) (dd|ds) (dd|dp): 1
// In FP64 (dp|pp) (dp|ds) (dp|dp): 3   (dd|ps) (dd|pp) (dd|ds) (dd|dp): 1; what does not fit the registers
// spills to L1, whose traffic (two wavefronts per warp and value) hides behind the FP64 pipe (16 SM cycles per
// warp instruction).
constexpr int chunk_width(bool fp32)
{
    if (!fp32)
        return (QC >= 12 && QC <= 14) ? 3 : (QC >= 16 && QC <= 19) ? 1 : 0;
    return (QC == 12 || QC == 13) ? 3 : QC == 14 ? 2 : (QC >= 16 && QC <= 19) ? 1 : 0;
}
// The form a launch with form 0 runs (before or without autotuning): the chunked form where the tuner
// keeps it at full size ((H2O)_64/6-31G**: (dp|pp), (dp|ds), (dp|dp), (dd|pp), (dd|ds), (dd|dp) in FP32; in FP64
// wherever it is compiled, at every size: an FP64 build of (H2O)_27/6-31G** takes 346 ms with the warp form and
// 35 / 29 / 18 / 12 ms less with (dp|pp) / (dp|ds) / (dp|dp) / (dd|ps) chunked, whose lanes are all busy), else
// warp or thread.
constexpr int default_form(bool fp32)
{
    const bool chunk = fp32 ? (QC == 12 || QC == 13 || QC == 14 || (QC >= 17 && QC <= 19)) : chunk_width(false) > 0;
    return chunk ? kFormChunk : (warp_form(fp32) ? kFormWarp : kFormThread);
}
constexpr unsigned form_mask(bool fp32)
{
    return (warp_form(fp32) || dual_form(fp32) ? (1u << kFormWarp) : 0u) |
           (!warp_form(fp32) || dual_form(fp32) ? (1u << kFormThread) : 0u) | (kGroup ? (1u << kFormGroup) : 0u) |
           (chunk_width(fp32) > 0 ? (1u << kFormChunk) : 0u);
}

// The split of a launch (SplitArgs): eight warps per SM fill it in FP64 (two per scheduler; the FP64 pipe takes a
// warp instruction every 64 cycles of one).  FP32 lists are not split.
template <typename Real> SplitArgs split_args(const ClassLaunch& c)
{
    SplitArgs s;
    // FP32 windows are short (some 10 us): four at a time, which also keep their bra's rows in L1.
    if (sizeof(Real) == 4)
    {
        s.run = 4;
        return s;
    }
    s.lanes     = static_cast<unsigned>(c.num_sms) * 256u;
    s.prims     = c.prims;
    s.prims_dev = c.prims_dev;
    return s;
}

// Sets the split for the list's longest quartet (pmax) and the order its items are taken in, for `cap` resident
// blocks that take `per_block` windows or groups each, and at most `windows` of them; returns the blocks to launch.
// Up to four waves of blocks go round robin, more through the counter `next`; `expected` windows decide that (a captured
// build's grid holds every quartet that the thresholds allow, its lists a tenth of them, and in runs of four windows
// those kept a quarter of the warps busy: 2.22 ms a replay of the mixed build of (H2O)_4/6-31G**, 1.79 ms eager).
inline unsigned long long plan_items(SplitArgs& s, bool split, unsigned long long pmax, unsigned long long windows,
                                     unsigned long long expected, unsigned per_block, unsigned long long cap,
                                     unsigned long long* next, cudaStream_t stream, cudaError_t& err)
{
    err             = cudaSuccess;
    auto warps_for = [&](bool queued, int most) {
        int w = 1;
        if (split)
            while (w < most && w * split_share(s.prims, s.lanes, queued) < pmax) w <<= 1;
        return w;
    };
    s.smax                  = warps_for(false, 128);
    unsigned long long need = (windows * s.smax + per_block - 1) / per_block;
    if (next == nullptr || (expected * s.smax + per_block - 1) / per_block <= 4 * cap)
    {
        s.run = 1;
        return need < cap ? need : cap;
    }
    // Eight takers a window at most: the slices beyond a window's own G are empty.
    s.smax = warps_for(true, 32);
    s.run  = s.smax >= 8 ? s.smax / 8 : s.run;
    s.next = next;
    need   = (windows * s.smax + per_block - 1) / per_block;
    err    = cudaMemsetAsync(next, 0, sizeof(unsigned long long), stream);
    return need < cap ? need : cap;
}

inline unsigned long long expected_windows(const ClassLaunch& c) { return ((c.listed != 0 ? c.listed : c.count_host) + 31) / 32; }

// Allows the kernel its shared memory and asks how many of its blocks an SM holds, once per engine (`slot`, zero
// before): the two calls cost more host time than the launch, 72 times in a build of two waters.
template <typename Kern> cudaError_t resident_blocks(Kern kern, int threads, size_t smem, int* slot, int& per_sm)
{
    if (slot != nullptr && *slot > 0)
    {
        per_sm = *slot;
        return cudaSuccess;
    }
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
    per_sm = per_sm > 0 ? per_sm : 1;
    if (slot != nullptr && e == cudaSuccess)
        *slot = per_sm;
    return e;
}

// Resident blocks per SM a grid may take: the occupancy limit times the share, at least one.
inline unsigned long long resident(int per_sm, float share)
{
    const int r = static_cast<int>(static_cast<float>(per_sm > 0 ? per_sm : 1) * share);
    return static_cast<unsigned long long>(r > 0 ? r : 1);
}

// Store mode: thread per quartet, or warp per quartet for the classes whose FP64 warp form is compiled.
template <bool Warp> cudaError_t launch_store(const ClassLaunch& c)
{
    size_t smem = sizeof(double) * BoysGrid<double>::kPoints * BoysGrid<double>::kRow;
    if constexpr (Warp)
        smem += sizeof(double) * WarpLayout<LA, LB, LC, LD, double>::kPerWarp * kWarpKernelWarps;
    auto kern = [] {
        if constexpr (Warp)
            return jk_class_warp_kernel<LA, LB, LC, LD, double, false>;
        else
            return jk_store_kernel<LA, LB, LC, LD>;
    }();
    constexpr unsigned threads = Warp ? 32 * kWarpKernelWarps : 128, per_block = Warp ? kWarpKernelWarps : 128;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess)
        return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, static_cast<int>(threads), smem);
    if (e != cudaSuccess)
        return e;
    const unsigned long long need = (c.count_host + per_block - 1) / per_block;
    const unsigned long long cap  = static_cast<unsigned long long>(c.num_sms) * (per_sm > 0 ? per_sm : 1);
    const unsigned grid           = static_cast<unsigned>(need < cap ? need : cap);
    const double* slice           = static_cast<const double*>(c.boys_slice);
    if constexpr (Warp)
        kern<<<grid, threads, smem, c.stream>>>(c.list, c.count_dev, c.view, slice, c.tables);
    else
        kern<<<grid, threads, smem, c.stream>>>(c.list, c.count_dev, c.view, slice);
    return cudaGetLastError();
}

template <typename Real, bool UHF> cudaError_t launch_t(const ClassLaunch& c)
{
    constexpr bool kWarpForm = warp_form(sizeof(Real) == 4);
    if (c.count_host == 0)
        return cudaSuccess;
    if constexpr (sizeof(Real) == 8 && !UHF)
        if (c.view.store != nullptr)
            return launch_store<warp_form(false)>(c);
    const int form = c.form == 0 ? default_form(sizeof(Real) == 4) : c.form;
    if (!((form_mask(sizeof(Real) == 4) >> form) & 1u))
        return cudaErrorInvalidValue;
    // The thread and chunk forms stage the BoysFast slice in FP64, the others the BoysGrid slice.
    const size_t slice_bytes = sizeof(Real) * BoysGrid<Real>::kPoints * BoysGrid<Real>::kRow;
    constexpr size_t kFastBytes = sizeof(Real) * boys_slice_size<Real>();
    const Real* fast = static_cast<const Real*>(sizeof(Real) == 8 ? c.boys_fast : c.boys_slice);
    if constexpr (kGroup)
    {
        if (form == kFormGroup)
        {
            auto kern         = jk_class_group_kernel<LA, LB, LC, LD, Real, UHF>;
            const size_t smem = slice_bytes;
            int per_sm    = 0;
            cudaError_t e = resident_blocks(kern, 128, smem, c.occ ? c.occ + kMaxChunks + 2 : nullptr, per_sm);
            if (e != cudaSuccess)
                return e;
            const unsigned long long need = (c.count_host + 127) / 128; // 4 warps x 32-quartet windows
            const unsigned long long cap  = static_cast<unsigned long long>(c.num_sms) * resident(per_sm, c.share);
            kern<<<static_cast<unsigned>(need < cap ? need : cap), 128, smem, c.stream>>>(
                c.list, c.count_dev, c.view, static_cast<const Real*>(c.boys_slice));
            return cudaGetLastError();
        }
    }
    constexpr int kChunk = chunk_width(sizeof(Real) == 4);
    if constexpr (kChunk > 0)
    {
        if (form == kFormChunk)
        {
            // One launch per chunk of kChunk ket components, each over the whole list.
            constexpr int nch = num_chunks<LC, LD, kChunk>();
            cudaError_t err   = cudaSuccess;
            static_for<0, nch>(
                [&](auto C)
                {
                    constexpr int k0 = decltype(C)::value * kChunk;
                    constexpr int k1 = k0 + kChunk < NCD ? k0 + kChunk : NCD;
                    if (err != cudaSuccess)
                        return;
                    auto kern         = jk_class_chunk_kernel<LA, LB, LC, LD, Real, UHF, k0, k1>;
                    SplitArgs sp = split_args<Real>(c);
                    const size_t smem = kFastBytes + (sizeof(Real) == 8 ? sizeof(Real) * split_scratch<LA, LB, k0, k1>() : 0);
                    int per_sm = 0;
                    err = resident_blocks(kern, 128, smem, c.occ ? c.occ + decltype(C)::value : nullptr, per_sm);
                    if (err != cudaSuccess)
                        return;
                    const unsigned long long grid =
                        plan_items(sp, sizeof(Real) == 8, c.pmax, (c.count_host + 31) / 32, expected_windows(c), 4,
                                   static_cast<unsigned long long>(c.num_sms) * resident(per_sm, c.share),
                                   c.next ? c.next + decltype(C)::value : nullptr, c.stream, err);
                    if (err != cudaSuccess)
                        return;
                    kern<<<static_cast<unsigned>(grid), 128, smem, c.stream>>>(
                        c.list, c.count_dev, c.view, fast, sp);
                    err = cudaGetLastError();
                });
            return err;
        }
    }
    constexpr bool kHasWarp = kWarpForm || dual_form(sizeof(Real) == 4);
    constexpr bool kHasThread = !kWarpForm || dual_form(sizeof(Real) == 4);
    if constexpr (kHasWarp)
    {
        if (form == kFormWarp)
        {
            using W             = WarpLayout<LA, LB, LC, LD, Real>;
            const size_t smem   = slice_bytes + sizeof(Real) * W::kPerWarp * kWarpKernelWarps;
            auto kern           = jk_class_warp_kernel<LA, LB, LC, LD, Real, UHF>;
            int per_sm    = 0;
            cudaError_t e = resident_blocks(kern, 32 * kWarpKernelWarps, smem, c.occ ? c.occ + kMaxChunks + 1 : nullptr, per_sm);
            if (e != cudaSuccess)
                return e;
            const unsigned long long need = (c.count_host + kWarpKernelWarps - 1) / kWarpKernelWarps;
            const unsigned long long cap  = static_cast<unsigned long long>(c.num_sms) * resident(per_sm, c.share);
            const unsigned grid           = static_cast<unsigned>(need < cap ? need : cap);
            kern<<<grid, 32 * kWarpKernelWarps, smem, c.stream>>>(c.list, c.count_dev, c.view,
                                                                  static_cast<const Real*>(c.boys_slice), c.tables);
            return cudaGetLastError();
        }
    }
    if constexpr (kHasThread)
    {
        if (form == kFormThread)
        {
            auto kern           = jk_class_kernel<LA, LB, LC, LD, Real, UHF>;
            SplitArgs sp        = split_args<Real>(c);
            const size_t smem   = kFastBytes + (sizeof(Real) == 8 ? sizeof(Real) * split_scratch<LA, LB, 0, NCD>() : 0);
            int per_sm    = 0;
            cudaError_t e = resident_blocks(kern, 128, smem, c.occ ? c.occ + kMaxChunks : nullptr, per_sm);
            if (e != cudaSuccess)
                return e;
            const unsigned long long grid =
                plan_items(sp, sizeof(Real) == 8, c.pmax, (c.count_host + 31) / 32, expected_windows(c), 4,
                           static_cast<unsigned long long>(c.num_sms) * resident(per_sm, c.share), c.next, c.stream, e);
            if (e != cudaSuccess)
                return e;
            kern<<<static_cast<unsigned>(grid), 128, smem, c.stream>>>(c.list, c.count_dev, c.view, fast, sp);
            return cudaGetLastError();
        }
    }
    return cudaErrorInvalidValue;
}
} // namespace

#define HFG_CAT2(a, b) a##b
#define HFG_CAT(a, b) HFG_CAT2(a, b)

#if HFG_PART == 3
cudaError_t HFG_CAT(launch_class64u_, HFG_QCLASS)(const ClassLaunch& c) { return launch_t<double, true>(c); }
#elif HFG_PART == 0
cudaError_t HFG_CAT(launch_class64u_, HFG_QCLASS)(const ClassLaunch& c);
cudaError_t HFG_CAT(launch_class64_, HFG_QCLASS)(const ClassLaunch& c)
{
    return c.uhf ? HFG_CAT(launch_class64u_, HFG_QCLASS)(c) : launch_t<double, false>(c);
}

cudaError_t HFG_CAT(launch_stored_, HFG_QCLASS)(const StoredLaunch& c)
{
    if (c.count == 0)
        return cudaSuccess;
    constexpr int nch = num_chunks<LC, LD, stored_chunk<LA, LB, LC, LD>()>();
    auto kern = c.uhf ? jk_stored_kernel<LA, LB, LC, LD, true> : jk_stored_kernel<LA, LB, LC, LD, false>;
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 128, 0);
    if (e != cudaSuccess)
        return e;
    const unsigned long long need = (c.count + 127) / 128;
    unsigned long long cap = static_cast<unsigned long long>(c.num_sms) * (per_sm > 0 ? per_sm : 1) / nch;
    if (cap < 1)
        cap = 1;
    const unsigned long long qblocks = need < cap ? need : cap;
    kern<<<static_cast<unsigned>(qblocks * nch), 128, 0, c.stream>>>(c.list, c.count, c.view, c.store);
    return cudaGetLastError();
}

// Bits 0-15: compiled forms; 16-23: the default form; 24-31: kernel launches of one chunk-form launch.
unsigned HFG_CAT(class_form_mask_, HFG_QCLASS)(bool fp32)
{
    const unsigned nch = chunk_width(fp32) > 0 ? static_cast<unsigned>((NCD + chunk_width(fp32) - 1) / chunk_width(fp32)) : 0u;
    return form_mask(fp32) | (static_cast<unsigned>(default_form(fp32)) << 16) | (nch << 24);
}
#elif HFG_PART == 1
cudaError_t HFG_CAT(launch_class32_, HFG_QCLASS)(const ClassLaunch& c)
{
    return c.uhf ? launch_t<float, true>(c) : launch_t<float, false>(c);
}
#else
namespace
{
// Thread-per-quartet gradient form, by the values a thread holds at its peak (GradThread).  What does not fit the
// registers spills to L1; the lane-group form keeps half its lanes idle in its dynamic index loops.
//   FP64, ss or ps ket (single-pass form): every class ((dd|ps), 465 values, is kept in local memory by ptxas and
//     still takes 5.5 ms of a (H2O)_16 6-31G** gradient against 13.6 in the lane-group form);
//   FP64, other kets: (ds|pp), (ds|ds) and (pp|pp) ((H2O)_8 cc-pVDZ 18.5 -> 15.5 ms, (H2O)_16 9.0 -> 9.8);
//   FP32: up to 160 values ((pp|ps) (ds|ps) (dp|ss) and smaller), and to 300 with d shells: (ds|pp) (ds|ds) (dp|ps)
//     (dd|ss), 38 -> 7 ms of a (H2O)_16 gradient.  (pp|pp) is not in it: with it mixed gradients in 6-31G take
//     5.2 ms for 5.6 ((H2O)_8) and 66.4 for 72.1 ((H2O)_27), but its error against the lane-group form is not measured.
template <typename Real> constexpr bool grad_thread_form()
{
    using W = GradThread<LA, LB, LC, LD>;
    if (sizeof(Real) == 8 && grad_single_pass(LC, LD))
        return W::kValuesSingle <= 480;
    return W::kValues <= (sizeof(Real) == 8 ? 410 : LA == 2 ? 300 : 160);
}

// The split of a gradient launch: `width` lanes work on one slice together.
template <typename Real> SplitArgs grad_split(const GradLaunch& c, int width)
{
    SplitArgs s;
    s.run = width == 1 ? 1 : 4;
    if (sizeof(Real) == 4)
        return s;
    s.lanes = static_cast<unsigned>(c.num_sms) * 256u / width;
    s.prims = c.prims;
    return s;
}

template <typename Real> cudaError_t launch_grad_thread(const GradLaunch& c)
{
    const size_t smem = sizeof(Real) * boys_slice_size<Real>();
    auto kern         = grad_thread_kernel<LA, LB, LC, LD, Real>;
    int per_sm    = 0;
    cudaError_t e = resident_blocks(kern, 128, smem, c.occ, per_sm);
    if (e != cudaSuccess)
        return e;
    SplitArgs sp                  = grad_split<Real>(c, 1);
    const unsigned long long grid = plan_items(sp, sizeof(Real) == 8, c.pmax, (c.count + 31) / 32, (c.count + 31) / 32, 4,
                                               static_cast<unsigned long long>(c.num_sms) * (per_sm > 0 ? per_sm : 1), c.next,
                                               c.stream, e);
    if (e != cudaSuccess)
        return e;
    kern<<<static_cast<unsigned>(grid), 128, smem, c.stream>>>(
        c.list, c.count, c.view, static_cast<const Real*>(c.boys_slice), sp);
    return cudaGetLastError();
}

template <typename Real> cudaError_t launch_grad_t(const GradLaunch& c)
{
    if constexpr (grad_thread_form<Real>())
        if (!c.group_form)
            return launch_grad_thread<Real>(c);
    using W           = GradLayout<LA, LB, LC, LD>;
    const size_t smem = sizeof(Real) * (boys_slice_size<Real>() + W::kPerWarp * kGradWarps);
    auto kern         = grad_class_kernel<LA, LB, LC, LD, Real>;
    int per_sm    = 0;
    cudaError_t e = resident_blocks(kern, 32 * kGradWarps, smem, c.occ + 1, per_sm);
    if (e != cudaSuccess)
        return e;
    constexpr unsigned per_block = kGradWarps * (32 / W::kGroup); // quartets in flight per block
    SplitArgs sp                  = grad_split<Real>(c, W::kGroup);
    const unsigned long long grid = plan_items(sp, sizeof(Real) == 8, c.pmax, c.count, c.count, per_block,
                                               static_cast<unsigned long long>(c.num_sms) * (per_sm > 0 ? per_sm : 1), c.next,
                                               c.stream, e);
    if (e != cudaSuccess)
        return e;
    kern<<<static_cast<unsigned>(grid), 32 * kGradWarps, smem, c.stream>>>(
        c.list, c.count, c.view, static_cast<const Real*>(c.boys_slice), c.tables, sp);
    return cudaGetLastError();
}
} // namespace

cudaError_t HFG_CAT(launch_grad_, HFG_QCLASS)(const GradLaunch& c)
{
    if (c.count == 0)
        return cudaSuccess;
    return c.fp32 ? launch_grad_t<float>(c) : launch_grad_t<double>(c);
}
#endif
} // namespace hfg
