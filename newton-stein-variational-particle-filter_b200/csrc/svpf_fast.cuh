// svpf_fast.cuh -- the pair sums of a Stein iteration in close to O(N).
//
// Particles are scalars, so every sum over pairs that the iteration needs (the
// mixture prior's exponentials, the IMQ kernel's attraction, repulsion and
// Hessian weights) is a smooth function of one variable.  The particles are
// binned into panels of width kPanelW bandwidths.  A panel with more than kP
// particles is stood for by kP points: the sums over its particles become
// sums over its points with interpolated weights, and the sums at its
// particles are interpolated from the sums at its points; a panel with fewer
// particles keeps them as they are.  The pair loops then run over M points
// (150 to 300 of them at N = 512 .. 4096) instead of N particles.
//
// Interpolation is by degree kP - 1 polynomials in the Chebyshev basis.  The
// IMQ kernel 1 / (1 + u^2) has its poles at u = +-i: on a panel of half-width
// 0.375 its expansion falls by 5.5 per degree.  With kP = 12 the largest error
// of an interpolated kernel value is 2.5e-9 for K, 1.4e-8 for u K^2, 5.9e-8 for
// K (3 - 4K) (the Hessian's) and 2.0e-7 for K^2 (3 - 4K) (the KSD's, three
// poles at each end), on values of up to 1.  The points are
// near-Chebyshev offsets rounded to 2^-14 bandwidths, so that point positions
// and their differences are exact in FP32 and the basis change matrix
// (inverted in rational arithmetic for those very offsets) belongs to them:
// the sums come out as near to FP64 as the direct loops', whose longer FP32
// accumulations weigh more than the interpolation (measured: 3e-7 rms against
// 5e-7 at N = 4096).
//
// Two sums are not smooth:
//  * the Hessian's sum K^2 |3u^2 - 1| has a kink at u = 1/sqrt(3).  It is the
//    smooth sum K (3 - 4K) plus twice the sum of K (4K - 3) over the window
//    |u| < 1/sqrt(3).  Fine bins of an eighth of a panel give the window's
//    ends, whose particles are summed one by one; the bins between count
//    through the panels' weights accumulated up to each fine bin (prefix).
//  * the mixture's log-weights span hundreds of powers of two.  Sums at a
//    panel's points are scaled by 2^(quadratic of the point's offset), the
//    curvature of one Gaussian and a tilt that levels the panel's ends, before
//    they are interpolated (numerator and denominator apart: both entire).
//    Where the expansion has not converged -- a gap of many sigma between the
//    prior means -- and at points far outside the means, the sum goes over the
//    means themselves that matter there, which stay sorted in global memory.
//
// A tick whose particles do not fit these tables (kFineBins bins, kMaxPts
// points) finishes with the direct loops.
//
// Measured on B200, two CTAs per SM: an iteration of N = 4096 particles takes
// 250 k cycles (the window 88 k of them: about 36 kernel values per particle;
// point sums 31 k, rows 27 k, mixture points 22 k, binning 16 k, weights 12 k)
// against 4.7 M with the sweeps, one of N = 512 55 k against 100 k.  The batch
// tick of 4096 filters (N 256 to 4096) went from 83.7 to 4.8 ms, its first
// tick from 83 to 12 ms, 300 filters of 100 to 1500 particles from 4.0 to
// 0.37 ms (CTAs of 512 threads), one filter of 4096 on a cluster from 0.68 to
// 0.22 ms.  The two-factor tick's transports (no mixture, no Hessian) take the
// same way: a request round of 200 instruments of 256 to 2048 particles went
// from 7.5 to 1.9 ms, bound by the ticks of N = 2048.
#pragma once

#include "svpf_device.cuh"

namespace svpf {

constexpr int kMaxWarps = 16;       // CTAs of 8 or 16 warps
constexpr int kBinWarps = 8;        // warps that rank particles
constexpr int kP = 12;              // points of a panel
constexpr int kFine = 8;            // fine bins of a transport panel
constexpr int kFineBins = 1024;
constexpr int kFineZero = kFineBins / 2;   // bin that starts at coordinate 0
constexpr float kFineW = 0.09375f;  // fine bin in bandwidths (in scaled units for the prior means)
constexpr float kPanelW = kFine * kFineW;
constexpr float kInvHalfW = 2.0f / kPanelW;
constexpr float kFineScale = 1.0f / kFineW;
constexpr int kMaxPts = 512;             // points of the transport
constexpr int kMaxComp = kMaxPts / kP;   // its interpolated panels
constexpr int kMixPts = 1408;            // points the mixture is summed at
constexpr int kMixComp = kMixPts / kP;
constexpr int kMaxSrc = 1280;            // points standing for the prior means
constexpr int kPtRows = 11;              // arrays of kMaxPts floats
constexpr int kMaxPts2f = 1120;          // two factors: 5 arrays of up to this many
constexpr float kKink = 0.57735026918962576f;   // 3 u^2 = 1
// Widest panel in the mixture's scaled units: at half-width 0.75 the Gaussian
// sums interpolate to 6e-9 with kP points (2e-7 at half-width 1).
constexpr float kMixPanelMax = 1.5f;
// Last two Chebyshev coefficients of a panel's mixture sums, relative to the
// first: rounding leaves 1e-7, and an expansion that has fallen to this has
// 1e-7 left beyond them.
constexpr float kMixTail = 6e-7f;
// A prior mean further than this (scaled units) from a point weighs less than
// 2^-26 of the sum when some mean lies within 3 units (N <= 8192).
constexpr float kMixReach = 7.0f;

// Point offsets from the panel's centre, panel width kPanelW.
__device__ const float kNode[kP] = {
    0.37176513671875f, 0.346435546875f, 0.2974853515625f,
    0.228271484375f, 0.14349365234375f, 0.0489501953125f,
    -0.0489501953125f, -0.14349365234375f, -0.228271484375f,
    -0.2974853515625f, -0.346435546875f, -0.37176513671875f};
// Basis change for those points: coefficient k = sum_q kBasis[k][q] value_q,
// and the weight of point q for a particle at t is sum_k kBasis[k][q] T_k(t).
__device__ const float kBasis[kP * kP] = {
    8.352009291e-02f, 8.311931339e-02f, 8.341916710e-02f, 8.326756260e-02f, 8.335347356e-02f, 8.332039043e-02f,
    8.332039043e-02f, 8.335347356e-02f, 8.326756260e-02f, 8.341916710e-02f, 8.311931339e-02f, 8.352009291e-02f,
    1.656212610e-01f, 1.535113938e-01f, 1.324545355e-01f, 1.012401522e-01f, 6.394615259e-02f, 2.158509742e-02f,
    -2.158509742e-02f, -6.394615259e-02f, -1.012401522e-01f, -1.324545355e-01f, -1.535113938e-01f, -1.656212610e-01f,
    1.613449381e-01f, 1.173976594e-01f, 4.331251417e-02f, -4.328051283e-02f, -1.177689899e-01f, -1.610056090e-01f,
    -1.610056090e-01f, -1.177689899e-01f, -4.328051283e-02f, 4.331251417e-02f, 1.173976594e-01f, 1.613449381e-01f,
    1.543230023e-01f, 6.328772335e-02f, -6.355818846e-02f, -1.541628722e-01f, -1.538057420e-01f, -6.390707310e-02f,
    6.390707310e-02f, 1.538057420e-01f, 1.541628722e-01f, 6.355818846e-02f, -6.328772335e-02f, -1.543230023e-01f,
    1.446385927e-01f, -4.637017693e-04f, -1.441532077e-01f, -1.444047547e-01f, 6.153561787e-05f, 1.443215358e-01f,
    1.443215358e-01f, 6.153561787e-05f, -1.444047547e-01f, -1.441532077e-01f, -4.637017693e-04f, 1.446385927e-01f,
    1.324967901e-01f, -6.425586294e-02f, -1.649764687e-01f, -2.187329603e-02f, 1.541217348e-01f, 1.012962171e-01f,
    -1.012962171e-01f, -1.541217348e-01f, 2.187329603e-02f, 1.649764687e-01f, 6.425586294e-02f, -1.324967901e-01f,
    1.180690728e-01f, -1.182590450e-01f, -1.175965671e-01f, 1.177751560e-01f, 1.178877478e-01f, -1.178763646e-01f,
    -1.178763646e-01f, 1.178877478e-01f, 1.177751560e-01f, -1.175965671e-01f, -1.182590450e-01f, 1.180690728e-01f,
    1.016391313e-01f, -1.543481275e-01f, -2.143876108e-02f, 1.650471077e-01f, -6.365622145e-02f, -1.323339924e-01f,
    1.323339924e-01f, 6.365622145e-02f, -1.650471077e-01f, 2.143876108e-02f, 1.543481275e-01f, -1.016391313e-01f,
    8.345565005e-02f, -1.669232374e-01f, 8.358207442e-02f, 8.316110139e-02f, -1.666038209e-01f, 8.332823242e-02f,
    8.332823242e-02f, -1.666038209e-01f, 8.316110139e-02f, 8.358207442e-02f, -1.669232374e-01f, 8.345565005e-02f,
    6.386713621e-02f, -1.541706206e-01f, 1.542113518e-01f, -6.401422600e-02f, -6.359937329e-02f, 1.538240886e-01f,
    -1.538240886e-01f, 6.359937329e-02f, 6.401422600e-02f, -1.542113518e-01f, 1.541706206e-01f, -6.386713621e-02f,
    4.317674795e-02f, -1.179310734e-01f, 1.610878894e-01f, -1.610950875e-01f, 1.179312537e-01f, -4.316973012e-02f,
    -4.316973012e-02f, 1.179312537e-01f, -1.610950875e-01f, 1.610878894e-01f, -1.179310734e-01f, 4.317674795e-02f,
    2.177622225e-02f, -6.382738858e-02f, 1.015309800e-01f, -1.323219542e-01f, 1.540981758e-01f, -1.653583677e-01f,
    1.653583677e-01f, -1.540981758e-01f, 1.323219542e-01f, -1.015309800e-01f, 6.382738858e-02f, -2.177622225e-02f};

// A partition of the fine bins into panels of fb = 2^sft bins.  A panel with
// more than kP particles is interpolated (comp lists those), the others keep
// their particles as points; pt[b] is a panel's first point, interpolated
// panels before the others, or in panel order (sources).
struct Panels {
    unsigned short* pt;
    unsigned short* comp;
    int sft;
    int nc, m;                // interpolated panels, points
    float narrow;             // kFine / fb
    __device__ __forceinline__ float centre(int b) const {   // exact: a multiple of half a fine bin
        return ((float)((b << sft) - kFineZero) + 0.5f * (float)(1 << sft)) * kFineW;
    }
    // Outliers share the first and the last panel, which therefore keep theirs.
    __device__ __forceinline__ bool interpolated(int b, int count) const {
        return count > kP && b > 0 && b < (kFineBins >> sft) - 1;
    }
    __device__ __forceinline__ float local(float x, int b) const { return (x - centre(b)) * (kInvHalfW * narrow); }
};

// Shared scalars, behind the tables: a static variable would take them from
// every kernel's dynamic shared memory limit (max_dyn_smem).
struct FastSh {
    unsigned scan[kMaxWarps];
    int over;                 // points do not fit
    int n_far;                // mixture points far from every mean, listed in pref's space
};

// Shared-memory tables of the fast sums (dynamic part: fast_table_floats()).
struct FastTab {
    float* basis;             // kBasis, then kNode
    float* pts;               // binning counters and ranks (into pref); mixture sums [4][kMixPts]: X, den, num, e; then
                              // [kPtRows][kMaxPts]: X, weights 1 / g / c, transport sums
    float* pref;              // [kMaxComp][kFine][kP] weights up to and including each fine bin
    float* src_x;             // the prior means' points (scaled units), in panel order
    float* src_w;
    unsigned short* fstart;   // [kFineBins + 1] first slot of each fine bin
    unsigned short* src_pt;   // [kFineBins / kFine + 1] first point of each panel of the prior means
    unsigned short* src_slot; // the same for the sorted means themselves
    unsigned short* pt;       // transport panels: first points, [kFineBins / kFine]
    unsigned short* comp;     // [kFineBins / kFine]
    unsigned short* mpt;      // mixture panels: first points, [kFineBins]
    unsigned short* mcomp;    // [kMixComp]
    unsigned char* bad;       // [kMixComp] mixture panel not interpolated
    FastSh* sh;
};
constexpr int kTabBasis = kP * kP + 16;
constexpr int kTabPts = kPtRows * kMaxPts;
constexpr int kTabPref = kMaxComp * kFine * kP;
// (an even number: FastSh follows)
constexpr int kTabShorts = (kFineBins + 8) + 2 * (kFineBins / kFine + 8) + 2 * (kFineBins / kFine) + kFineBins +
                           2 * kMixComp;
static_assert(kTabShorts % 2 == 0 && sizeof(FastSh) % sizeof(float) == 0, "FastSh behind the tables");
// binning counters and ranks take the points' space and the one behind it
static_assert(kMixPts / 2 <= kTabPref, "the list of far points takes pref's space");
static_assert(kBinWarps * kFineBins / 2 + SVPF_MAX_PARTICLES / 2 <= kTabPts + kTabPref && 4 * kMixPts <= kTabPts,
              "uses of the points' space");

// Without the mixture the binning ranks of many particles extend the points' space.
__host__ __device__ inline int fast_points_floats(int np, bool mixture) {
    const int bins = kBinWarps * kFineBins / 2 + np / 2;
    return mixture || bins < kTabPts ? kTabPts : bins;
}
__host__ __device__ inline int fast_table_floats(int np, bool mixture) {
    return round_up(kTabBasis + fast_points_floats(np, mixture) + kTabShorts / 2 + 8 +
                        (int)(sizeof(FastSh) / sizeof(float)) + (mixture ? kTabPref + 2 * kMaxSrc : 0), 16);
}

__device__ inline FastTab carve_fast(float* p, int np, bool mixture) {
    FastTab t;
    t.basis = p;
    p += kTabBasis;
    t.pts = p;
    p += fast_points_floats(np, mixture);
    t.pref = t.src_x = t.src_w = nullptr;
    if (mixture) {
        t.pref = p;
        p += kTabPref;
        t.src_x = p;
        p += kMaxSrc;
        t.src_w = p;
        p += kMaxSrc;
    }
    unsigned short* q = reinterpret_cast<unsigned short*>(p);
    t.fstart = q;
    q += kFineBins + 8;
    t.src_pt = q;
    q += kFineBins / kFine + 8;
    t.src_slot = q;
    q += kFineBins / kFine + 8;
    t.pt = q;
    q += kFineBins / kFine;
    t.comp = q;
    q += kFineBins / kFine;
    t.mpt = q;
    q += kFineBins;
    t.mcomp = q;
    q += kMixComp;
    t.bad = reinterpret_cast<unsigned char*>(q);
    t.sh = reinterpret_cast<FastSh*>(p + kTabShorts / 2);
    return t;
}

__device__ __forceinline__ void fast_load_tables(const FastTab& t) {
    for (int i = threadIdx.x; i < kP * kP + kP; i += blockDim.x) t.basis[i] = i < kP * kP ? kBasis[i] : kNode[i - kP * kP];
}

// Fine bin of coordinate x; outliers share the first and the last bin, NaN the first.
__device__ __forceinline__ int fine_bin(float x, float fs = kFineScale) {
    return __float2int_rd(fminf(fmaxf(x * fs, -(float)kFineZero), (float)(kFineBins - kFineZero) - 0.5f)) + kFineZero;
}

// Exclusive block scan of one packed value per thread; all: the total.
__device__ __forceinline__ unsigned block_scan(unsigned own, unsigned& all, FastSh& sh) {
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    unsigned inc = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
    }
    if (lane == 31) sh.scan[wp] = inc;
    __syncthreads();
    unsigned ex = inc - own;
    all = 0u;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
        const unsigned v = sh.scan[w];
        if (w < wp) ex += v;
        all += v;
    }
    return ex;
}

// Sorts the n coordinates x(i) into fine bins, within a bin by particle, so that
// the order and with it every later sum is reproducible: xs[slot], pidx[slot]
// (the particle) and fstart.  Each warp ranks its own stretch of particles
// with match_any, two groups of 32 at a time.  (Shared-memory atomics and a
// count of the smaller indices in the bin took twice as long at N = 4096; a
// ballot per bit instead of match_any 5 % longer.)  Ends with a barrier.
template <class FX>
__device__ __forceinline__ void fast_bin(FX x, int n, float fs, float* xs, unsigned short* pidx, const FastTab& t,
                                         FastSh& sh) {
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    unsigned short* hist = reinterpret_cast<unsigned short*>(t.pts);     // [kBinWarps][kFineBins]
    unsigned short* rank = hist + kBinWarps * kFineBins;                    // by particle
    {
        uint4* h4 = reinterpret_cast<uint4*>(hist);
        for (int i = tid; i < kBinWarps * kFineBins / 8; i += blockDim.x) h4[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    if (tid == 0) sh.over = sh.n_far = 0;
    __syncthreads();
    const int per = round_up((n + kBinWarps - 1) / kBinWarps, 32);
    const int lo = min(wp * per, n), hi = wp < kBinWarps ? min(lo + per, n) : lo;
    unsigned short* hw = hist + wp * kFineBins;
    const unsigned below = (1u << lane) - 1u;
    for (int base = lo; base < hi; base += 64) {
        const int i0 = base + lane, i1 = i0 + 32;
        const int f0 = i0 < hi ? fine_bin(x(i0), fs) : kFineBins, f1 = i1 < hi ? fine_bin(x(i1), fs) : kFineBins;
        const unsigned m0 = __match_any_sync(0xffffffffu, f0), m1 = __match_any_sync(0xffffffffu, f1);
        int at = 0;
        if (i0 < hi) at = hw[f0];
        __syncwarp();
        if (i0 < hi) {
            rank[i0] = (unsigned short)(at + __popc(m0 & below));
            if ((m0 & below) == 0u) hw[f0] = (unsigned short)(at + __popc(m0));
        }
        __syncwarp();
        if (i1 < hi) at = hw[f1];
        __syncwarp();
        if (i1 < hi) {
            rank[i1] = (unsigned short)(at + __popc(m1 & below));
            if ((m1 & below) == 0u) hw[f1] = (unsigned short)(at + __popc(m1));
        }
        __syncwarp();
    }
    __syncthreads();
    {
        // four fine bins for each of 256 threads: the warps' counts become their first slots
        const bool on = tid < kFineBins / 4;
        unsigned c4[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int w = 0; w < kBinWarps; ++w) {
            if (!on) break;
            const ushort4 v = reinterpret_cast<const ushort4*>(hist + w * kFineBins)[tid];
            c4[0] += v.x; c4[1] += v.y; c4[2] += v.z; c4[3] += v.w;
        }
        unsigned all;
        unsigned first = block_scan(c4[0] + c4[1] + c4[2] + c4[3], all, sh);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (!on) break;
            t.fstart[4 * tid + j] = (unsigned short)first;
            const unsigned next = first + c4[j];
            c4[j] = first;
            first = next;
        }
#pragma unroll
        for (int w = 0; w < kBinWarps; ++w) {
            if (!on) break;
            ushort4* h = reinterpret_cast<ushort4*>(hist + w * kFineBins) + tid;
            const ushort4 v = *h;
            *h = make_ushort4(c4[0], c4[1], c4[2], c4[3]);
            c4[0] += v.x; c4[1] += v.y; c4[2] += v.z; c4[3] += v.w;
        }
        if (tid == 0) t.fstart[kFineBins] = (unsigned short)n;
    }
    __syncthreads();
    for (int i = tid; i < n; i += blockDim.x) {
        const float v = x(i);
        const int slot = hist[i / per * kFineBins + fine_bin(v, fs)] + rank[i];
        xs[slot] = v;
        pidx[slot] = (unsigned short)i;
    }
    __syncthreads();
}

// The panels of 2^sft fine bins.  sh.over is set when there are more than
// max_comp interpolated ones or max_pts points.  Ends with a barrier.
__device__ inline Panels fast_panels(int sft, unsigned short* pt, unsigned short* comp, int max_comp, int max_pts,
                                     bool ordered, const FastTab& t, FastSh& sh) {
    Panels p;
    p.pt = pt;
    p.comp = comp;
    p.sft = sft;
    p.narrow = (float)kFine / (float)(1 << sft);
    const int np = kFineBins >> sft;
    const int per = np > kThreads ? np / kThreads : 1;   // panels per thread (of the first 256)
    const int b0 = threadIdx.x * per;
    unsigned own = 0u;   // interpolated panels, and from bit 16 points kept as they are
    if (b0 < np) {
        for (int b = b0; b < b0 + per; ++b) {
            const int c = t.fstart[(b + 1) << sft] - t.fstart[b << sft];
            own += p.interpolated(b, c) ? 1u : (unsigned)c << 16;
        }
    }
    unsigned all;
    unsigned ex = block_scan(own, all, sh);
    p.nc = (int)(all & 0xffffu);
    p.m = kP * p.nc + (int)(all >> 16);
    if (b0 < np) {
        for (int b = b0; b < b0 + per; ++b) {
            const int c = t.fstart[(b + 1) << sft] - t.fstart[b << sft];
            const int ci = (int)(ex & 0xffffu), nd = (int)(ex >> 16);
            const bool ip = p.interpolated(b, c);
            pt[b] = (unsigned short)(ordered ? kP * ci + nd : ip ? kP * ci : kP * p.nc + nd);
            if (ip && ci < max_comp) comp[ci] = (unsigned short)b;
            ex += ip ? 1u : (unsigned)c << 16;
        }
    }
    if (threadIdx.x == 0 && (p.nc > max_comp || p.m > max_pts)) sh.over = 1;
    __syncthreads();
    return p;
}

// T_0 .. T_{kP-1} at t.
__device__ __forceinline__ void cheb(float t, float (&T)[kP]) {
    T[0] = 1.0f;
    T[1] = t;
    const float t2 = 2.0f * t;
#pragma unroll
    for (int k = 2; k < kP; ++k) T[k] = fmaf(t2, T[k - 1], -T[k - 2]);
}

// sum_k T_k coef_k of an interpolated panel's sum (coef 16-byte aligned).
__device__ __forceinline__ float cheb_dot(const float (&T)[kP], const float* __restrict__ coef) {
    float a = 0.0f, b = 0.0f;
#pragma unroll
    for (int k = kP - 4; k >= 0; k -= 4) {   // the small terms first
        const float4 c = *reinterpret_cast<const float4*>(coef + k);
        a = fmaf(T[k + 3], c.w, a);
        b = fmaf(T[k + 2], c.z, b);
        a = fmaf(T[k + 1], c.y, a);
        b = fmaf(T[k], c.x, b);
    }
    return a + b;
}

// Weights of the panels' points (panels of kFine fine bins), one thread per
// fine bin of an interpolated panel: each accumulates the Chebyshev moments of
// its particles (of 1, and of g and c when G / C), the eight bins of a panel
// are combined with shuffles (a running sum for the moments of 1 when PREF)
// and the moments become point weights.  Panels with few particles hand their
// own values over.  gv(slot), cv(slot): the particle's g and c.
template <bool G, bool C, bool PREF, class FG, class FC>
__device__ __forceinline__ void fast_weights(const float* __restrict__ xs, float up, const FastTab& t, const Panels& p,
                                             float* __restrict__ q1, float* __restrict__ qg, float* __restrict__ qc,
                                             FG gv, FC cv) {
    const int tid = threadIdx.x;
    for (int base = 0; base < p.nc * kFine; base += (int)blockDim.x) {
        const int item = base + tid;
        const bool on = item < p.nc * kFine;
        const int s = item % kFine;
        int j0 = 0, j1 = 0, at = 0;
        float cen = 0.0f;
        if (on) {
            const int b = p.comp[item / kFine];
            j0 = t.fstart[kFine * b + s];
            j1 = t.fstart[kFine * b + s + 1];
            cen = p.centre(b);
            at = p.pt[b];
        }
        float m1[kP], mg[kP], mc[kP];
#pragma unroll
        for (int k = 0; k < kP; ++k) m1[k] = mg[k] = mc[k] = 0.0f;
        for (int j = j0; j < j1; ++j) {
            float T[kP];
            cheb((xs[j] * up - cen) * kInvHalfW, T);
            const float g = G ? gv(j) : 0.0f;
            const float c = C ? cv(j) : 0.0f;
#pragma unroll
            for (int k = 0; k < kP; ++k) {
                m1[k] += T[k];
                if (G) mg[k] = fmaf(g, T[k], mg[k]);
                if (C) mc[k] = fmaf(c, T[k], mc[k]);
            }
        }
#pragma unroll
        for (int o = 1; o < kFine; o <<= 1) {
#pragma unroll
            for (int k = 0; k < kP; ++k) {
                if (PREF) {
                    const float v = __shfl_up_sync(0xffffffffu, m1[k], o, kFine);
                    if (s >= o) m1[k] += v;
                } else {
                    m1[k] += __shfl_xor_sync(0xffffffffu, m1[k], o, kFine);
                }
                if (G) mg[k] += __shfl_xor_sync(0xffffffffu, mg[k], o, kFine);
                if (C) mc[k] += __shfl_xor_sync(0xffffffffu, mc[k], o, kFine);
            }
        }
        if (on) {
            if (PREF) {
#pragma unroll
                for (int q = 0; q < kP; q += 4) {
                    float4 w = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                    for (int k = 0; k < kP; ++k) {
                        const float4 v = *reinterpret_cast<const float4*>(t.basis + k * kP + q);
                        w.x = fmaf(v.x, m1[k], w.x);
                        w.y = fmaf(v.y, m1[k], w.y);
                        w.z = fmaf(v.z, m1[k], w.z);
                        w.w = fmaf(v.w, m1[k], w.w);
                    }
                    *reinterpret_cast<float4*>(t.pref + (size_t)item * kP + q) = w;
                    if (s == kFine - 1) *reinterpret_cast<float4*>(q1 + at + q) = w;
                }
            } else {
                for (int q = s; q < kP; q += kFine) {
                    float w = 0.0f;
#pragma unroll
                    for (int k = 0; k < kP; ++k) w = fmaf(t.basis[k * kP + q], m1[k], w);
                    q1[at + q] = w;
                }
            }
            if (G) {
                // 12 (24 with c) weights over the panel's eight threads
                constexpr int per = C ? 2 * kP / kFine : (kP + kFine - 1) / kFine;
#pragma unroll
                for (int e = 0; e < per; ++e) {
                    const int o = s * per + e;
                    const int q = o % kP;
                    if (!C && o >= kP) break;
                    float w = 0.0f;
#pragma unroll
                    for (int k = 0; k < kP; ++k) {
                        const float m = C && o >= kP ? mc[k] : mg[k];
                        w = fmaf(t.basis[k * kP + q], m, w);
                    }
                    (C && o >= kP ? qc : qg)[at + q] = w;
                }
            }
        }
    }
    for (int b = tid; b < kFineBins / kFine; b += (int)blockDim.x) {
        const int j0 = t.fstart[kFine * b], cnt = t.fstart[kFine * (b + 1)] - j0;
        if (cnt == 0 || p.interpolated(b, cnt)) continue;
        const int o = p.pt[b];
        for (int j = 0; j < cnt; ++j) {
            q1[o + j] = 1.0f;
            if (G) qg[o + j] = gv(j0 + j);
            if (C) qc[o + j] = cv(j0 + j);
        }
    }
}

// Positions of the panels' points (up: coordinates are stored times 1 / up),
// and far points up to m_pad.
__device__ __forceinline__ void fast_points(const float* __restrict__ xs, float up, const FastTab& t, const Panels& p,
                                            float* __restrict__ px, int m_pad, float far) {
    const float* node = t.basis + kP * kP;
    const float sc = (1.0f / p.narrow) * (1.0f / up), dn = 1.0f / up;
    for (int i = threadIdx.x; i < kP * p.nc; i += (int)blockDim.x) {
        const int b = p.comp[i / kP], q = i % kP;
        px[p.pt[b] + q] = fmaf(node[q], sc, p.centre(b) * dn);
    }
    for (int b = threadIdx.x; b < kFineBins >> p.sft; b += (int)blockDim.x) {
        const int j0 = t.fstart[b << p.sft], cnt = t.fstart[(b + 1) << p.sft] - j0;
        if (cnt == 0 || p.interpolated(b, cnt)) continue;
        const int o = p.pt[b];
        for (int j = 0; j < cnt; ++j) px[o + j] = xs[j0 + j];
    }
    for (int i = p.m + threadIdx.x; i < m_pad; i += (int)blockDim.x) px[i] = far;
}

// Sums at the points of panels c0 .. c1 - 1 -> Chebyshev coefficients, in place, one thread per
// (panel, sum); sums are arrays r0 .. r0 + nq - 1 of STRIDE floats in pts.
template <int STRIDE = kMaxPts>
__device__ __forceinline__ void fast_coefficients(const FastTab& t, int c0, int c1, int r0, int nq) {
    const int nc = c1 - c0;
    for (int it = threadIdx.x; it < nc * nq; it += (int)blockDim.x) {
        float* v = t.pts + (r0 + it / nc) * STRIDE + (c0 + it % nc) * kP;
        float a[kP];
#pragma unroll
        for (int q = 0; q < kP; q += 4) *reinterpret_cast<float4*>(a + q) = *reinterpret_cast<const float4*>(v + q);
        float out[kP];
#pragma unroll
        for (int k = 0; k < kP; ++k) {
            float s = 0.0f;
#pragma unroll
            for (int q = 0; q < kP; q += 4) {
                const float4 w = *reinterpret_cast<const float4*>(t.basis + k * kP + q);
                s = fmaf(w.x, a[q], fmaf(w.y, a[q + 1], fmaf(w.z, a[q + 2], fmaf(w.w, a[q + 3], s))));
            }
            out[k] = s;
        }
#pragma unroll
        for (int q = 0; q < kP; q += 4) *reinterpret_cast<float4*>(v + q) = *reinterpret_cast<const float4*>(out + q);
    }
}

// The points a CTA sums at: all of them, or a cluster member's, those of the
// panels its slots lie in (interpolated ones, then single points).
struct PointRange {
    int c0, c1;               // its interpolated panels
    int nc, d0, count;        // points of interpolated panels, first single point, all
    __device__ __forceinline__ int at(int k) const { return k < nc ? kP * c0 + k : d0 + (k - nc); }
};
__device__ __forceinline__ PointRange all_points(const Panels& p) { return PointRange{0, p.nc, kP * p.nc, kP * p.nc, p.m}; }
__device__ inline PointRange member_points(const Panels& p, const float* __restrict__ xs, int s0, int s1,
                                           const FastTab& t) {
    PointRange r{0, 0, 0, 0, 0};
    if (s0 >= s1) return r;
    const int b0 = fine_bin(xs[s0]) >> p.sft, b1 = fine_bin(xs[s1 - 1]) >> p.sft;
    auto before = [&](int b) {   // interpolated panels below b
        int lo = 0, hi = p.nc;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (p.comp[mid] < b) lo = mid + 1; else hi = mid;
        }
        return lo;
    };
    r.c0 = before(b0);
    r.c1 = before(b1 + 1);
    r.nc = kP * (r.c1 - r.c0);
    int d0 = 1 << 20, d1 = 0;
    for (int b = b0 + (threadIdx.x & 31); b <= b1; b += 32) {
        const int c = t.fstart[(b + 1) << p.sft] - t.fstart[b << p.sft];
        if (c == 0 || p.interpolated(b, c)) continue;
        d0 = min(d0, (int)p.pt[b]);
        d1 = max(d1, (int)p.pt[b] + c);
    }
    d0 = __reduce_min_sync(0xffffffffu, d0);
    d1 = __reduce_max_sync(0xffffffffu, d1);
    r.d0 = d0;
    r.count = r.nc + max(d1 - d0, 0);
    return r;
}

// Transport sums at the points (arrays OUT.. of STRIDE floats in pts: sum K g, sum u K^2, then for
// full Newton sum K, sum K c, sum K (3 - 4K), then for the KSD sum g u K^2 and
// sum K^2 (3 - 4K)) over the points' weights.  Eight lanes share the columns of
// two points: with 150 to 300 points that keeps every thread in work.
template <bool FULL, bool KSD, int STRIDE = kMaxPts, int OUT = 4>
__device__ __forceinline__ void fast_point_sums(const FastTab& t, const PointRange& own, int m_pad) {
    constexpr int S = 8, R = 2;
    const float* __restrict__ X = t.pts;
    const float* __restrict__ Q1 = t.pts + STRIDE;
    const float* __restrict__ QG = t.pts + 2 * STRIDE;
    const float* __restrict__ QC = t.pts + 3 * STRIDE;
    const int grp = threadIdx.x / S, q = threadIdx.x % S;
    for (int base = 0; base < own.count; base += R * (int)blockDim.x / S) {
        const int r0 = base + R * grp;
        float2 xi[R], kg[R], gk[R], ks[R], kc[R], nk[R], gd[R], hs[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            xi[r] = f2(X[own.at(min(r0 + r, own.count - 1))]);
            kg[r] = gk[r] = ks[r] = kc[r] = nk[r] = gd[r] = hs[r] = f2(0.0f);
        }
#pragma unroll 2
        for (int cb = q * 4; cb < m_pad; cb += 4 * S) {
            const float4 x4 = *reinterpret_cast<const float4*>(X + cb);
            const float4 a4 = *reinterpret_cast<const float4*>(Q1 + cb);
            const float4 g4 = *reinterpret_cast<const float4*>(QG + cb);
            float4 c4 = make_float4(0.f, 0.f, 0.f, 0.f);
            if (FULL) c4 = *reinterpret_cast<const float4*>(QC + cb);
            const float2 xx[2] = {make_float2(x4.x, x4.y), make_float2(x4.z, x4.w)};
            const float2 aa[2] = {make_float2(a4.x, a4.y), make_float2(a4.z, a4.w)};
            const float2 gg[2] = {make_float2(g4.x, g4.y), make_float2(g4.z, g4.w)};
            const float2 cc[2] = {make_float2(c4.x, c4.y), make_float2(c4.z, c4.w)};
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float2 u = fma2(xx[hf], f2(-1.0f), xi[r]);
                    const float2 b2 = fma2(u, u, f2(1.0f));
                    const float2 K = make_float2(rcp_approx(b2.x), rcp_approx(b2.y));
                    const float2 uk2 = mul2(u, mul2(K, K));
                    kg[r] = fma2(K, gg[hf], kg[r]);
                    gk[r] = fma2(uk2, aa[hf], gk[r]);
                    if (FULL || KSD) {
                        const float2 kt = mul2(K, fma2(K, f2(-4.0f), f2(3.0f)));
                        if (FULL) {
                            ks[r] = fma2(K, aa[hf], ks[r]);
                            kc[r] = fma2(K, cc[hf], kc[r]);
                            nk[r] = fma2(kt, aa[hf], nk[r]);
                        }
                        if (KSD) {
                            gd[r] = fma2(uk2, gg[hf], gd[r]);
                            hs[r] = fma2(mul2(K, kt), aa[hf], hs[r]);
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            float v[7] = {kg[r].x + kg[r].y, gk[r].x + gk[r].y, ks[r].x + ks[r].y, kc[r].x + kc[r].y,
                          nk[r].x + nk[r].y, gd[r].x + gd[r].y, hs[r].x + hs[r].y};
#pragma unroll
            for (int k = 0; k < 7; ++k) {
                if ((k >= 2 && k < 5 && !FULL) || (k >= 5 && !KSD)) continue;
#pragma unroll
                for (int o = S / 2; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
                if (q == 0 && r0 + r < own.count) t.pts[(OUT + k) * STRIDE + own.at(r0 + r)] = v[k];
            }
        }
    }
}

// Twice-counted window of the Hessian's sum: sum over |x - x_j| < kKink of
// K (4K - 3), u = x - x_j.
__device__ __forceinline__ float fast_window(float x, const float* __restrict__ xs, const FastTab& t, const Panels& p) {
    const int fl = fine_bin(x - kKink), fh = fine_bin(x + kKink);
    const float2 x2 = f2(x);
    float2 acc = f2(0.0f);
    // particles one by one, clipped at the window's end
    auto two = [&](float xa, float xb, float2& a) {
        const float2 u = fma2(make_float2(xa, xb), f2(-1.0f), x2);
        const float2 b2 = fma2(u, u, f2(1.0f));
        const float2 K = make_float2(rcp_approx(b2.x), rcp_approx(b2.y));
        const float2 w = fma2(K, f2(4.0f), f2(-3.0f));
        a = fma2(make_float2(fmaxf(w.x, 0.0f), fmaxf(w.y, 0.0f)), K, a);
    };
    float2 acc1 = f2(0.0f);
    auto range = [&](int j, int e) {
        for (; j + 3 < e; j += 4) {
            two(xs[j], xs[j + 1], acc);
            two(xs[j + 2], xs[j + 3], acc1);
        }
        if (j < e) two(xs[j], j + 1 < e ? xs[j + 1] : kHPad, acc);
        if (j + 2 < e) two(xs[j + 2], kHPad, acc1);
    };
    range(t.fstart[fl], t.fstart[fl + 1]);
    if (fh != fl) range(t.fstart[fh], t.fstart[fh + 1]);
    for (int b = fl / kFine; b <= fh / kFine; ++b) {
        const int s0 = b == fl / kFine ? fl % kFine + 1 : 0;
        const int s1 = b == fh / kFine ? fh % kFine : kFine;
        if (s1 <= s0) continue;
        const int j0 = t.fstart[kFine * b + s0], j1 = t.fstart[kFine * b + s1];
        if (j0 == j1) continue;
        if (!p.interpolated(b, t.fstart[kFine * (b + 1)] - t.fstart[kFine * b])) {
            range(j0, j1);
            continue;
        }
        const float* hi = t.pref + ((p.pt[b] / kP) * kFine + s1 - 1) * kP;
        const float* lo = s0 > 0 ? hi - (s1 - s0) * kP : nullptr;
        const float2 d = f2(x - p.centre(b));
#pragma unroll
        for (int q = 0; q < kP; q += 4) {
            const float4 h4 = *reinterpret_cast<const float4*>(hi + q);
            float2 w0 = make_float2(h4.x, h4.y), w1 = make_float2(h4.z, h4.w);
            if (lo) {
                const float4 l4 = *reinterpret_cast<const float4*>(lo + q);
                w0 = fma2(make_float2(l4.x, l4.y), f2(-1.0f), w0);
                w1 = fma2(make_float2(l4.z, l4.w), f2(-1.0f), w1);
            }
            const float4 nd = *reinterpret_cast<const float4*>(t.basis + kP * kP + q);
            const float2 u0 = fma2(make_float2(nd.x, nd.y), f2(-1.0f), d), u1 = fma2(make_float2(nd.z, nd.w), f2(-1.0f), d);
            const float2 b0 = fma2(u0, u0, f2(1.0f)), b1 = fma2(u1, u1, f2(1.0f));
            const float2 K0 = make_float2(rcp_approx(b0.x), rcp_approx(b0.y));
            const float2 K1 = make_float2(rcp_approx(b1.x), rcp_approx(b1.y));
            acc = fma2(mul2(fma2(K0, f2(4.0f), f2(-3.0f)), K0), w0, acc);
            acc1 = fma2(mul2(fma2(K1, f2(4.0f), f2(-3.0f)), K1), w1, acc1);
        }
    }
    acc = add2(acc, acc1);
    return acc.x + acc.y;
}

// The prior means' points: ns of them, panels of width kPanelW / up scaled units.
struct Sources {
    int ns;
    float up;
    int near;          // a mean within this many panels of a point's own: the point is not far
    float far2;        // squared distance to which an interpolated panel's sum keeps its accuracy
    const float* sorted;   // the means themselves by slot, in global memory
};

// Mixture sums at x over the prior means themselves, by one warp (every lane
// gets them): den = sum w, num = sum w d, w = 2^-(d^2 - e), e about the
// smallest d^2.  Means that weigh less than 2^-40 of the nearest are left out.
__device__ __forceinline__ void mixture_exact(float x, const FastTab& t, const Sources& src, float e, float& den,
                                              float& num) {
    const int lane = threadIdx.x & 31;
    const float fs = kFineScale * src.up, reach = sqrtf(e + 40.0f);
    const int k0 = t.src_slot[fine_bin(x - reach, fs) / kFine], k1 = t.src_slot[fine_bin(x + reach, fs) / kFine + 1];
    float a = 0.0f, b = 0.0f;
    for (int k = k0 + lane; k < k1; k += 32) {
        const float d = x - src.sorted[k];
        const float w = ex2_approx(e - d * d);
        a += w;
        b = fmaf(w, d, b);
    }
    den = warp_sum(a);
    num = warp_sum(b);
}

// Whether a point may be far from every mean: no mean in the panels around its
// own, or these reach the first or last panel, whose outliers may lie anywhere
// beyond.
__device__ __forceinline__ bool mixture_is_far(float x, const FastTab& t, const Sources& src) {
    const int b = fine_bin(x, kFineScale * src.up) / kFine;
    const int lo = b - src.near, hi = b + src.near;
    return lo <= 0 || hi >= kFineBins / kFine - 1 || t.src_pt[hi + 1] == t.src_pt[lo];
}

// Mixture sums at a point far from every mean, by one warp.  An interpolated
// panel's sum is accurate relative to its largest term; single means must
// outweigh it by 2^34, or the means themselves are summed.
__device__ __forceinline__ void mixture_far(float x, const FastTab& t, const Sources& src, float& den, float& num,
                                         float& e) {
    const int lane = threadIdx.x & 31;
    float ec = 3.0e38f, ed = 3.0e38f;   // nearest interpolated point, nearest single mean (weight exactly 1)
    for (int k = lane; k < src.ns; k += 32) {
        const float d = x - t.src_x[k];
        if (t.src_w[k] == 1.0f) ed = fminf(ed, d * d);
        else ec = fminf(ec, d * d);
    }
    ec = warp_min(ec);
    ed = warp_min(ed);
    e = fminf(ec, ed);
    if (e > src.far2 && ec < ed + 34.0f) {
        mixture_exact(x, t, src, e, den, num);
        return;
    }
    float a = 0.0f, b = 0.0f;
    for (int k = lane; k < src.ns; k += 32) {
        const float d = x - t.src_x[k];
        const float w = ex2_approx(e - d * d) * t.src_w[k];
        a += w;
        b = fmaf(w, d, b);
    }
    den = warp_sum(a);
    num = warp_sum(b);
}

// Mixture sums at one point by one warp.
__device__ __forceinline__ void mixture_warp(float x, const FastTab& t, const Sources& src, float& den, float& num) {
    const int lane = threadIdx.x & 31;
    const float fs = kFineScale * src.up;
    if (mixture_is_far(x, t, src)) {
        float e;
        mixture_far(x, t, src, den, num, e);
        return;
    }
    const int c0 = t.src_pt[fine_bin(x - kMixReach, fs) / kFine], c1 = t.src_pt[fine_bin(x + kMixReach, fs) / kFine + 1];
    float a0 = 0.0f, a1 = 0.0f;
    for (int k = c0 + lane; k < c1; k += 32) {
        const float d = x - t.src_x[k];
        const float w = ex2_approx(-d * d) * t.src_w[k];
        a0 += w;
        a1 = fmaf(w, d, a1);
    }
    den = warp_sum(a0);
    num = warp_sum(a1);
}

// Mixture sums at the points, [4][kMixPts] of pts: den, num, e (w = 2^-(d^2 - e);
// e = 0 unless the point is far from every mean) over the prior means' points
// within reach.  Eight lanes share the columns of two neighbouring points.
template <class FX>
__device__ __forceinline__ void fast_mixture_points(const FastTab& t, FastSh& sh, const PointRange& own,
                                                    const Sources& src, FX scaled) {
    constexpr int S = 8, R = 2;
    const int grp = threadIdx.x / S, q = threadIdx.x % S;
    unsigned short* far_list = reinterpret_cast<unsigned short*>(t.pref);
    const float fs = kFineScale * src.up;
    for (int base = 0; base < own.count; base += R * (int)blockDim.x / S) {
        const int r0 = base + R * grp;
        float x[R];
        float2 x2[R], den2[R], num2[R];
        bool far[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            x[r] = scaled(t.pts[own.at(min(r0 + r, own.count - 1))]);
            x2[r] = f2(x[r]);
            den2[r] = num2[r] = f2(0.0f);
            far[r] = mixture_is_far(x[r], t, src);
        }
        const int c0 = t.src_pt[fine_bin(fminf(x[0], x[1]) - kMixReach, fs) / kFine] & ~3;
        const int c1 = t.src_pt[fine_bin(fmaxf(x[0], x[1]) + kMixReach, fs) / kFine + 1];
        for (int cb = c0 + q * 4; cb < c1; cb += 4 * S) {
            const float4 m4 = *reinterpret_cast<const float4*>(t.src_x + cb);
            const float4 w4 = *reinterpret_cast<const float4*>(t.src_w + cb);
            const float2 mm[2] = {make_float2(m4.x, m4.y), make_float2(m4.z, m4.w)};
            const float2 ww[2] = {make_float2(w4.x, w4.y), make_float2(w4.z, w4.w)};
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float2 d = fma2(mm[hf], f2(-1.0f), x2[r]);
                    const float2 qq = mul2(d, d);
                    const float2 w = mul2(make_float2(ex2_approx(-qq.x), ex2_approx(-qq.y)), ww[hf]);
                    den2[r] = add2(den2[r], w);
                    num2[r] = fma2(w, d, num2[r]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            float den = den2[r].x + den2[r].y, num = num2[r].x + num2[r].y;
#pragma unroll
            for (int o = S / 2; o > 0; o >>= 1) {
                den += __shfl_xor_sync(0xffffffffu, den, o);
                num += __shfl_xor_sync(0xffffffffu, num, o);
            }
            if (q == 0 && r0 + r < own.count) {
                const int at = own.at(r0 + r);
                t.pts[kMixPts + at] = den;
                t.pts[2 * kMixPts + at] = num;
                t.pts[3 * kMixPts + at] = 0.0f;
                if (far[r]) far_list[atomicAdd(&sh.n_far, 1)] = (unsigned short)at;
            }
        }
    }
    __syncthreads();
    // the far ones, a warp each (in any order: they are independent)
    for (int k = threadIdx.x >> 5; k < sh.n_far; k += (int)(blockDim.x >> 5)) {
        const int r = far_list[k];
        float den, num, e;
        mixture_far(scaled(t.pts[r]), t, src, den, num, e);
        if ((threadIdx.x & 31) == 0) {
            t.pts[kMixPts + r] = den;
            t.pts[2 * kMixPts + r] = num;
            t.pts[3 * kMixPts + r] = e;
        }
    }
}

// The panels' mixture sums, levelled, as Chebyshev coefficients, in place:
// sixteen lanes per panel.  unit: scaled units per bandwidth.  A panel whose
// last coefficients have not fallen to FP32 rounding (the sums change over
// from one prior mean to another many sigma away) is marked: its particles
// are summed one by one.
__device__ __forceinline__ void fast_mixture_panels(const FastTab& t, const Panels& p, const PointRange& own, float unit) {
    const int lane = threadIdx.x & 31, q = lane & 15;
    for (int base = own.c0; base < own.c1; base += (int)blockDim.x / 16) {
        const int ci = base + threadIdx.x / 16;
        const bool on = ci < own.c1 && q < kP;
        const int at = min(ci, own.c1 - 1) * kP + min(q, kP - 1);
        const float den = t.pts[kMixPts + at], num = t.pts[2 * kMixPts + at], e = t.pts[3 * kMixPts + at];
        const float y = t.basis[kP * kP + min(q, kP - 1)] * unit / p.narrow;
        const float L = e - lg2_approx(den) - y * y;   // -log2 of the sum, less one Gaussian's curvature
        const float L0 = __shfl_sync(0xffffffffu, L, lane & 16), y0 = __shfl_sync(0xffffffffu, y, lane & 16);
        const float L1 = __shfl_sync(0xffffffffu, L, (lane & 16) + kP - 1);
        const float y1 = __shfl_sync(0xffffffffu, y, (lane & 16) + kP - 1);
        const float slope = (L0 - L1) / (y0 - y1);
        const float sc = ex2_approx(fmaf(y, y, fmaf(slope, y - y0, L0)) - e);
        const float a = den * sc, b = num * sc;
        float mx = q < kP ? a : 0.0f, mn = q < kP ? a : 3.0e38f;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        }
        float ca = 0.0f, cb = 0.0f;
#pragma unroll
        for (int k = 0; k < kP; ++k) {
            const float w = t.basis[min(q, kP - 1) * kP + k];
            ca = fmaf(w, __shfl_sync(0xffffffffu, a, (lane & 16) + k), ca);
            cb = fmaf(w, __shfl_sync(0xffffffffu, b, (lane & 16) + k), cb);
        }
        const float c0 = __shfl_sync(0xffffffffu, fabsf(ca), lane & 16);
        const float d0 = __shfl_sync(0xffffffffu, fabsf(cb), lane & 16);
        const bool tail = on && q >= kP - 2 && !(fabsf(ca) <= kMixTail * c0 && fabsf(cb) <= kMixTail * (c0 + d0));
        const unsigned tails = __ballot_sync(0xffffffffu, tail);
        if (on) {
            t.pts[kMixPts + at] = ca;
            t.pts[2 * kMixPts + at] = cb;
            if (q == 0) t.bad[ci] = !(mx <= 4.0f * mn) || !(mn > 0.0f) || ((tails >> (lane & 16)) & 0xffffu) != 0u;
        }
    }
}

}  // namespace svpf
