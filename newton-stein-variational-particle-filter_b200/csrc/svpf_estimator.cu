// svpf_estimator.cu -- the reference's differentiable torch model,
// SVPFParamEstimator (py-torch/diff_svpf_torch.py:147-217), as a batched CUDA
// forward and a hand-written reverse-mode adjoint, for F independent paths
// with their own theta = (mu, rho, sigma_z, nu).
//
// The model (per path, N particles, N even):
//   init    h = mu + sigma_z / sqrt(1 - rho^2 + 1e-6) z                 (:168-170)
//   tick t  TBPTT: the particle path is cut when t % truncate_every == 0 (:177-179)
//           eps = (z_1..z_{N/2}, -z_1..-z_{N/2})                        (:184-185)
//           m_i = mu + rho (h_i - mu),  hp_i = m_i + sigma_z eps_i      (:187-188)
//           loglik_t = logsumexp_i log t_nu(y_t; scale e^{hp_i/2}) - log N
//                      (before the transport; _student_t_log_prob :112-119)
//           b = (std(hp) + 0.1)^2 + 1e-8, no derivative through it      (:201)
//           n_stein times (Jacobi over particles):
//             g_i = clamp(-(h_i - m_i)/(sigma_z^2 + 1e-8) + lik score, +-10)  (:204-209)
//             h_i += lr/N sum_j [K_ij g_j - d_ij K_ij^3 / b],
//             d_ij = h_i - h_j, K_ij = (1 + d_ij^2/b)^(-1/2)            (:127-145)
//           vol_t = mean_i e^{h_i/2}                                     (:213)
//   loss    sum_t w_t loglik_t (the reference's NLL is w_t = -1/(T - burn_in)
//           after the burn-in, :214-215)
//
// One CTA per path (grid-stride over paths); all particle arrays of a tick
// live in shared memory.  Two ways to the backward, same bits:
//  * run records (when they fit in memory): the forward keeps every tick's
//    record -- inputs, predicted means, log-densities, the particles before
//    each Stein step -- and the backward sweeps the ticks in reverse from them,
//    the next record copied to shared memory while one is worked on;
//  * checkpoints: the forward stores the particles every k ticks; the
//    backward, segment by segment from the last, recomputes the segment from
//    its checkpoint keeping each tick's input, then walks the ticks in
//    reverse, recomputing each tick once more with its record.
//
// One thread per particle, 256 at most (64 threads for the usual 64
// particles): a tick is a chain of short phases, and a CTA of two warps has
// cheap barriers and leaves room for 16 paths on an SM.  (Two rows per thread
// in packed FP32x2 on one warp took 4.4 ms where this takes 3.2, and no less
// for 2048 paths.)  The row sums keep their order: all columns in turn,
// reductions over 32 consecutive particles, then over these groups.
// Measured on B200, N = 64, 2 Stein steps, 250 ticks, value and gradient: one
// path 5.2 -> 3.2 ms, 1024 paths 13.9 -> 5.1 ms (256 threads a path, each
// tick recomputed twice in the backward).
//
// Adjoint of one Stein step (a_i = lr xbar_i / N, G(d) = -d K^3 / b,
// G'(d) = -K^3/b + 3 d^2 K^5 / b^2, row sums over j with d = d_ij):
//   xbar_i += a_i (-S1/b + S2) - g_i C1/b - C2 + g'_i C3
//   S1 = sum g_j d K^3, S2 = sum G'(d), C1 = sum a_j d K^3, C2 = sum a_j G'(d),
//   C3 = sum a_j K = dL/dg_i;  g'_i = dg_i/dh_i (zero outside the clamp).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "svpf.h"
#include "svpf_device.cuh"
#include "svpf_internal.h"
#include "svpf_math.h"
#include "svpf_trace.h"

namespace svpf {
namespace est {

struct EArgs {
    int F, T, k, n, np, S, trunc, nseg;
    float lr;
    const float* theta;     // [F][4]
    const float* y;         // [F][T]
    const float* w;         // [F][T] or nullptr (all ones)
    const float* tape;      // [F][n + T n/2] or nullptr (Philox)
    unsigned long long seed;
    float* loglik;          // [F][T] or nullptr
    float* vol;             // [F][T] or nullptr
    double* ll_sum;         // [F]
    float* fx;              // [F][np] particles between forward launches
    float* ck;              // [F][nseg][np] checkpoints
    float* ax;              // [F][np] adjoint of the particles between backward launches
    double* ath;            // [F][4] accumulated d loss / d theta
    float* seg;             // [grid][k][np] tick inputs of the segment being reversed
    float* run;             // [F][T_max][rec_floats] run records, or nullptr
    int rec_floats, T_max;
    int* status;            // [F]
};

// A tick's record: xin, m, lp, eps, then the particles before each Stein step
// (max(S, 1) arrays of np floats), then mx, se, b and a pad.
__host__ __device__ inline int record_arrays(int S) { return 4 + (S > 1 ? S : 1); }
__host__ __device__ inline int record_floats(int np, int S) { return record_arrays(S) * np + 4; }

// Per-path scalars of the tick being processed (thread 0 writes, all read).
struct TickShared {
    float mu, rho, sz, nu, C;
    float mx, se, b;        // logsumexp max and sum, kernel scale b
    float red[8][kWarps];
    double acc[4];
    int bad;                // this path's theta is outside the domain (theta_ok)
};

__device__ __forceinline__ size_t tape_stride(const EArgs& a) { return (size_t)a.n + (size_t)a.T * (a.n / 2); }

// Initial standard normal of particle i (torch.randn(N), :170).
__device__ __forceinline__ float init_normal(const EArgs& a, int f, int i) {
    if (a.tape) return a.tape[(size_t)f * tape_stride(a) + i];
    const uint4 r = philox10(philox_key(a.seed, f), make_uint4((uint32_t)i, 0u, 0u, 2u));
    return normal_from_bits(r.x, r.y);
}

// Antithetic predict noise of particle i at tick t (:184-185).
__device__ __forceinline__ float tick_eps(const EArgs& a, int f, int t, int i) {
    const int half = a.n / 2;
    const int ii = i < half ? i : i - half;
    float z;
    if (a.tape) {
        z = a.tape[(size_t)f * tape_stride(a) + a.n + (size_t)t * half + ii];
    } else {
        const uint4 r = philox10(philox_key(a.seed, f), make_uint4((uint32_t)ii, 0u, (uint32_t)t, 0u));
        z = normal_from_bits(r.x, r.y);
    }
    return i < half ? z : -z;
}

// Block sums and, in the same pass, the maximum of mx (MAX).
template <int K, bool MAX = false>
__device__ __forceinline__ void block_sum(float (&v)[K], TickShared& sh, float* mx = nullptr) {
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int q = 0; q < K; ++q) {
        v[q] = warp_sum(v[q]);
        if (lane == 0) sh.red[q][wp] = v[q];
    }
    if (MAX) {
        const float m = warp_max(*mx);
        if (lane == 0) sh.red[K][wp] = m;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < K; ++q) {
        float s = 0.0f;
        for (int i = 0; i < nw; ++i) s += sh.red[q][i];
        v[q] = s;
    }
    if (MAX) {
        float m = sh.red[K][0];
        for (int i = 1; i < nw; ++i) m = fmaxf(m, sh.red[K][i]);
        *mx = m;
    }
    __syncthreads();
}

// 1 / sqrt(x) for x >= 1 (no subnormals to scale).
__device__ __forceinline__ float rsqrt_normal(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// col(x_j, a_j, c_j) for all columns in turn, read eight at a time (the loads
// and reciprocal roots of eight columns overlap; the sums stay in order).
template <class F>
__device__ __forceinline__ void columns(const float* __restrict__ x, const float* __restrict__ a,
                                        const float* __restrict__ c, int n, F&& col) {
    int j = 0;
#pragma unroll 1
    for (; j + 8 <= n; j += 8) {
        float4 x4[2], a4[2], c4[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            x4[k] = *reinterpret_cast<const float4*>(x + j + 4 * k);
            a4[k] = *reinterpret_cast<const float4*>(a + j + 4 * k);
            c4[k] = *reinterpret_cast<const float4*>(c + j + 4 * k);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            col(x4[k].x, a4[k].x, c4[k].x);
            col(x4[k].y, a4[k].y, c4[k].y);
            col(x4[k].z, a4[k].z, c4[k].z);
            col(x4[k].w, a4[k].w, c4[k].w);
        }
    }
    for (; j < n; ++j) col(x[j], a[j], c[j]);
}

// Shared-memory arrays of one path (np floats each).  xin, m, lp, eps and rec are
// one tick's record; the backward from run records has two of them in turn.
struct Arrays {
    float *xin, *m, *lp, *eps, *rec;
    float *h, *hn, *g, *gd, *ab, *xb, *mb;
    float *rec0, *rec1;
};
__device__ __forceinline__ void set_record(Arrays& s, float* r, int np) {
    s.xin = r;
    s.m = r + np;
    s.lp = r + 2 * np;
    s.eps = r + 3 * np;
    s.rec = r + 4 * np;   // S np floats: h before each Stein step
}
__device__ inline Arrays carve(float* base, int np, int S) {
    Arrays s;
    float* p = base;
    s.h = p; p += np;
    s.hn = p; p += np;
    s.g = p; p += np;
    s.gd = p; p += np;
    s.ab = p; p += np;
    s.xb = p; p += np;
    s.mb = p; p += np;
    s.rec0 = p; p += record_floats(np, S);
    s.rec1 = p;
    set_record(s, s.rec0, np);
    return s;
}
__host__ __device__ inline int smem_floats_est(int np, int S, bool run) {
    return 7 * np + (run ? 2 : 1) * record_floats(np, S);
}

// Likelihood score (:205-207): A = y^2 / (e^h nu + 1e-8),
// g_lik = -1/2 + (nu+1)/2 A/(1+A).  With derivatives d/dh and d/dnu.
struct LikScore {
    float gl, dgl_dh, dgl_dnu;
};
__device__ __forceinline__ LikScore lik_score(float h, float y2, float nu) {
    const float v = expf(0.5f * h);
    const float ev = v * v;
    const float den = ev * nu + 1e-8f;
    const float A = y2 / den;
    const float opA = 1.0f + A;
    LikScore r;
    r.gl = -0.5f + 0.5f * (nu + 1.0f) * A / opA;
    const float dgl_dA = 0.5f * (nu + 1.0f) / (opA * opA);
    const float q = ev / den;               // dA/dh = -A nu q, dA/dnu = -A q
    r.dgl_dh = dgl_dA * (-A * nu * q);
    r.dgl_dnu = 0.5f * A / opA + dgl_dA * (-A * q);
    return r;
}

// Forward of tick t for path f: xin -> h (the tick's output particles).
// rec != nullptr records h before each Stein step (rec[0] = the predicted
// particles, also when there are no Stein steps).  Returns loglik_t on every
// thread; *vol_out (thread 0) the volatility estimate.
template <int RP>
__device__ float fwd_tick(const EArgs& a, int f, int t, const Arrays& s, TickShared& sh, float* rec,
                          float* vol_out) {
    const int tid = threadIdx.x, nt = blockDim.x, n = a.n, np = a.np;
    const float mu = sh.mu, rho = sh.rho, sz = sh.sz, nu = sh.nu;
    const float y = a.y[(size_t)f * a.T + t];
    const float y2 = y * y;
    // predict + predictive log-likelihood terms (:183-198)
    float lmax = -3.0e38f, psum[1] = {0.0f};
    for (int i = tid; i < n; i += nt) {
        const float eps = tick_eps(a, f, t, i);
        const float mi = mu + rho * (s.xin[i] - mu);
        const float hp = mi + sz * eps;
        s.eps[i] = eps;
        s.m[i] = mi;
        s.h[i] = hp;
        if (rec) rec[i] = hp;
        const float sc = expf(0.5f * hp);
        const float z = y / (sc + 1e-8f);
        const float lp = sh.C - logf(sc + 1e-8f) - (nu + 1.0f) * 0.5f * log1pf(z * z / nu);
        s.lp[i] = lp;
        lmax = fmaxf(lmax, lp);
        psum[0] += hp;
    }
    block_sum<1, true>(psum, sh, &lmax);
    const float hm = psum[0] / (float)n;
    float sq[1] = {0.0f};
    for (int i = tid; i < n; i += nt) {
        const float d = s.h[i] - hm;
        sq[0] += d * d;
    }
    block_sum<1>(sq, sh);
    const float bw = sqrtf(sq[0] / (float)n) + 0.1f;
    const float b = bw * bw + 1e-8f;
    const float ib = 1.0f / b;
    // Stein transport (:203-211)
    const float is2e = 1.0f / (sz * sz + 1e-8f);
    const float scale = a.lr / (float)n;
    for (int st = 0; st < a.S; ++st) {
        for (int i = tid; i < n; i += nt) {
            const float hi = s.h[i];
            if (rec && st > 0) rec[(size_t)st * np + i] = hi;
            const LikScore L = lik_score(hi, y2, nu);
            s.g[i] = clampf(-(hi - s.m[i]) * is2e + L.gl, -10.0f, 10.0f);
        }
        __syncthreads();
        if constexpr (RP == 1) {
            for (int i = tid; i < n; i += nt) {
                const float hi = s.h[i];
                float att = 0.0f, rep = 0.0f;
                columns(s.h, s.g, s.g, n, [&](float hj, float gj, float) {
                    const float d = __fadd_rn(hi, -hj);
                    const float K = rsqrt_normal(__fmaf_rn(__fmul_rn(d, d), ib, 1.0f));
                    att = __fmaf_rn(K, gj, att);
                    rep = __fmaf_rn(__fmul_rn(-d, K), __fmul_rn(K, K), rep);
                });
                s.hn[i] = hi + scale * (att + rep * ib);
            }
        } else
        for (int i0 = tid; i0 < n; i0 += 2 * nt) {
            const bool two = i0 + nt < n;
            const int i1 = two ? i0 + nt : i0;
            const float2 hi = make_float2(s.h[i0], s.h[i1]);
            float2 att = f2(0.0f), rep = f2(0.0f);
            columns(s.h, s.g, s.g, n, [&](float hj, float gj, float) {
                const float2 d = add2(hi, f2(-hj));
                const float2 q = fma2(mul2(d, d), f2(ib), f2(1.0f));
                const float2 K = make_float2(rsqrt_normal(q.x), rsqrt_normal(q.y));
                att = fma2(K, f2(gj), att);
                rep = fma2(mul2(make_float2(-d.x, -d.y), K), mul2(K, K), rep);
            });
            s.hn[i0] = hi.x + scale * (att.x + rep.x * ib);
            if (two) s.hn[i1] = hi.y + scale * (att.y + rep.y * ib);
        }
        __syncthreads();
        for (int i = tid; i < n; i += nt) s.h[i] = s.hn[i];
        __syncthreads();
    }
    float out[2] = {0.0f, 0.0f};   // sum exp(lp - lmax), sum e^(h/2)
    for (int i = tid; i < n; i += nt) {
        out[0] += expf(s.lp[i] - lmax);
        out[1] += expf(0.5f * s.h[i]);
    }
    block_sum<2>(out, sh);
    const float ll = lmax + logf(out[0]) - logf((float)n);
    if (tid == 0) {
        sh.mx = lmax;
        sh.se = out[0];
        sh.b = b;
        if (vol_out) *vol_out = out[1] / (float)n;
    }
    return ll;
}

// Backward of tick t: s.xb holds d loss / d(output particles) on entry and
// d loss / d(input particles) on exit; theta adjoints accumulate in sh.acc.
// Requires the tick's record (s.xin, s.m, s.lp, rec, sh.mx, sh.se, sh.b).
// cut: the particle path is cut before this tick.  Not inlined, with plain
// arguments: both backward kernels run the same code, and so give the same bits.
template <int RP>
__device__ __noinline__ void bwd_tick(float* base, float* record, TickShared& sh, int n, int np, int S, float lr,
                                      float y, float wt, bool cut) {
    Arrays s = carve(base, np, S);
    set_record(s, record, np);
    const float* rec = s.rec;
    const int tid = threadIdx.x, nt = blockDim.x;
    const float mu = sh.mu, rho = sh.rho, sz = sh.sz, nu = sh.nu;
    const float y2 = y * y;
    const float b = sh.b, ib = 1.0f / b, ib2 = ib * ib;
    const float is2e = 1.0f / (sz * sz + 1e-8f);
    const float scale = lr / (float)n;
    float p[5] = {};   // d/d mu, rho, sigma_z, nu, 1 / (sigma_z^2 + 1e-8)
    for (int i = tid; i < n; i += nt) s.mb[i] = 0.0f;
    for (int st = S - 1; st >= 0; --st) {
        const float* hs = rec + (size_t)st * np;
        for (int i = tid; i < n; i += nt) {
            const float hi = hs[i];
            const LikScore L = lik_score(hi, y2, nu);
            const float gpre = -(hi - s.m[i]) * is2e + L.gl;
            const bool in = gpre >= -10.0f && gpre <= 10.0f;   // torch.clamp passes the gradient inclusive
            s.g[i] = clampf(gpre, -10.0f, 10.0f);
            s.gd[i] = in ? -is2e + L.dgl_dh : 0.0f;
            s.ab[i] = scale * s.xb[i];
            s.hn[i] = in ? 1.0f : 0.0f;   // clamp mask of this step
        }
        __syncthreads();
        auto row = [&](int i, float h_, float s1, float s2, float c1, float c2, float c3) {
            const float ai = s.ab[i];
            s.xb[i] += ai * (s2 - s1 * ib) - s.g[i] * c1 * ib - c2 + s.gd[i] * c3;
            const float gb = s.hn[i] * c3;   // d loss / d g_i
            s.mb[i] += gb * is2e;
            p[4] += gb * (h_ - s.m[i]) * is2e * is2e;
            p[3] += gb * lik_score(h_, y2, nu).dgl_dnu;
        };
        if constexpr (RP == 1) {
            for (int i = tid; i < n; i += nt) {
                const float hi = hs[i];
                float S1 = 0.0f, S2 = 0.0f, C1 = 0.0f, C2 = 0.0f, C3 = 0.0f;
                columns(hs, s.ab, s.g, n, [&](float hj, float aj, float gj) {
                    const float d = __fadd_rn(hi, -hj);
                    const float K = rsqrt_normal(__fmaf_rn(__fmul_rn(d, d), ib, 1.0f));
                    const float K2 = __fmul_rn(K, K);
                    const float dK3 = __fmul_rn(__fmul_rn(d, K), K2);
                    const float Gp = __fmul_rn(__fmul_rn(K, K2),
                                               __fmaf_rn(__fmul_rn(__fmul_rn(__fmul_rn(3.0f, d), d), K2), ib2, -ib));
                    S1 = __fmaf_rn(gj, dK3, S1);
                    S2 = __fadd_rn(S2, Gp);
                    C1 = __fmaf_rn(aj, dK3, C1);
                    C2 = __fmaf_rn(aj, Gp, C2);
                    C3 = __fmaf_rn(aj, K, C3);
                });
                row(i, hi, S1, S2, C1, C2, C3);
            }
        } else
        for (int i0 = tid; i0 < n; i0 += 2 * nt) {
            const bool two = i0 + nt < n;
            const int i1 = two ? i0 + nt : i0;
            const float2 hi = make_float2(hs[i0], hs[i1]);
            float2 S1 = f2(0.0f), S2 = f2(0.0f), C1 = f2(0.0f), C2 = f2(0.0f), C3 = f2(0.0f);
            columns(hs, s.ab, s.g, n, [&](float hj, float aj_, float gj) {
                const float2 aj = f2(aj_);
                const float2 d = add2(hi, f2(-hj));
                const float2 q = fma2(mul2(d, d), f2(ib), f2(1.0f));
                const float2 K = make_float2(rsqrt_normal(q.x), rsqrt_normal(q.y));
                const float2 K2 = mul2(K, K);
                const float2 dK3 = mul2(mul2(d, K), K2);
                const float2 Gp = mul2(mul2(K, K2), fma2(mul2(mul2(mul2(f2(3.0f), d), d), K2), f2(ib2), f2(-ib)));
                S1 = fma2(f2(gj), dK3, S1);
                S2 = add2(S2, Gp);
                C1 = fma2(aj, dK3, C1);
                C2 = fma2(aj, Gp, C2);
                C3 = fma2(aj, K, C3);
            });
            row(i0, hi.x, S1.x, S2.x, C1.x, C2.x, C3.x);
            if (two) row(i1, hi.y, S1.y, S2.y, C1.y, C2.y, C3.y);
        }
        __syncthreads();
    }
    // predictive log-likelihood: d/dhp_i and d/dnu of w_t logsumexp(lp) (:192-198)
    const float mx = sh.mx, inv_se = 1.0f / sh.se;
    for (int i = tid; i < n; i += nt) {
        const float hp = rec[i];   // h before the first Stein step = hp
        const float pw = wt * expf(s.lp[i] - mx) * inv_se;
        const float sc = expf(0.5f * hp);
        const float se = sc + 1e-8f;
        const float z = y / se;
        const float q = z * z / nu;
        const float dlp_dsc = -1.0f / se + (nu + 1.0f) * q / ((1.0f + q) * se);
        s.xb[i] += pw * dlp_dsc * 0.5f * sc;
        p[3] += pw * (-0.5f * log1pf(q) + 0.5f * (nu + 1.0f) * q / (nu * (1.0f + q)));
    }
    __syncthreads();
    // predict: hp = m + sigma_z eps, m = mu + rho (xin - mu)
    for (int i = tid; i < n; i += nt) {
        const float hpb = s.xb[i];
        const float mt = s.mb[i] + hpb;
        const float xi = s.xin[i];
        p[0] += (1.0f - rho) * mt;
        p[1] += (xi - mu) * mt;
        p[2] += hpb * s.eps[i];
        s.xb[i] = cut ? 0.0f : rho * mt;
    }
    block_sum<5>(p, sh);
    if (tid == 0) {
        // d/dnu of the normaliser lgamma((nu+1)/2) - lgamma(nu/2) - log(nu pi)/2 (:75-80)
        const double dC = 0.5 * digamma_bounded(0.5 * ((double)nu + 1.0)) - 0.5 * digamma_bounded(0.5 * (double)nu) -
                          0.5 / (double)nu;
        sh.acc[0] += p[0];
        sh.acc[1] += p[1];
        sh.acc[2] += (double)p[2] + (double)p[4] * 2.0 * (double)sz;
        // the constant enters every log-density; the softmax weights sum to one
        sh.acc[3] += (double)p[3] + dC * (double)wt;
    }
    __syncthreads();
}

__device__ inline void load_theta(const EArgs& a, int f, TickShared& sh) {
    sh.mu = a.theta[4 * f + 0];
    sh.rho = a.theta[4 * f + 1];
    sh.sz = a.theta[4 * f + 2];
    sh.nu = a.theta[4 * f + 3];
    const float nu = sh.nu;
    sh.C = lgammaf((nu + 1.0f) * 0.5f) - lgammaf(nu * 0.5f) - 0.5f * logf(nu * 3.14159265358979f);
    sh.bad = !theta_ok(sh.mu, sh.rho, sh.sz, sh.nu);
}

// RP: rows of a thread in a pair sweep, one up to 256 particles, above that two (256 apart) in packed FP32x2.
template <int RP>
__global__ void __launch_bounds__(kThreads) est_forward_kernel(const EArgs a, int t0, int t1) {
    extern __shared__ __align__(16) float smem[];
    __shared__ TickShared sh;
    const Arrays s = carve(smem, a.np, a.S);
    const int tid = threadIdx.x, nt = blockDim.x, n = a.n, np = a.np;
    for (int f = blockIdx.x; f < a.F; f += gridDim.x) {
        if (threadIdx.x == 0) load_theta(a, f, sh);
        __syncthreads();
        if (sh.bad) {
            // parameters no filter can run with: report them and leave the path out
            for (int t = t0 + threadIdx.x; t < t1; t += blockDim.x) {
                if (a.loglik) a.loglik[(size_t)f * a.T + t] = NAN;
                if (a.vol) a.vol[(size_t)f * a.T + t] = NAN;
            }
            if (threadIdx.x == 0) {
                a.status[f] = SVPF_ERR_INVALID_ARG;
                a.ll_sum[f] = NAN;
            }
            __syncthreads();
            continue;
        }
        if (t0 == 0) {
            // :168-170
            const float hs = sh.sz / sqrtf(1.0f - sh.rho * sh.rho + 1e-6f);
            for (int i = tid; i < n; i += nt) s.xin[i] = sh.mu + hs * init_normal(a, f, i);
            if (threadIdx.x == 0) a.ll_sum[f] = 0.0;
        } else {
            for (int i = tid; i < n; i += nt) s.xin[i] = a.fx[(size_t)f * np + i];
        }
        __syncthreads();
        double lls = 0.0;
        for (int t = t0; t < t1; ++t) {
            if (!a.run && t % a.k == 0) {
                float* ck = a.ck + ((size_t)f * a.nseg + t / a.k) * np;
                for (int i = tid; i < n; i += nt) ck[i] = s.xin[i];
            }
            float vol = 0.0f;
            const float ll = fwd_tick<RP>(a, f, t, s, sh, a.run ? s.rec : nullptr, &vol);
            if (a.run) {   // keep the tick's record: the backward replays none of the forward
                float* r = a.run + ((size_t)f * a.T_max + t) * a.rec_floats;
                // xin by the thread that overwrites it below, the arrays behind it 16
                // bytes at a time, pads too (one path of N = 64, 250 ticks: 1.25 ms a
                // forward; all by 4 bytes 1.41)
                for (int i = tid; i < n; i += nt) r[i] = s.xin[i];
                for (int k = np + 4 * tid; k < record_arrays(a.S) * np; k += 4 * nt)
                    *reinterpret_cast<float4*>(r + k) = *reinterpret_cast<const float4*>(s.xin + k);
                if (threadIdx.x == 0) {
                    float* c = r + record_arrays(a.S) * np;
                    c[0] = sh.mx;
                    c[1] = sh.se;
                    c[2] = sh.b;
                }
            }
            if (threadIdx.x == 0) {
                if (a.loglik) a.loglik[(size_t)f * a.T + t] = ll;
                if (a.vol) a.vol[(size_t)f * a.T + t] = vol;
                lls += (double)ll;
                if (!isfinite(ll)) a.status[f] = SVPF_ERR_NONFINITE;
            }
            for (int i = tid; i < n; i += nt) s.xin[i] = s.h[i];
            __syncthreads();
        }
        for (int i = tid; i < n; i += nt) a.fx[(size_t)f * np + i] = s.xin[i];
        if (threadIdx.x == 0) a.ll_sum[f] += lls;
        __syncthreads();
    }
}

// Asynchronous copy of a run record to shared memory (one group per call).
__device__ __forceinline__ void fetch_record(float* dst, const float* src, int floats) {
    for (int k = 4 * threadIdx.x; k < floats; k += 4 * blockDim.x)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst + k)),
                     "l"(src + k));
    asm volatile("cp.async.commit_group;");
}

// RUN: from run records, ticks [0, T); else segment sg.
template <int RP, bool RUN>
__global__ void __launch_bounds__(kThreads, RP == 1 ? 2 : 4)
    est_backward_kernel(const EArgs a, int sg) {
    extern __shared__ __align__(16) float smem[];
    __shared__ TickShared sh;
    Arrays s = carve(smem, a.np, a.S);
    const int tid = threadIdx.x, nt = blockDim.x, n = a.n, np = a.np;
    float* seg = a.seg + (size_t)blockIdx.x * a.k * np;
    const int t0 = RUN ? 0 : sg * a.k;
    const int t1 = RUN ? a.T : min(a.T, t0 + a.k);
    for (int f = blockIdx.x; f < a.F; f += gridDim.x) {
        if (threadIdx.x == 0) {
            load_theta(a, f, sh);
            for (int q = 0; q < 4; ++q) sh.acc[q] = a.ath[4 * (size_t)f + q];
        }
        __syncthreads();
        if (sh.bad) {
            if (threadIdx.x == 0) {
                for (int q = 0; q < 4; ++q) a.ath[4 * (size_t)f + q] = NAN;
                a.status[f] = SVPF_ERR_INVALID_ARG;
            }
            __syncthreads();
            continue;
        }
        for (int i = tid; i < n; i += nt) s.xb[i] = a.ax[(size_t)f * np + i];
        if constexpr (RUN) {
            const float* run = a.run + (size_t)f * a.T_max * a.rec_floats;
            fetch_record((t1 - 1) & 1 ? s.rec1 : s.rec0, run + (size_t)(t1 - 1) * a.rec_floats, a.rec_floats);
            for (int t = t1 - 1; t >= t0; --t) {
                float* r = t & 1 ? s.rec1 : s.rec0;
                if (t > t0) {
                    // every thread is past the tick that read the other buffer (its last barrier)
                    fetch_record(t & 1 ? s.rec0 : s.rec1, run + (size_t)(t - 1) * a.rec_floats, a.rec_floats);
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                } else {
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                }
                __syncthreads();
                set_record(s, r, np);
                if (threadIdx.x == 0) {
                    const float* c = r + record_arrays(a.S) * np;
                    sh.mx = c[0];
                    sh.se = c[1];
                    sh.b = c[2];
                }
                __syncthreads();
                const float wt = a.w ? a.w[(size_t)f * a.T + t] : 1.0f;
                bwd_tick<RP>(smem, s.xin, sh, n, np, a.S, a.lr, a.y[(size_t)f * a.T + t], wt,
                             a.trunc > 0 && t > 0 && t % a.trunc == 0);
            }
        } else {
            const float* ck = a.ck + ((size_t)f * a.nseg + sg) * np;
            for (int i = tid; i < n; i += nt) s.xin[i] = ck[i];
            __syncthreads();
            // recompute the segment, keeping each tick's input particles
            for (int t = t0; t < t1; ++t) {
                float* sx = seg + (size_t)(t - t0) * np;
                for (int i = tid; i < n; i += nt) sx[i] = s.xin[i];
                fwd_tick<RP>(a, f, t, s, sh, nullptr, nullptr);
                for (int i = tid; i < n; i += nt) s.xin[i] = s.h[i];
                __syncthreads();
            }
            // reverse over the segment's ticks
            for (int t = t1 - 1; t >= t0; --t) {
                const float* sx = seg + (size_t)(t - t0) * np;
                for (int i = tid; i < n; i += nt) s.xin[i] = sx[i];
                __syncthreads();
                fwd_tick<RP>(a, f, t, s, sh, s.rec, nullptr);
                __syncthreads();   // thread 0 wrote mx, se and b last
                const float wt = a.w ? a.w[(size_t)f * a.T + t] : 1.0f;
                bwd_tick<RP>(smem, s.xin, sh, n, np, a.S, a.lr, a.y[(size_t)f * a.T + t], wt,
                             a.trunc > 0 && t > 0 && t % a.trunc == 0);
            }
        }
        if (t0 == 0) {
            // h0 = mu + hs z, hs = sigma_z / sqrt(q), q = 1 - rho^2 + 1e-6
            float p[2] = {};
            for (int i = tid; i < n; i += nt) {
                p[0] += s.xb[i];
                p[1] += s.xb[i] * init_normal(a, f, i);
            }
            block_sum<2>(p, sh);
            if (threadIdx.x == 0) {
                const double rho = sh.rho, sz = sh.sz;
                const double q = 1.0 - rho * rho + 1e-6;
                sh.acc[0] += p[0];
                sh.acc[2] += (double)p[1] / sqrt(q);
                sh.acc[1] += (double)p[1] * sz * rho / (q * sqrt(q));
            }
        }
        for (int i = tid; i < n; i += nt) a.ax[(size_t)f * np + i] = s.xb[i];
        if (threadIdx.x == 0)
            for (int q = 0; q < 4; ++q) a.ath[4 * (size_t)f + q] = sh.acc[q];
        __syncthreads();
    }
}

}  // namespace est
}  // namespace svpf

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
using namespace svpf;
using namespace svpf::est;

struct svpf_estimator {
    int F = 0, n = 0, np = 0, S = 0, T_max = 0, k = 64, nseg = 0, trunc = 0, grid = 0, T = 0, threads = 0;
    float lr = 0.1f;
    size_t smem = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    bool forward_done = false;
    unsigned long long seed = 0;
    float *d_theta = nullptr, *d_y = nullptr, *d_w = nullptr, *d_tape = nullptr, *d_loglik = nullptr,
          *d_vol = nullptr, *d_fx = nullptr, *d_ck = nullptr, *d_ax = nullptr, *d_seg = nullptr, *d_run = nullptr;
    double *d_llsum = nullptr, *d_ath = nullptr;
    int* d_status = nullptr;
    const float *u_theta = nullptr, *u_y = nullptr, *u_tape = nullptr;
};

namespace {

// Run records hold at most kRunBytes, and beyond kRunFreely no more than a
// kRunShare-th of the device's free memory (asking the driver for that costs
// more than a small run).
constexpr size_t kRunBytes = (size_t)4 << 30, kRunFreely = (size_t)64 << 20;
constexpr size_t kRunShare = 16;

template <class T>
bool ealloc(T** p, size_t count) {
    return cudaMalloc((void**)p, std::max<size_t>(count, 1) * sizeof(T)) == cudaSuccess;
}

EArgs make_eargs(const svpf_estimator* e, const float* theta, const float* y, const float* tape, const float* w,
                 float* loglik, float* vol) {
    EArgs a;
    std::memset(&a, 0, sizeof(a));
    a.F = e->F;
    a.T = e->T;
    a.k = e->k;
    a.n = e->n;
    a.np = e->np;
    a.S = e->S;
    a.trunc = e->trunc;
    a.nseg = e->nseg;
    a.lr = e->lr;
    a.theta = theta;
    a.y = y;
    a.w = w;
    a.tape = tape;
    a.seed = e->seed;
    a.loglik = loglik;
    a.vol = vol;
    a.ll_sum = e->d_llsum;
    a.fx = e->d_fx;
    a.ck = e->d_ck;
    a.ax = e->d_ax;
    a.ath = e->d_ath;
    a.seg = e->d_seg;
    a.run = e->d_run;
    a.rec_floats = record_floats(e->np, e->S);
    a.T_max = e->T_max;
    a.status = e->d_status;
    return a;
}

using Forward = void (*)(EArgs, int, int);
using Backward = void (*)(EArgs, int);
Forward forward_kernel(const svpf_estimator* e) {
    return e->n > kThreads ? est_forward_kernel<2> : est_forward_kernel<1>;
}
Backward backward_kernel(const svpf_estimator* e) {
    if (e->n > kThreads) return e->d_run ? est_backward_kernel<2, true> : est_backward_kernel<2, false>;
    return e->d_run ? est_backward_kernel<1, true> : est_backward_kernel<1, false>;
}

// Shared memory and grid of the engine's kernels, with or without records.
bool configure(svpf_estimator* e) {
    // the opt-in is the device's whole limit (engines of different sizes share the kernels)
    const void* kernels[] = {(const void*)forward_kernel(e), (const void*)backward_kernel(e)};
    for (const void* k : kernels) {
        if (configure_kernel(k, (int)kernel_smem_cap(k), false) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
    }
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    e->smem = (size_t)smem_floats_est(e->np, e->S, e->d_run != nullptr) * sizeof(float);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernels[1], e->threads, e->smem);
    e->grid = std::min(e->F, std::max(1, per_sm) * std::max(sms, 1));
    return true;
}

// Back to checkpoints, whose buffers every engine has.
bool drop_records(svpf_estimator* e) {
    cudaGetLastError();
    if (!e->d_run || cudaStreamSynchronize(e->stream) != cudaSuccess) return false;
    cudaFree(e->d_run);
    e->d_run = nullptr;
    e->forward_done = false;
    return configure(e);
}

// Run records, when two of them fit in shared memory and all of them the
// memory that is left.
bool take_records(svpf_estimator* e, size_t optin) {
    const size_t two = (size_t)smem_floats_est(e->np, e->S, true) * sizeof(float);
    const size_t bytes = (size_t)e->F * e->T_max * record_floats(e->np, e->S) * sizeof(float);
    if (two + sizeof(TickShared) + 64 > optin || bytes > kRunBytes) return true;
    if (bytes > kRunFreely) {
        size_t left = 0, total = 0;
        if (cudaMemGetInfo(&left, &total) != cudaSuccess || bytes > left / kRunShare) {
            cudaGetLastError();
            return true;
        }
    }
    if (!ealloc(&e->d_run, bytes / sizeof(float))) {
        e->d_run = nullptr;
        cudaGetLastError();
        return true;
    }
    return configure(e) || drop_records(e);
}

}  // namespace

extern "C" {

long long svpf_estimator_tape_floats(int n_particles, int T) {
    if (n_particles < 2 || T < 0) return 0;
    return (long long)n_particles + (long long)T * (n_particles / 2);
}

svpf_estimator_t* svpf_estimator_create(int n_filters, int n_particles, int n_stein_steps, float stein_lr,
                                        int T_max, int checkpoint_every, int truncate_every, cudaStream_t stream) {
    SVPF_TRACE();
    if (n_filters < 1 || n_particles < 2 || (n_particles & 1) || n_particles > SVPF_MAX_PARTICLES ||
        n_stein_steps < 0 || n_stein_steps > 64 || T_max < 1 || checkpoint_every < 1 || truncate_every < 0 ||
        !std::isfinite(stein_lr))
        return nullptr;
    svpf_estimator* e = new svpf_estimator();
    e->F = n_filters;
    e->n = n_particles;
    e->np = round_up(n_particles, 64);
    e->S = n_stein_steps;
    e->lr = stein_lr;
    e->T_max = T_max;
    e->k = checkpoint_every;
    e->nseg = (T_max + checkpoint_every - 1) / checkpoint_every;
    e->trunc = truncate_every;
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if ((size_t)smem_floats_est(e->np, e->S, false) * sizeof(float) + sizeof(TickShared) + 64 > (size_t)optin) {
        delete e;
        return nullptr;
    }
    e->threads = std::min(kThreads, round_up(n_particles, 32));
    if (stream) {
        e->stream = stream;
    } else {
        cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking);
        e->own_stream = true;
    }
    if (!configure(e)) {
        svpf_estimator_destroy(e);
        return nullptr;
    }
    const size_t F = (size_t)n_filters, np = (size_t)e->np;
    const bool ok = ealloc(&e->d_theta, 4 * F) && ealloc(&e->d_y, F * T_max) && ealloc(&e->d_w, F * T_max) &&
                    ealloc(&e->d_loglik, F * T_max) && ealloc(&e->d_vol, F * T_max) && ealloc(&e->d_fx, F * np) &&
                    ealloc(&e->d_ck, F * e->nseg * np) && ealloc(&e->d_ax, F * np) &&
                    ealloc(&e->d_seg, (size_t)e->grid * e->k * np) && ealloc(&e->d_llsum, F) &&
                    ealloc(&e->d_ath, 4 * F) && ealloc(&e->d_status, F);
    // the records last: what the checkpoints need is there without them
    if (!ok || !take_records(e, (size_t)optin)) {
        cudaGetLastError();
        svpf_estimator_destroy(e);
        return nullptr;
    }
    return e;
}

void svpf_estimator_destroy(svpf_estimator_t* e) {
    if (!e) return;
    if (e->stream) cudaStreamSynchronize(e->stream);
    void* ptrs[] = {e->d_theta, e->d_y, e->d_w, e->d_tape, e->d_loglik, e->d_vol, e->d_fx, e->d_ck,
                    e->d_ax, e->d_seg, e->d_run, e->d_llsum, e->d_ath, e->d_status};
    for (void* p : ptrs) cudaFree(p);
    if (e->own_stream) cudaStreamDestroy(e->stream);
    delete e;
}

int svpf_estimator_forward_device(svpf_estimator_t* e, const float* d_theta, const float* d_y, int T,
                                  unsigned long long seed, const float* d_tape, float* d_loglik, float* d_vol) {
    SVPF_TRACE();
    if (!e || !d_theta || !d_y || T < 1 || T > e->T_max) return SVPF_ERR_INVALID_ARG;
    e->T = T;
    e->seed = seed;
    e->u_theta = d_theta;
    e->u_y = d_y;
    e->u_tape = d_tape;
    if (cudaMemsetAsync(e->d_status, 0, e->F * sizeof(int), e->stream) != cudaSuccess) return SVPF_ERR_CUDA;
    const EArgs a = make_eargs(e, d_theta, d_y, d_tape, nullptr, d_loglik ? d_loglik : e->d_loglik,
                               d_vol ? d_vol : e->d_vol);
    const int step = e->d_run ? T : e->k;   // one launch, or one per segment
    for (int t0 = 0; t0 < T; t0 += step) {
        forward_kernel(e)<<<e->grid, e->threads, e->smem, e->stream>>>(a, t0, std::min(T, t0 + step));
        if (cudaGetLastError() != cudaSuccess) return SVPF_ERR_CUDA;
    }
    e->forward_done = true;
    return SVPF_OK;
}

int svpf_estimator_backward_device(svpf_estimator_t* e, const float* d_w, double* d_grad) {
    SVPF_TRACE();
    if (!e || !e->forward_done) return SVPF_ERR_NOT_INITIALIZED;
    if (cudaMemsetAsync(e->d_ax, 0, (size_t)e->F * e->np * sizeof(float), e->stream) != cudaSuccess ||
        cudaMemsetAsync(e->d_ath, 0, (size_t)e->F * 4 * sizeof(double), e->stream) != cudaSuccess)
        return SVPF_ERR_CUDA;
    const EArgs a = make_eargs(e, e->u_theta, e->u_y, e->u_tape, d_w, nullptr, nullptr);
    const int nseg = e->d_run ? 1 : (e->T + e->k - 1) / e->k;
    for (int sg = nseg - 1; sg >= 0; --sg) {
        backward_kernel(e)<<<e->grid, e->threads, e->smem, e->stream>>>(a, sg);
        if (cudaGetLastError() != cudaSuccess) return SVPF_ERR_CUDA;
    }
    if (d_grad && cudaMemcpyAsync(d_grad, e->d_ath, (size_t)e->F * 4 * sizeof(double), cudaMemcpyDeviceToDevice,
                                  e->stream) != cudaSuccess)
        return SVPF_ERR_CUDA;
    return SVPF_OK;
}

int svpf_estimator_forward(svpf_estimator_t* e, const float* theta, const float* y, int T, unsigned long long seed,
                           const float* tape, float* loglik, float* vol, double* loglik_sum) {
    SVPF_TRACE();
    if (!e || !theta || !y || T < 1 || T > e->T_max) return SVPF_ERR_INVALID_ARG;
    const size_t F = (size_t)e->F;
    for (size_t f = 0; f < F; ++f)
        if (!theta_ok(theta[4 * f], theta[4 * f + 1], theta[4 * f + 2], theta[4 * f + 3])) return SVPF_ERR_INVALID_ARG;
    if (cudaMemcpyAsync(e->d_theta, theta, 4 * F * sizeof(float), cudaMemcpyHostToDevice, e->stream) != cudaSuccess ||
        cudaMemcpyAsync(e->d_y, y, F * T * sizeof(float), cudaMemcpyHostToDevice, e->stream) != cudaSuccess)
        return SVPF_ERR_CUDA;
    const float* d_tape = nullptr;
    if (tape) {
        const size_t tf = F * (size_t)svpf_estimator_tape_floats(e->n, T);
        // the tape's size depends on T: keep one buffer, grown on demand
        if (cudaStreamSynchronize(e->stream) != cudaSuccess) return SVPF_ERR_CUDA;
        cudaFree(e->d_tape);
        e->d_tape = nullptr;
        if (!ealloc(&e->d_tape, tf) && !(drop_records(e) && ealloc(&e->d_tape, tf))) {
            e->d_tape = nullptr;
            cudaGetLastError();
            return SVPF_ERR_CUDA;
        }
        if (cudaMemcpyAsync(e->d_tape, tape, tf * sizeof(float), cudaMemcpyHostToDevice, e->stream) != cudaSuccess)
            return SVPF_ERR_CUDA;
        d_tape = e->d_tape;
    }
    int rc = svpf_estimator_forward_device(e, e->d_theta, e->d_y, T, seed, d_tape, e->d_loglik, e->d_vol);
    if (rc != SVPF_OK) return rc;
    if (loglik && cudaMemcpyAsync(loglik, e->d_loglik, F * T * sizeof(float), cudaMemcpyDeviceToHost, e->stream) !=
                      cudaSuccess)
        return SVPF_ERR_CUDA;
    if (vol && cudaMemcpyAsync(vol, e->d_vol, F * T * sizeof(float), cudaMemcpyDeviceToHost, e->stream) != cudaSuccess)
        return SVPF_ERR_CUDA;
    if (loglik_sum &&
        cudaMemcpyAsync(loglik_sum, e->d_llsum, F * sizeof(double), cudaMemcpyDeviceToHost, e->stream) != cudaSuccess)
        return SVPF_ERR_CUDA;
    if (cudaStreamSynchronize(e->stream) != cudaSuccess) return SVPF_ERR_CUDA;
    std::vector<int> st(F);
    if (cudaMemcpy(st.data(), e->d_status, F * sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
        return SVPF_ERR_CUDA;
    for (int s : st)
        if (s) return s;
    return SVPF_OK;
}

int svpf_estimator_get_status(svpf_estimator_t* e, int* status) {
    if (!e || !status) return SVPF_ERR_INVALID_ARG;
    if (cudaStreamSynchronize(e->stream) != cudaSuccess) return SVPF_ERR_CUDA;
    return cudaMemcpy(status, e->d_status, (size_t)e->F * sizeof(int), cudaMemcpyDeviceToHost) == cudaSuccess
               ? SVPF_OK : SVPF_ERR_CUDA;
}

int svpf_estimator_backward(svpf_estimator_t* e, const float* w, double* grad) {
    SVPF_TRACE();
    if (!e || !grad) return SVPF_ERR_INVALID_ARG;
    if (!e->forward_done) return SVPF_ERR_NOT_INITIALIZED;
    const size_t F = (size_t)e->F;
    const float* dw = nullptr;
    if (w) {
        if (cudaMemcpyAsync(e->d_w, w, F * e->T * sizeof(float), cudaMemcpyHostToDevice, e->stream) != cudaSuccess)
            return SVPF_ERR_CUDA;
        dw = e->d_w;
    }
    int rc = svpf_estimator_backward_device(e, dw, nullptr);
    if (rc == SVPF_OK &&
        cudaMemcpyAsync(grad, e->d_ath, 4 * F * sizeof(double), cudaMemcpyDeviceToHost, e->stream) != cudaSuccess)
        rc = SVPF_ERR_CUDA;
    if (rc == SVPF_OK && cudaStreamSynchronize(e->stream) != cudaSuccess) rc = SVPF_ERR_CUDA;
    return rc;
}

}  // extern "C"
