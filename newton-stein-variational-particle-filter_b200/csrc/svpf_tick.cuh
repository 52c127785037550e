// svpf_tick.cuh -- one complete SVPF tick of one filter on a team (CTA or
// cluster), particles resident in shared memory from predict to outputs.
//
// Stage order and semantics follow the reference driver
// src/svpf_optimized_graph.cu:915-1389; each stage cites its kernel.
#pragma once

#include "svpf_device.cuh"
#include "svpf_fast.cuh"

namespace svpf {

// Global-memory arrays of one filter.
struct FilterIO {
    float* h;       // [n] positions (read at start, written at end)
    float* h_prev;  // [n] positions of the previous tick
    float* v;       // [n] RMSProp second moment
    float* lw;      // [n] log-weights of the last gradient pass
    int n;
};

template <int R, int S, int KIND, bool KSD, int MODE, int U = 0>
__device__ __forceinline__ float stein_rows(const Smem& sm, int cur, const Plan& pl,
                                            const svpf_config_t& cfg, float bf, const Noise& nz,
                                            int kn, const Team& team, float* phi_out,
                                            const float* pre = nullptr) {
    return transport_pass<R, S, KIND, KSD, MODE, Plan, U>(sm, cur, pl, cfg, bf, nz, kn, team, phi_out, pre);
}

template <int R, int S, int MODE>
__device__ float stein_dispatch(int kind, bool ksd, const Smem& sm, int cur, const Plan& pl,
                                const svpf_config_t& cfg, float bf, const Noise& nz, int kn,
                                const Team& team, float* phi_out = nullptr, const float* pre = nullptr) {
    if (kind == 2) {
        return ksd ? stein_rows<R, S, 2, true, MODE>(sm, cur, pl, cfg, bf, nz, kn, team, phi_out, pre)
                   : stein_rows<R, S, 2, false, MODE>(sm, cur, pl, cfg, bf, nz, kn, team, phi_out, pre);
    } else if (kind == 1) {
        return ksd ? stein_rows<R, S, 1, true, MODE>(sm, cur, pl, cfg, bf, nz, kn, team, phi_out, pre)
                   : stein_rows<R, S, 1, false, MODE>(sm, cur, pl, cfg, bf, nz, kn, team, phi_out, pre);
    }
    return ksd ? stein_rows<R, S, 0, true, MODE>(sm, cur, pl, cfg, bf, nz, kn, team, phi_out, pre)
               : stein_rows<R, S, 0, false, MODE>(sm, cur, pl, cfg, bf, nz, kn, team, phi_out, pre);
}

template <int R, int S, bool SCAN>
__device__ __forceinline__ void grad_dispatch(bool student, const Smem& sm, int cur, const Plan& pl,
                                              const svpf_config_t& cfg, float beta, float* lw,
                                              const Team& team) {
    if (student) grad_pass<R, S, true, SCAN>(sm, cur, pl, cfg, beta, lw, team);
    else grad_pass<R, S, false, SCAN>(sm, cur, pl, cfg, beta, lw, team);
}

// KSD of the last iteration: block sum, then member partials into rank 0.
template <int NT = kThreads>
__device__ __forceinline__ void ksd_publish(float ksd_thread, Plan& pl, const Team& team) {
    float v[1] = {ksd_thread};
    const int op[1] = {0};
    block_reduce<1, NT>(v, op, pl);
    if (threadIdx.x == 0) team.at(pl.ksd_slot, 0)[team.rank] = v[0];
}

// A non-finite observation is refused: the tick leaves the filter's state as
// it was (particles, moments, control record, log-likelihood sum, timestep)
// and reports SVPF_ERR_NONFINITE with NaN outputs.  The reference runs such a
// tick: its fminf/fmaxf clamps pin the particles to a bound and the EKF and
// bandwidth EMAs carry the NaN, so its later ticks report finite nonsense.
// The kernels call it before the tick; every member of a team sees the same
// y_t, so all members skip the tick together.
__device__ __forceinline__ bool refuse_nonfinite(float y_t, svpf_ctl_t& ctl, svpf_out_t& out) {
    if (isfinite(y_t)) return false;
    if (threadIdx.x == 0) {
        const float qnan = __int_as_float(0x7fc00000);
        ctl.status = SVPF_ERR_NONFINITE;
        out.loglik = out.vol = out.h_mean = out.h_mean_raw = qnan;
        out.bw = ctl.bw;
        out.ksd = ctl.ksd_last;
        out.steps_used = 0;
        out.rejuv_fired = 0;
    }
    return true;
}

// A non-finite previous observation is read as 0 (no leverage): the kernels
// pass the returned value to the tick and then flag the tick's status.
__device__ __forceinline__ float readable_y_prev(float y_prev) { return isfinite(y_prev) ? y_prev : 0.0f; }
__device__ __forceinline__ void flag_y_prev(float y_prev, svpf_ctl_t& ctl) {
    if (threadIdx.x == 0 && !isfinite(y_prev) && ctl.status == SVPF_OK) ctl.status = SVPF_ERR_NONFINITE;
}

// Prior mean of a particle at h (svpf_opt_kernels.cu:384-392).
__device__ __forceinline__ float prior_mean(float h, const Plan& pl, const SVPFParams& prm, float y_prev) {
    const float lev = prm.gamma * y_prev;
    return pl.mu_eff + prm.rho * (h - pl.mu_eff) + (lev != 0.0f ? lev / (expf(h * 0.5f) + 1e-8f) : 0.0f);
}

// Workspace of the fast tick: arrays of n floats, the slots' particles, the
// tables (svpf_fast.cuh).  One CTA keeps three arrays: g takes the positions'
// place once they are binned, the next positions the curvatures'.  The members
// of a cluster each have all particles, write one another's arrays and keep
// four.
struct FastWork {
    float* x;                 // positions, by particle
    float* xs;                // positions, by slot
    float* g;                 // transport score, by slot
    float* c;                 // curvature, by slot
    float* xn;                // next positions, by particle
    float* means;             // scaled prior means, until the sources are built
    unsigned short* pidx;     // particle of a slot
    FastTab tab;
    Sources src;              // the prior means
    int sft;                  // fine bins of a mixture panel, log2
};

// Floats of dynamic shared memory of a fast tick, on one CTA or a cluster.
__host__ __device__ inline int fast_smem_floats(int n, bool cluster = false) {
    const int np = round_up(n, 64);
    return (cluster ? 4 : 3) * np + np / 2 + fast_table_floats(np, true);
}
__device__ inline void carve_fast_work(FastWork& w, const Smem& sm, bool cluster) {
    w.x = sm.h[0];
    w.xs = sm.h[1];
    w.means = sm.g;
    float* rest = cluster ? sm.mu : sm.c;   // sm: h, h, g, c, mu, ... of np floats each
    if (cluster) {
        w.g = sm.g;
        w.c = sm.c;
        w.xn = w.x;
    } else {
        w.g = w.x;
        w.c = w.xn = sm.g;
    }
    w.pidx = reinterpret_cast<unsigned short*>(rest);
    w.tab = carve_fast(rest + sm.np / 2, sm.np, true);
}

// The scaled prior means as points, once per tick, in panels of 0.75
// scaled units, or of 1.5 where that many do not fit.  False: they do not fit,
// or one fine bin is too wide for the mixture.
__device__ inline bool fast_sources(FastWork& w, const Plan& pl, const FilterIO& io, FastSh& sh) {
    const int n = io.n;
    const float unit = pl.bw * pl.prior_scale;   // scaled units per bandwidth
    w.sft = 3;
    while (w.sft > 0 && kFineW * unit * (float)(1 << w.sft) > kMixPanelMax) --w.sft;
    if (!(kFineW * unit * (float)(1 << w.sft) <= kMixPanelMax)) return false;
    const FastTab& t = w.tab;
    for (int wide = 0; wide < 2; ++wide) {
        w.src.up = wide ? 0.5f : 1.0f;
        w.src.near = wide ? 0 : 3;
        w.src.far2 = wide ? 5.0625f : 20.25f;
        fast_bin([&](int i) { return w.means[i]; }, n, kFineScale * w.src.up, w.xs, w.pidx, t, sh);
        const Panels p = fast_panels(3, t.src_pt, t.comp, kFineBins / kFine, kMaxSrc, true, t, sh);
        if (sh.over) {
            __syncthreads();   // everyone has read it
            continue;
        }
        w.src.ns = p.m;
        if (threadIdx.x == 0) t.src_pt[kFineBins / kFine] = (unsigned short)p.m;
        // The sorted means stay in h_prev, which has been read and is rewritten at
        // the tick's end (the members of a cluster write the same values).
        for (int k = threadIdx.x; k < n; k += blockDim.x) io.h_prev[k] = w.xs[k];
        for (int b = threadIdx.x; b <= kFineBins / kFine; b += blockDim.x) t.src_slot[b] = t.fstart[kFine * b];
        w.src.sorted = io.h_prev;
        const int pad = min(round_up(p.m, 4), kMaxSrc);
        fast_points(w.xs, w.src.up, t, p, t.src_x, pad, kMuPad);
        auto none = [](int) { return 0.0f; };
        fast_weights<false, false, false>(w.xs, w.src.up, t, p, t.src_w, nullptr, nullptr, none, none);
        for (int i = p.m + threadIdx.x; i < pad; i += blockDim.x) t.src_w[i] = 0.0f;
        __syncthreads();
        return true;
    }
    return false;
}

// One Stein iteration of a filter through the fast sums (svpf_fast.cuh): gradient pass (svpf_opt_kernels.cu:354-521), vanilla or
// full-Newton transport (:527-1103) as grad_pass and transport_pass take it.
// Positions: w.x before, w.xn after (w.x untouched when it returns false: the
// particles do not fit the tables).  ksd: this thread's KSD terms (each slot's
// term takes its score's place, which only that slot's thread still reads, and
// is summed from there in the order of block_reduce).
// In a cluster every member bins all particles (a copy of the same work: it
// costs less than exchanging the order) and sums at the points and moves the
// particles of its own slots; scores, curvatures and new positions go to every
// member through distributed shared memory, one cluster barrier after each.
template <bool PROD, int NT>
__device__ bool fast_iteration(const FastWork& w, const Plan& pl, const svpf_config_t& cfg,
                               const FilterIO& io, const Noise& nz, int kn, float beta, float bf, bool last,
                               const Team& team, FastSh& sh, float& ksd) {
    const int tid = threadIdx.x, nt = blockDim.x, n = io.n;
    const FastTab& t = w.tab;
    fast_bin([&](int i) { return w.x[i]; }, n, kFineScale, w.xs, w.pidx, t, sh);
    const Panels p = fast_panels(3, t.pt, t.comp, kMaxComp, kMaxPts, false, t, sh);
    // the mixture's panels: the same ones unless they are too many sigma wide
    const Panels q = w.sft == 3 ? p : fast_panels(w.sft, t.mpt, t.mcomp, kMixComp, kMixPts, false, t, sh);
    if (sh.over) return false;
    const int per = (n + team.size - 1) / team.size;
    const int s0 = min(team.rank * per, n), s1 = min(s0 + per, n);   // own slots
    const bool alone = team.size == 1;
    const PointRange own = alone ? all_points(p) : member_points(p, w.xs, s0, s1, t);
    const PointRange mix = alone ? all_points(q) : w.sft == 3 ? own : member_points(q, w.xs, s0, s1, t);
    fast_points(w.xs, 1.0f, t, q, t.pts, q.m, kHPad);
    __syncthreads();
    auto scaled = [&](float x) { return (fmaf(x, pl.bw, pl.center) - pl.mu_center) * pl.prior_scale; };
    fast_mixture_points(t, sh, mix, w.src, scaled);
    __syncthreads();
    fast_mixture_panels(t, q, mix, pl.bw * pl.prior_scale);
    __syncthreads();
    const int kind = PROD ? 2 : pl.transport;
    const float inv_s2 = 1.0f / (pl.sz_eff * pl.sz_eff);
    const float nu = cfg.nu;
    const float y2 = pl.y_t * pl.y_t;
    for (int base = s0; base < s1; base += nt) {
        const int s = base + tid;
        const bool on = s < s1;
        const float x = w.xs[min(s, s1 - 1)];
        const int b = fine_bin(x) >> q.sft;
        const int j0 = t.fstart[b << q.sft];
        const bool comp = q.interpolated(b, t.fstart[(b + 1) << q.sft] - j0);
        const int at = q.pt[b];
        float den, num;
        if (comp) {
            float T[kP];
            cheb(q.local(x, b), T);
            den = cheb_dot(T, t.pts + kMixPts + at);
            num = cheb_dot(T, t.pts + 2 * kMixPts + at);
        } else {
            const int r = at + (min(s, s1 - 1) - j0);
            den = t.pts[kMixPts + r];
            num = t.pts[2 * kMixPts + r];
        }
        unsigned todo = __ballot_sync(0xffffffffu, on && comp && t.bad[at / kP]);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1u;
            float d_, n_;
            mixture_warp(__shfl_sync(0xffffffffu, scaled(x), src), t, w.src, d_, n_);
            if ((tid & 31) == src) {
                den = d_;
                num = n_;
            }
        }
        if (!on) continue;
        // likelihood, combination and curvature as in grad_pass
        const float h = fmaf(x, pl.bw, pl.center);
        const float gp = -(num / pl.prior_scale) * inv_s2 / den;
        const float vol = expf(fminf(h, 20.0f));
        const float A = y2 / (vol + 1e-8f) / nu;
        const float opA = 1.0f + A;
        float glik;
        if (cfg.use_exact_gradient) glik = -0.5f + 0.5f * (nu + 1.0f) * A / opA - cfg.lik_offset;
        else glik = (logf(y2 + 1e-10f) - h + cfg.lik_offset) / 1.4f;
        const float eb = pl.fan ? 1.0f : beta;
        const float score = clampf(gp + eb * glik, -10.0f, 10.0f);
        float curv = 0.0f;
        if (kind == 2) {
            const float hl = -0.5f * (nu + 1.0f) * A / (opA * opA);
            curv = clampf(-(hl - inv_s2), 0.1f, 100.0f);
        }
        if (alone) {
            w.g[s] = score;
            if (kind == 2) w.c[s] = curv;
        } else {
            for (int rk = 0; rk < team.size; ++rk) {
                team.at(w.g, rk)[s] = score;
                if (kind == 2) team.at(w.c, rk)[s] = curv;
            }
        }
        if (last)
            io.lw[w.pidx[s]] = pl.fan ? 0.0f
                                      : pl.stc - 0.5f * h - (nu + 1.0f) * 0.5f * log1pf(fmaxf(A, -0.999f));
    }
    team.sync();
    const int m = p.m, m_pad = round_up(m, 32);
    fast_points(w.xs, 1.0f, t, p, t.pts, m_pad, kHPad);
    for (int i = m + tid; i < m_pad; i += nt)
        t.pts[kMaxPts + i] = t.pts[2 * kMaxPts + i] = t.pts[3 * kMaxPts + i] = 0.0f;
    auto gv = [&](int j) { return w.g[j]; };
    auto cv = [&](int j) { return w.c[j]; };
    if (kind == 2)
        fast_weights<true, true, true>(w.xs, 1.0f, t, p, t.pts + kMaxPts, t.pts + 2 * kMaxPts, t.pts + 3 * kMaxPts, gv, cv);
    else
        fast_weights<true, false, false>(w.xs, 1.0f, t, p, t.pts + kMaxPts, t.pts + 2 * kMaxPts, nullptr, gv, cv);
    __syncthreads();
    if (kind == 2) {
        if (last) fast_point_sums<true, true>(t, own, m_pad);
        else fast_point_sums<true, false>(t, own, m_pad);
    } else {
        if (last) fast_point_sums<false, true>(t, own, m_pad);
        else fast_point_sums<false, false>(t, own, m_pad);
    }
    __syncthreads();
    if (kind == 2) {
        fast_coefficients(t, own.c0, own.c1, 4, last ? 7 : 5);
    } else {
        fast_coefficients(t, own.c0, own.c1, 4, 2);
        if (last) fast_coefficients(t, own.c0, own.c1, 9, 2);
    }
    __syncthreads();
    const float sign = cfg.stein_repulsive_sign == 1 ? 1.0f : -1.0f;
    const float inv_bw = pl.inv_bw, inv_bw2 = pl.inv_bw2, inv_n = 1.0f / (float)n;
    const float es = pl.eps_step * bf, rr = cfg.rmsprop_rho;
    ksd = 0.0f;
    for (int s = s0 + tid; s < s1; s += nt) {
        const float x = w.xs[s];
        const int i = w.pidx[s];
        // a particle's member may change between iterations: its moment lives in L2
        const float v0 = alone ? io.v[i] : __ldcg(io.v + i);
        const int b = fine_bin(x) / kFine;
        const int j0 = t.fstart[kFine * b];
        float sum[7] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        const float* row = t.pts + 4 * kMaxPts + p.pt[b];
        if (p.interpolated(b, t.fstart[kFine * (b + 1)] - j0)) {
            float T[kP];
            cheb(p.local(x, b), T);
            sum[0] = cheb_dot(T, row);
            sum[1] = cheb_dot(T, row + kMaxPts);
            if (kind == 2) {
                sum[2] = cheb_dot(T, row + 2 * kMaxPts);
                sum[3] = cheb_dot(T, row + 3 * kMaxPts);
                sum[4] = cheb_dot(T, row + 4 * kMaxPts);
            }
            if (last) {
                sum[5] = cheb_dot(T, row + 5 * kMaxPts);
                sum[6] = cheb_dot(T, row + 6 * kMaxPts);
            }
        } else {
            row += s - j0;
#pragma unroll
            for (int k = 0; k < 7; ++k)
                if (k < 2 || (k < 5 ? kind == 2 : last)) sum[k] = row[k * kMaxPts];
        }
        float phi = (sum[0] + sign * 2.0f * inv_bw * sum[1]) * inv_n;
        if (kind == 2) {
            const float nk = sum[4] + 2.0f * fast_window(x, w.xs, t, p);
            float H = (sum[3] + 2.0f * inv_bw2 * nk) / fmaxf(sum[2], 1e-6f);
            H = clampf(H, 0.1f, 100.0f);
            phi = phi * (1.0f / H) * 0.7f;
        }
        if (last) {
            const float si = w.g[s];
            w.g[s] = si * sum[0] + 2.0f * inv_bw * (si * sum[1] - sum[5]) + 2.0f * inv_bw2 * sum[6];
        }
        const float vn = rr * v0 + (1.0f - rr) * phi * phi;
        if (alone) io.v[i] = vn;
        else __stcg(io.v + i, vn);
        const float drift = es * phi * rsqrtf(vn + cfg.rmsprop_eps);
        float diff = 0.0f;
        if (pl.temp > 1e-6f) diff = sqrtf(2.0f * es * pl.temp) * nz.normal(i, kn);
        const float h_new = clamp_h(fmaf(x, pl.bw, pl.center) + drift + diff);
        const float hs_new = (h_new - pl.center) * inv_bw;
        if (alone) {
            w.xn[i] = hs_new;
        } else {
            for (int rk = 0; rk < team.size; ++rk) team.at(w.xn, rk)[i] = hs_new;
        }
    }
    team.sync();
    if (last)
        for (int s = s0 + first_lane<NT>(s1); s < s1; s += kThreads) ksd += w.g[s];
    return true;
}

// One Stein iteration of a fast tick by sweeps over the pairs.  ksd: this thread's
// KSD terms of the last iteration, summed in the order of block_reduce from the
// prior means' place (nothing reads them again).
template <int R, int S, bool PROD, int NT>
__device__ __forceinline__ void sweep_iteration(const Smem& sm, int cur, const Plan& pl, const svpf_config_t& cfg,
                                                const FilterIO& io, const Noise& nz, int kn, float beta, float bf,
                                                bool last, const Team& team, float& ksd) {
    grad_pass<R, S, false, false, 0, NT>(sm, cur, pl, cfg, beta, io.lw, team);
    team.sync();
    auto transport = [&](auto kind) {
        constexpr int K = decltype(kind)::value;
        if (last) transport_pass<R, S, K, true, kTransport, Plan, 0, NT, true>(sm, cur, pl, cfg, bf, nz, kn, team,
                                                                             nullptr, nullptr, sm.mu);
        else transport_pass<R, S, K, false, kTransport, Plan, 0, NT>(sm, cur, pl, cfg, bf, nz, kn, team);
    };
    if (PROD || pl.transport == 2) transport(std::integral_constant<int, 2>());
    else transport(std::integral_constant<int, 0>());
    if (!last) return;
    __syncthreads();
    ksd = 0.0f;
    for (int i = sm.row0 + first_lane<NT>(sm.row1 - sm.row0); i < sm.row1; i += kThreads) ksd += sm.mu[i];
}

// Its tile.  On a cluster (S > 1) the widest column split up to S that takes a
// member's rows in one go: a tick of N = 2048 315 us where one row per thread of
// 256 took 585, 4096 976 and 1117, 8192 3.6 and 4.2 ms.  On one CTA two rows per
// thread, on all threads of a wide one where they have rows (200 filters of 1024
// 1.70 ms, on half of them 1.95), and four on CTAs of 256 threads above 1024
// particles (300 of 4096 34.0 ms, two 36.8).  A wide kernel that holds a second
// tile runs its fast iterations 0.7 % slower.  Two and four rows give the same
// bits (the columns' order is the same; test_gpu_cta_width.py holds it), one row
// and two did not: the compiler fuses the row's end differently.
template <int S, bool PROD, int NT, class... A>
__device__ __forceinline__ void sweep_any(int rows, A&&... a) {
    if constexpr (S > 1) {
        if (rows * S <= NT) sweep_iteration<1, S, PROD, NT>(a...);
        else if (rows * (S / 2) <= NT) sweep_iteration<1, S / 2, PROD, NT>(a...);
        else sweep_iteration<1, 1, PROD, NT>(a...);
    } else {
        if (NT == kThreads && rows > 4 * kThreads) sweep_iteration<NT == kThreads ? 4 : 2, 1, PROD, NT>(a...);
        else sweep_iteration<2, 1, PROD, NT>(a...);
    }
}

// The tick.  cfg/prm/ctl are shared-memory copies owned by the caller; only
// thread 0 of rank 0 mutates ctl after make_plan.  Returns on every member; the
// caller stores ctl/out from rank 0 thread 0.  SCAN: the mixture's row
// maximum comes from a min pass over the unsorted prior means instead of the
// means sorted once per tick (the single-filter latency kernel).  PROD: the
// caller guarantees full-Newton transport, Gaussian state noise and no Heun
// step (the production configuration), so only those code paths are compiled
// and the kernel body stays small (instruction fetch bounds the latency kernel).
// FAST: the Stein iterations go through the fast sums (Gaussian state
// noise, vanilla or full-Newton transport, no Heun step, dynamic shared memory
// of fast_smem_floats); a tick whose particles do not fit them finishes with
// sweeps (sweep_any: S = 1 on one CTA, else the widest column split; R is not
// used).  NT: threads of the CTA (no Heun step above kThreads).
template <int R, int S, bool SCAN = false, bool PROD = false, int U = 0, bool FAST = false, int NT = kThreads>
__device__ void run_tick(const svpf_config_t& cfg, const SVPFParams& prm, svpf_ctl_t& ctl, float y_t,
                         float y_prev, const FilterIO& io, const Noise& nz, const Smem& sm, Plan& pl,
                         const Team& team, svpf_out_t& out) {
    const int tid = threadIdx.x;
    const int n = sm.n;
    FastWork fw;
    if constexpr (FAST) {
        carve_fast_work(fw, sm, team.size > 1);
        fast_load_tables(fw.tab);
    }
    if (tid == 0) {
        pl.flag = 0;
        make_plan(cfg, prm, ctl, y_t, y_prev, pl);
        if (cfg.use_heun) pl.transport = (cfg.use_newton && cfg.use_full_newton) ? 2 : 0;
    }
    // pads: particle columns [n, np) and prior slots [n, m_len)
    auto pads = [&]() {
        for (int i = n + tid; i < sm.np; i += NT) {
            sm.h[0][i] = kHPad; sm.h[1][i] = kHPad; sm.g[i] = 0.0f; sm.c[i] = 0.0f;
        }
        for (int i = n + tid; i < sm.m_len; i += NT) sm.mu[i] = kMuPad;
    };
    if constexpr (!FAST) pads();
    __syncthreads();

    // ---- predict (svpf_opt_kernels.cu:125-276), guide (:282-327), prior means
    //      (:384-392); every team member does all N rows, no exchange needed.
    float st[4] = {0.0f, 0.0f, 1e10f, -1e10f};
    float sum_mk[1] = {0.0f};
    auto moments = [&](float hp) {
        st[0] += hp;
        st[1] += hp * hp;
        st[2] = fminf(st[2], hp);
        st[3] = fmaxf(st[3], hp);
    };
    {
        const float hbar = ctl.h_mean_prev;
        const bool mim = cfg.use_mim || cfg.use_guided;
        const float gmean = pl.guide_mean;
        const float gsn = pl.gs;
        const float nm_pres = (1.0f - gsn) * hbar + gsn * gmean;
        const float ly2 = logf(y_t * y_t + 1e-10f);
        const float mimp = fmaxf(ly2 + pl.off, -5.0f);
        for (int i = tid; i < n; i += NT) {
            const float hi = io.h[i];
            const float hpi = io.h_prev[i];
            float z;
            if (cfg.use_student_t_state && cfg.nu_state <= 30.0f) {
                const float z0 = nz.normal(i, 0);
                const int nu_int = max((int)(cfg.nu_state + 0.5f), 3);
                float chi2 = 0.0f;
                for (int m = 0; m < nu_int; ++m) { const float u = nz.normal(i, 1 + m); chi2 += u * u; }
                z = z0 * sqrtf((float)nu_int / (chi2 + 1e-8f));
            } else {
                z = nz.normal(i, 0);
            }
            const float lev = prm.gamma * y_prev / (expf(fminf(hi * 0.5f, 20.0f)) + 1e-8f);
            float hp;
            if (mim) {
                const float dev = hi - hbar;
                const float rho_adj = pl.drho * tanhf(dev);
                const float sscale = 1.0f + pl.dsig * fabsf(dev);
                const float sel = nz.uniform(i, 0);
                const float scale = sel < cfg.mim_jump_prob ? cfg.mim_jump_scale : 1.0f;
                const float br = hi > hpi ? pl.rho_up : pl.rho_dn;
                const float rho = clampf(br + rho_adj, 0.0f, 0.999f);
                float mp = pl.mu_eff + rho * (hi - pl.mu_eff) + lev;
                if (cfg.use_guided) {
                    const float zz = (mimp - mp) / 2.5f;
                    const float act = zz > cfg.guided_innovation_threshold
                                          ? tanhf(zz - cfg.guided_innovation_threshold) : 0.0f;
                    const float ga = cfg.guided_alpha_base + (cfg.guided_alpha_shock - cfg.guided_alpha_base) * act;
                    mp = (1.0f - ga) * mp + ga * mimp;
                }
                hp = clamp_h(mp + pl.sz_eff * sscale * scale * z);
            } else {
                hp = clamp_h(pl.mu_eff + prm.rho * (hi - pl.mu_eff) + pl.sz_eff * z + lev);
            }
            if (cfg.use_guide) {
                hp = cfg.use_guide_preserving ? clamp_h(nm_pres + (hp - hbar)) : clamp_h(hp + gsn * (gmean - hp));
            }
            sm.h[0][i] = hp;
            if constexpr (FAST) {
                const float mk = prior_mean(hi, pl, prm, y_prev);
                sm.g[i] = mk;
                if constexpr (NT == kThreads) sum_mk[0] += mk;
            } else {
                sm.mu[i] = pl.mu_eff + prm.rho * (hi - pl.mu_eff) + prm.gamma * y_prev / (expf(hi * 0.5f) + 1e-8f);
            }
            if constexpr (NT == kThreads) moments(hp);
        }
    }
    if constexpr (NT != kThreads) {
        // in the order of a CTA of kThreads (block_reduce)
        __syncthreads();
        for (int i = first_lane<NT>(n); i < n; i += kThreads) {
            moments(sm.h[0][i]);
            if constexpr (FAST) sum_mk[0] += sm.g[i];
        }
    }
    {
        const int op[4] = {0, 0, 2, 1};
        block_reduce<4, NT>(st, op, pl);
        const int add[1] = {0};
        if constexpr (FAST) block_reduce<1, NT>(sum_mk, add, pl);
    }
    // ---- bandwidth (svpf_fused_bandwidth_kernel, svpf_opt_kernels.cu:1159-1235)
    if (tid == 0) {
        const float inv_n = 1.0f / (float)n;
        const float mean = st[0] * inv_n;
        const float var = st[1] * inv_n - mean * mean;
        const float spread = st[3] - st[2];
        const float bw2_new = fmaxf(2.0f * var / logf((float)n + 1.0f), 1e-6f);
        float bw2 = ctl.bw_sq > 0.0f ? 0.3f * bw2_new + 0.7f * ctl.bw_sq : bw2_new;
        const float a = fabsf(y_t);
        float ema = ctl.return_ema, rv = ctl.return_var;
        ema = ema > 0.0f ? 0.05f * a + 0.95f * ema : a;
        rv = rv > 0.0f ? 0.05f * a * a + 0.95f * rv : a * a;
        ctl.return_ema = ema;
        ctl.return_var = rv;
        const float ratio = a / fmaxf(ema, 1e-8f);
        const float comb = fmaxf(ratio, fminf(spread * 0.5f, 2.0f));
        const float scale = clampf(1.0f - 0.25f * fminf(comb - 1.0f, 2.0f), 0.5f, 1.0f);
        bw2 *= scale;
        const float bw = clampf(sqrtf(bw2), 0.01f, 2.0f);
        ctl.bw_sq = bw2;
        ctl.bw = bw;
        pl.bw = bw;
        pl.inv_bw = 1.0f / bw;
        pl.inv_bw2 = 1.0f / (bw * bw);
        pl.center = mean;
        if constexpr (FAST) pl.mu_center = sum_mk[0] * inv_n;   // the panels of the prior means are centred on them
        else pl.mu_center = pl.mu_eff;
        pl.prior_scale = sqrtf(kLog2e * 0.5f / (pl.sz_eff * pl.sz_eff));
    }
    // ---- sort prior means once per tick (used for the per-row maximum)
    if constexpr (!SCAN && !FAST) bitonic_sort(sm.mu, sm.p2);
    else __syncthreads();   // plan scalars of thread 0 visible to all
    // ---- Stein-loop coordinates: positions (h - center) / bw, Gaussian prior
    //      means (mu - mu_center) * prior_scale (order preserving)
    const bool student = PROD ? false : cfg.use_student_t_state != 0;
    if (pl.budget > 0) {
        for (int i = tid; i < n; i += NT) {
            sm.h[0][i] = (sm.h[0][i] - pl.center) * pl.inv_bw;
            if constexpr (FAST) sm.g[i] = (sm.g[i] - pl.mu_center) * pl.prior_scale;
            else if (!student) sm.mu[i] = (sm.mu[i] - pl.mu_center) * pl.prior_scale;
        }
    }
    // ---- own rows' RMSProp state (the fast iterations keep it in global memory)
    if constexpr (!FAST) {
        for (int li = tid; li < sm.row1 - sm.row0; li += NT) sm.v[li] = io.v[sm.row0 + li];
    }
    // ---- SVLD normals of own rows for the first Stein iterations, drawn in
    //      parallel (same draws, in the same slots, as the per-row epilogue takes)
    if (sm.pre != nullptr && pl.temp > 1e-6f && (PROD || !cfg.use_heun)) {
        const int nloc = sm.row1 - sm.row0;
        const int iters = min(pl.budget, kPreIters);
        for (int k = tid; k < iters * nloc; k += NT) {
            const int it = k / nloc, li = k - it * nloc;
            sm.pre[it * sm.Lp + li] = nz.normal(sm.row0 + li, pl.kn_pred + it);
        }
    }
    team.sync();   // every member has read io.h / io.h_prev; smem ready

    // ---- annealed Stein loop (svpf_optimized_graph.cu:1120-1317)
    int cur = 0;
    int kn = pl.kn_pred;
    const int budget = pl.budget;
    int it0 = 0;
    bool direct = !FAST;
    if constexpr (FAST) {
        if (budget > 0) {
            bool fits = fast_sources(fw, pl, io, *fw.tab.sh);
            if (team.size > 1) team.sync();   // no member reads its means any more
            while (fits && it0 < budget) {
                const float beta = pl.beta[stage_of(pl, it0)];
                float kt;
                fits = fast_iteration<PROD, NT>(fw, pl, cfg, io, nz, kn, beta, sqrtf(beta), it0 == budget - 1,
                                            team, *fw.tab.sh, kt);
                if (!fits) break;
                if (it0 == budget - 1) {
                    ksd_publish<NT>(kt, pl, team);
                    if (team.size > 1) team.sync();
                }
                if (team.size == 1) {
                    float* x = fw.xn;
                    fw.xn = fw.c = fw.x;
                    fw.x = fw.g = x;
                }
                if (pl.temp > 1e-6f) ++kn;
                ++it0;
            }
            if (!fits) {
                // the sweeps take over: positions, prior means (sorted) and moments where they expect them
                __syncthreads();
                direct = true;
                if (fw.x != sm.h[0])
                    for (int i = tid; i < n; i += NT) sm.h[0][i] = fw.x[i];
                __syncthreads();
                pads();
                for (int i = tid; i < n; i += NT) {
                    sm.mu[i] = (prior_mean(io.h[i], pl, prm, y_prev) - pl.mu_center) * pl.prior_scale;
                }
                for (int li = tid; li < sm.row1 - sm.row0; li += NT) sm.v[li] = __ldcg(io.v + sm.row0 + li);
                __syncthreads();
                bitonic_sort(sm.mu, sm.p2);
                if (team.size > 1) team.sync();
            }
        }
    }
    const bool sweeps = NT == kThreads || tid < kThreads;   // small filters' one-row tiles: the first threads
    for (int it = it0; it < budget; ++it) {
        const int ai = stage_of(pl, it);
        const float beta = pl.beta[ai];
        const float bf = sqrtf(beta);
        const bool last = it == budget - 1;
        if constexpr (FAST) {
            float kt = 0.0f;
            sweep_any<S, PROD, NT>((n + team.size - 1) / team.size, sm, cur, pl, cfg, io, nz, kn, beta, bf, last, team,
                                   kt);
            if (last) ksd_publish<NT>(kt, pl, team);
            team.sync();
            cur ^= 1;
        } else if (PROD || !cfg.use_heun) {
            const float* pre = (sm.pre != nullptr && it < kPreIters) ? sm.pre + it * sm.Lp : nullptr;
            float kt = 0.0f;
            if constexpr (PROD) {
                if (sweeps) grad_pass<R, S, false, SCAN, U>(sm, cur, pl, cfg, beta, io.lw, team);
                team.sync();
                if (sweeps)
                    kt = last ? stein_rows<R, S, 2, true, kTransport, U>(sm, cur, pl, cfg, bf, nz, kn, team, nullptr, pre)
                          : stein_rows<R, S, 2, false, kTransport, U>(sm, cur, pl, cfg, bf, nz, kn, team, nullptr, pre);
            } else {
                if (sweeps) grad_dispatch<R, S, SCAN>(student, sm, cur, pl, cfg, beta, io.lw, team);
                team.sync();
                if (sweeps)
                    kt = stein_dispatch<R, S, kTransport>(pl.transport, last, sm, cur, pl, cfg, bf, nz, kn, team,
                                                      nullptr, pre);
            }
            if (last) ksd_publish<NT>(kt, pl, team);
            team.sync();
            cur ^= 1;
        } else if constexpr (!PROD && NT == kThreads) {
            // Heun predictor-corrector (svpf_optimized_graph.cu:1147-1232,
            // kernels svpf_opt_kernels.cu:1293-1566)
            const int nloc = sm.row1 - sm.row0;
            const float es = pl.eps_step * bf;
            grad_dispatch<R, S, SCAN>(student, sm, cur, pl, cfg, beta, io.lw, team);
            team.sync();
            stein_dispatch<R, S, kPhiOnly>(pl.transport, false, sm, cur, pl, cfg, bf, nz, kn, team, sm.phi0);
            __syncthreads();
            for (int li = tid; li < nloc; li += NT) {
                const int i = sm.row0 + li;
                const float h0 = fmaf(sm.h[cur][i], pl.bw, pl.center);
                const float hpred = clamp_h(h0 + es * sm.phi0[li] * rsqrtf(sm.v[li] + cfg.rmsprop_eps));
                const float hs = (hpred - pl.center) * pl.inv_bw;
                for (int rk = 0; rk < team.size; ++rk) team.at(sm.h[cur ^ 1], rk)[i] = hs;
            }
            team.sync();
            grad_dispatch<R, S, SCAN>(student, sm, cur ^ 1, pl, cfg, beta, io.lw, team);
            team.sync();
            stein_dispatch<R, S, kPhiOnly>(pl.transport, false, sm, cur ^ 1, pl, cfg, bf, nz, kn, team, sm.phi1);
            if (last) {
                // KSD at the start point with the gradient at the predicted point
                const float kt = stein_dispatch<R, S, kKsdOnly>(0, true, sm, cur, pl, cfg, bf, nz, kn, team);
                ksd_publish<NT>(kt, pl, team);
            }
            team.sync();   // all members done reading the predicted positions
            for (int li = tid; li < nloc; li += NT) {
                const int i = sm.row0 + li;
                const float pa = 0.5f * (sm.phi0[li] + sm.phi1[li]);
                const float vn = cfg.rmsprop_rho * sm.v[li] + (1.0f - cfg.rmsprop_rho) * pa * pa;
                sm.v[li] = vn;
                float diff = 0.0f;
                if (pl.temp > 1e-6f) diff = sqrtf(2.0f * es * pl.temp) * nz.normal(i, kn);
                const float h0 = fmaf(sm.h[cur][i], pl.bw, pl.center);
                const float hn = clamp_h(h0 + es * pa * rsqrtf(vn + cfg.rmsprop_eps) + diff);
                const float hs = (hn - pl.center) * pl.inv_bw;
                for (int rk = 0; rk < team.size; ++rk) team.at(sm.h[cur ^ 1], rk)[i] = hs;
            }
            team.sync();
            cur ^= 1;
        }
        if (pl.temp > 1e-6f) ++kn;
    }

    // own rows' RMSProp state back to global memory
    if (direct) {
        for (int li = tid; li < sm.row1 - sm.row0; li += NT) io.v[sm.row0 + li] = sm.v[li];
    }
    if (team.rank != 0) return;

    if (tid == 0) {
        if (budget > 0) {
            float acc = 0.0f;
            for (int r = 0; r < team.size; ++r) acc += pl.ksd_slot[r];
            const float k2 = acc / ((float)n * (float)n);
            ctl.ksd_last = sqrtf(fmaxf(k2, 0.0f));
        }
        ctl.stein_steps_used = budget;
    }

    // ---- back to log-volatility coordinates
    float* hf = sm.h[cur];
    if constexpr (FAST)
        if (!direct) hf = fw.x;
    if (budget > 0) {
        for (int i = tid; i < n; i += NT) hf[i] = fmaf(hf[i], pl.bw, pl.center);
        __syncthreads();
    }
    // ---- partial rejuvenation (svpf_opt_kernels.cu:1248-1275)
    if (pl.rejuv) {
        const int ku = pl.uses_uniform_predict;
        const float b = cfg.rejuv_blend;
        for (int i = tid; i < n; i += NT) {
            const float u = nz.uniform(i, ku);
            if (u < cfg.rejuv_prob) {
                const float zz = nz.normal(i, kn);
                hf[i] = clamp_h((1.0f - b) * hf[i] + b * (pl.guide_mean + pl.gstd * zz));
            }
        }
    }
    __syncthreads();

    // ---- outputs (svpf_fused_outputs_kernel, svpf_opt_kernels.cu:1109-1153)
    float mx[1] = {-1e10f};
    for (int i = first_lane<NT>(n); i < n; i += kThreads) mx[0] = fmaxf(mx[0], io.lw[i]);
    {
        const int op[1] = {1};
        block_reduce<1, NT>(mx, op, pl);
    }
    float acc[3] = {0.0f, 0.0f, 0.0f};
    for (int i = first_lane<NT>(n); i < n; i += kThreads) {
        acc[0] += ex2_approx((io.lw[i] - mx[0]) * kLog2e);
        acc[1] += expf(fminf(hf[i] * 0.5f, 20.0f));
        acc[2] += hf[i];
    }
    {
        const int op[3] = {0, 0, 0};
        block_reduce<3, NT>(acc, op, pl);
    }
    // write back positions: h_prev <- positions at tick start, h <- final
    for (int i = tid; i < n; i += NT) {
        io.h_prev[i] = io.h[i];
        io.h[i] = hf[i];
    }
    if (tid == 0) {
        const float inv_n = 1.0f / (float)n;
        const float ll = mx[0] + logf(fmaxf(acc[0] * inv_n, 1e-10f));
        const float vol = acc[1] * inv_n;
        const float hm = acc[2] * inv_n;
        ctl.h_mean_prev = hm;
        // host tail (svpf_optimized_graph.cu:1361-1388): smoother, outputs, adaptive mu
        float hm_out = hm;
        const float bwl = ctl.bw;
        if (cfg.use_smoothing) {
            // svpf_smooth_backward (:658-717)
            const int k = min(max(cfg.smooth_lag, 1), SVPF_SMOOTH_MAX_LAG);
            const int head = ctl.smooth_head;
            ctl.smooth_h_mean[head] = hm;
            ctl.smooth_h_var[head] = bwl * bwl;
            ctl.smooth_y[head] = y_t;
            ctl.smooth_head = (head + 1) % k;
            if (ctl.timestep >= k) {
                const float rho = prm.rho;
                const float mu = cfg.use_adaptive_mu ? ctl.mu_state : prm.mu;
                const float q = prm.sigma_z * prm.sigma_z;
                for (int lag = 1; lag < k; ++lag) {
                    const int ic = (ctl.smooth_head - lag - 1 + k) % k;
                    const int inx = (ctl.smooth_head - lag + k) % k;
                    const float hc = ctl.smooth_h_mean[ic], hn = ctl.smooth_h_mean[inx];
                    const float vc = ctl.smooth_h_var[ic];
                    const float pv = rho * rho * vc + q;
                    const float J = rho * vc / (pv + 1e-8f);
                    ctl.smooth_h_mean[ic] = hc + J * (hn - (mu + rho * (hc - mu)));
                    ctl.smooth_h_var[ic] = vc * (1.0f - J * rho);
                }
            }
            // svpf_get_smoothed_output (:720-737)
            const int k2 = min(cfg.smooth_lag, SVPF_SMOOTH_MAX_LAG);
            if (k2 >= 1 && ctl.timestep >= k2 && cfg.smooth_output_lag > 0) {
                const int ol = min(cfg.smooth_output_lag, k2 - 1);
                hm_out = ctl.smooth_h_mean[(ctl.smooth_head - ol - 1 + k2) % k2];
            }
        }
        ctl.vol_prev = vol;
        ctl.ksd_prev = ctl.ksd_last;
        if (cfg.use_adaptive_mu && ctl.timestep > 10) {
            // svpf_adaptive_mu_update (:619-642)
            const float mp = ctl.mu_state, Pp = ctl.mu_var + cfg.mu_process_var;
            const float Rm = cfg.mu_obs_var_scale * bwl * bwl;
            const float K = Pp / (Pp + Rm + 1e-8f);
            ctl.mu_state = clampf(mp + K * (hm - mp), cfg.mu_min, cfg.mu_max);
            ctl.mu_var = (1.0f - K) * Pp;
        }
        ctl.loglik_sum += (double)ll;
        ctl.timestep += 1;
        // The reference's clamps (fmaxf/fminf) turn a NaN observation into finite
        // particles; the tick runs the same way here and the status reports it.
        int status = pl.flag;
        if (status == SVPF_OK && !(isfinite(y_t) && isfinite(y_prev) && isfinite(ll) && isfinite(vol) && isfinite(hm)))
            status = SVPF_ERR_NONFINITE;
        ctl.status = status;
        out.loglik = ll;
        out.vol = vol;
        out.h_mean = hm_out;
        out.h_mean_raw = hm;
        out.bw = bwl;
        out.ksd = ctl.ksd_last;
        out.steps_used = budget;
        out.rejuv_fired = pl.rejuv;
    }
}

}  // namespace svpf
