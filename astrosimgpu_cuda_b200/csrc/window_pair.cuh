// window_pair.cuh -- the FP32 form's window bodies: two cells per thread.
//
// The FP32 window kernel was bound by instruction issue (N = 1e6: 83 % of the issue slots
// busy, 348 warp instructions per warp of cells and step).  sm_100a multiplies, adds and
// fuses two floats per instruction (f32x2), each half rounded as the scalar instruction
// rounds it, so a thread that advances two cells of the same population issues half the
// stage arithmetic, and shares the step's loop, schedule and event test between them:
// 61 M warp instructions per window at N = 1e6 instead of 125 M, 105 us instead of 150 us
// (with 24 M and 33 us in the draws, which that figure included: poisson_window.cuh);
// N = 1e7: 1.37 -> 1.09 ms per window with the draws.  Cells j and j + blockDim.x share a thread, so every load
// and store stays coalesced and nothing depends on the alignment of the arrays.
//
// Every rounding is written out (fma2, mul2, add2 name one rounding each), and they are
// the roundings of the scalar form (adex_coef, adex_rhs_folded, astro_rhs_fast,
// neuron_ode_step, astro_advance): the per-step kernel and this one give the same bits.
#pragma once

#include "window_kernels.cuh"

namespace astrosim {

// The pair bodies, defined for R = float (the measurement build with IEEE float functions
// advances one cell per thread and has none).
template <typename R, bool EXC>
__device__ void neuron_pair_window(const RunConsts& rc, const NetScalars& ns, const StepPtrs<R>& p,
                                   const WinPtrs<R>& w, u32 j0, bool have1, i64 win_start, int s_begin, int s_end,
                                   int buf, bool window_done);
template <typename R>
__device__ void astro_pair_window(const RunConsts& rc, const NetScalars& ns, const StepPtrs<R>& p, const WinPtrs<R>& w,
                                  u32 a0, bool have1, i64 win_start, int s_begin, int s_end, int buf, i64 mark,
                                  bool window_done, bool& active0, bool& active1);

#ifndef ASTROSIM_FP32_IEEE

struct f32x2 {
    unsigned long long v;
};
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ f32x2 both(float x) { return pack2(x, x); }
__device__ __forceinline__ f32x2 pv(u64 both_halves) { return f32x2{both_halves}; }  // a PairK constant
__device__ __forceinline__ float lo2(f32x2 a) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
    return lo;
}
__device__ __forceinline__ float hi2(f32x2 a) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
    return hi;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f32x2 ex2_2(f32x2 a) { return pack2(ex2_ftz(lo2(a)), ex2_ftz(hi2(a))); }
__device__ __forceinline__ f32x2 rcp2(f32x2 a) { return pack2(rcp_ftz(lo2(a)), rcp_ftz(hi2(a))); }

// h6 (k1 + 2 k2 + 2 k3 + k4); the products by 2 are exact
__device__ __forceinline__ f32x2 rk4_sum(f32x2 h6, f32x2 k1, f32x2 k2, f32x2 k3, f32x2 k4) {
    const f32x2 two = both(2.0f);
    return mul2(h6, add2(fma2(two, k3, fma2(two, k2, k1)), k4));
}

// ------------------------------------------------------------------ neurons
// adex_coef and adex_rhs_folded of both cells at one set of conductances
struct AdexPairStage {
    const AdexPairK& c;
    f32x2 A, B;
    __device__ __forceinline__ AdexPairStage(const AdexPairK& k, f32x2 g_ex, f32x2 g_in, f32x2 iext_c)
        : c(k), A(fma2(pv(k.neg_inv_Cm), add2(g_ex, g_in), pv(k.A0))),
          B(fma2(g_ex, pv(k.Eex_c), fma2(g_in, pv(k.Ein_c), iext_c))) {}
    __device__ __forceinline__ void operator()(f32x2 V, f32x2 w, f32x2& dV, f32x2& dw) const {
        const f32x2 Vc = pack2(fminf(lo2(V), c.V_peak), fminf(hi2(V), c.V_peak));
        const f32x2 u = add2(Vc, pv(c.neg_E_L));
        const f32x2 spike = ex2_2(fma2(add2(Vc, pv(c.neg_V_th)), pv(c.K1), pv(c.K2)));
        dV = add2(fma2(A, u, fma2(pv(c.neg_inv_Cm), w, B)), spike);
        dw = fma2(pv(c.Wa), u, mul2(pv(c.neg_inv_tauw), w));
    }
};

// Neurons j0 and j1 = j0 + blockDim.x (when have1) through steps
// [s_begin, s_end); see neuron_window for the meaning of `special`.  The rare parts run in
// loops over the two cells, so that their code is there once.
template <typename R, bool EXC>
__device__ __forceinline__ void neuron_pair_window(const RunConsts& rc, const NetScalars& ns, const StepPtrs<R>& p,
                                                   const WinPtrs<R>& w, u32 j0, bool have1,
                                                   i64 win_start, int s_begin, int s_end, int buf,
                                                   bool window_done) {
    static_assert(std::is_same<R, float>::value, "FP32 form");
    const u64 nN = ns.n_neurons;
    const NeuronK& pk = EXC ? rc.pe : rc.pi;
    const u32 j1 = have1 ? j0 + blockDim.x : j0;  // without a second cell, the first one's state, never stored
    const InboxState inbox0 = inbox_state<float>(ns, w, j0, buf), inbox1 = inbox_state<float>(ns, w, j1, buf);
    const int pull = w.mode[buf];
    u64 counts0 = w.events[j0] >> (4 * s_begin), counts1 = w.events[j1] >> (4 * s_begin);
    double V0 = p.V[j0], V1 = p.V[j1], w0 = p.w[j0], w1 = p.w[j1];
    f32x2 g_ex = pack2(p.g_ex[j0], p.g_ex[j1]), dg_ex = pack2(p.dg_ex[j0], p.dg_ex[j1]);
    f32x2 g_in = pack2(p.g_in[j0], p.g_in[j1]), dg_in = pack2(p.dg_in[j0], p.dg_in[j1]);
    f32x2 I_sic = pack2(p.I_sic[j0], p.I_sic[j1]);
    int refr0 = p.refr[j0], refr1 = p.refr[j1];
    const int refr0_in = refr0, refr1_in = refr1;
    const f32x2 I_sic0 = I_sic;

    WindowSchedule sched = window_schedule(rc, win_start, s_begin, s_end);
    const double lambda = EXC ? ns.lambda_exc : ns.lambda_inh;
    const double limit = EXC ? ns.limit_exc : ns.limit_inh;
    const u64 lim53 = EXC ? ns.lim53_exc : ns.lim53_inh;
    const double nstd_d = EXC ? rc.noise_exc : rc.noise_inh;
    const float nstd = static_cast<float>(nstd_d);
    const bool has_noise = nstd_d > 0.0 && rc.independent_noise;
    auto noise_of = [&](u32 j) {
        return nstd * normal_fast(rng_base(ns.seed ^ kNeuronNoiseKey, sched.noise_idx * kNoiseStride + j));
    };
    f32x2 noise = both(0.0f);
    if (has_noise) noise = pack2(noise_of(j0), noise_of(j1));
    const Deposit<float> first0 = first_deposit<float>(ns, w, j0, buf, inbox0),
                         first1 = first_deposit<float>(ns, w, j1, buf, inbox1);
    const u32 exact0 = exact_steps(counts0) << s_begin, exact1 = exact_steps(counts1) << s_begin;

    WindowInput<float> x[2];
    x[1].mask = 0;
    x[1].sic = false;
    // a refresh without SIC input sets the current to w_a2n * 0
    const float no_sic = ns.f_w_a2n * 0.0f;
    bool sic_changes = lo2(I_sic) != no_sic || hi2(I_sic) != no_sic;
    u32 special = 0;
#pragma unroll 1
    for (int i = 0; i < (have1 ? 2 : 1); ++i) {
        window_input<float>(ns, p, w, i ? j1 : j0, i ? inbox1 : inbox0, i ? first1 : first0, s_begin, s_end, buf,
                            pull != 0, window_done, x[i]);
        special |= x[i].mask;
        sic_changes = sic_changes || x[i].sic;
    }
    special |= (has_noise ? sched.noise : 0u) | (sic_changes ? sched.refresh : 0u);
    special |= exact0 | exact1;
    // a weight that is not finite makes even an empty sum's input NaN at every step
    const float weight = EXC ? rc.f_weight_exc : rc.f_weight_inh;
    if (!(rc.f_w_e * 0.0f == 0.0f && rc.f_neg_w_i * 0.0f == 0.0f && weight * 0.0f == 0.0f)) special = 0xFFFFFFFFu;

    auto external = [&] {
        return fma2(has_noise ? add2(I_sic, noise) : I_sic, both(pk.f_inv_Cm), both(pk.f_C0));
    };
    f32x2 iext_c = external();

    const AdexPairK& k = EXC ? rc.pair_e : rc.pair_i;
    const f32x2 psc_ex = pv(k.psc_ex), psc_in = pv(k.psc_in), ex_decay = pv(k.ex_decay), in_decay = pv(k.in_decay);
    const f32x2 hs = pv(rc.pair_hs), half_hs = pv(rc.pair_half_hs), h6 = pv(rc.pair_h6), half = both(0.5f);
    u32 word0 = 0, word1 = 0;
    for (int st = s_begin; st < s_end; ++st) {
        const u32 events0 = static_cast<u32>(counts0) & kExactCount, events1 = static_cast<u32>(counts1) & kExactCount;
        counts0 >>= 4;
        counts1 >>= 4;
        f32x2 exc_input = mul2(both(weight), pack2(static_cast<float>(events0), static_cast<float>(events1)));
        if ((special >> st) & 1u) {
            float in[2][3];  // excitatory input, inhibitory sum, SIC sum
#pragma unroll 1
            for (int i = 0; i < 2; ++i) {
                const bool has = (x[i].mask >> st) & 1u;
                int events = static_cast<int>(i ? events1 : events0);
                if (events == static_cast<int>(kExactCount))
                    events = poisson_exact(step_base(ns.seed, kNeuronPoissonKey, win_start + st, i ? j1 : j0), lambda,
                                           limit, lim53);
                in[i][0] = exc_input_of<float>(rc, EXC, has ? x[i].ex[st] : 0.0f, events);
                in[i][1] = has ? x[i].in[st] : 0.0f;
                in[i][2] = x[i].sic ? x[i].sic_sum[st] : 0.0f;
            }
            exc_input = pack2(in[0][0], in[1][0]);
            dg_in = fma2(mul2(both(rc.f_neg_w_i), pack2(in[0][1], in[1][1])), psc_in, dg_in);
            if ((sched.refresh >> st) & 1u) I_sic = mul2(both(ns.f_w_a2n), pack2(in[0][2], in[1][2]));
            if (has_noise && ((sched.noise >> st) & 1u)) {
                ++sched.noise_idx;
                noise = pack2(noise_of(j0), noise_of(j1));
            }
            iext_c = external();
        }
        dg_ex = fma2(exc_input, psc_ex, dg_ex);
        for (int sub = 0; sub < rc.substeps; ++sub) {
            const f32x2 g_ex_next = mul2(ex_decay, fma2(hs, dg_ex, g_ex));
            const f32x2 g_in_next = mul2(in_decay, fma2(hs, dg_in, g_in));
            const f32x2 v = pack2(static_cast<float>(V0), static_cast<float>(V1));
            const f32x2 ww = pack2(static_cast<float>(w0), static_cast<float>(w1));
            f32x2 k1V, k1w, k2V, k2w, k3V, k3w, k4V, k4w;
            const AdexPairStage r1(k, g_ex, g_in, iext_c);
            r1(v, ww, k1V, k1w);
            const AdexPairStage rm(k, mul2(half, add2(g_ex, g_ex_next)), mul2(half, add2(g_in, g_in_next)), iext_c);
            rm(fma2(half_hs, k1V, v), fma2(half_hs, k1w, ww), k2V, k2w);
            rm(fma2(half_hs, k2V, v), fma2(half_hs, k2w, ww), k3V, k3w);
            const AdexPairStage r4(k, g_ex_next, g_in_next, iext_c);
            r4(fma2(hs, k3V, v), fma2(hs, k3w, ww), k4V, k4w);
            const f32x2 dV = rk4_sum(h6, k1V, k2V, k3V, k4V), dw = rk4_sum(h6, k1w, k2w, k3w, k4w);
            // the threshold test runs in double (src/astrosim_fused.cu:541-558)
            auto spike = [&](double& V, double& wv, int& refr, u32& word, u32 j) {
                V = p.V_reset[j];
                wv += p.b[j];
                refr = pk.ref_steps;
                word |= 1u << st;
            };
            if (refr0 > 0 || refr1 > 0) {
                auto advance = [&](double& V, double& wv, float dVf, float dwf, int& refr, u32& word, u32 j, float gx,
                                   float gi, float ic) {
                    if (refr > 0) {  // clamped: V at its reset value, w by an Euler step
                        V = p.V_reset[j];
                        const AdexCoef c{fmaf(-pk.f_inv_Cm, gx + gi, pk.f_A0),
                                         fmaf(gx, pk.f_Eex_c, fmaf(gi, pk.f_Ein_c, ic))};
                        adex_rhs_folded(pk, c, static_cast<float>(V), static_cast<float>(wv), dVf, dwf);
                        wv += static_cast<double>(rc.f_h_step * dwf);
                        --refr;
                    } else {
                        V += static_cast<double>(dVf);
                        wv += static_cast<double>(dwf);
                        if (V >= pk.V_peak) spike(V, wv, refr, word, j);
                    }
                };
                advance(V0, w0, lo2(dV), lo2(dw), refr0, word0, j0, lo2(g_ex), lo2(g_in), lo2(iext_c));
                advance(V1, w1, hi2(dV), hi2(dw), refr1, word1, j1, hi2(g_ex), hi2(g_in), hi2(iext_c));
            } else {
                V0 += static_cast<double>(lo2(dV));
                V1 += static_cast<double>(hi2(dV));
                w0 += static_cast<double>(lo2(dw));
                w1 += static_cast<double>(hi2(dw));
                if (V0 >= pk.V_peak || V1 >= pk.V_peak) {
                    if (V0 >= pk.V_peak) spike(V0, w0, refr0, word0, j0);
                    if (V1 >= pk.V_peak) spike(V1, w1, refr1, word1, j1);
                }
            }
            g_ex = g_ex_next;
            dg_ex = mul2(ex_decay, dg_ex);
            g_in = g_in_next;
            dg_in = mul2(in_decay, dg_in);
        }
        if (((word0 | word1) >> st) & 1u) {
#pragma unroll 1
            for (int i = 0; i < (have1 ? 2 : 1); ++i)
                if (((i ? word1 : word0) >> st) & 1u) record_spike<float>(rc, ns, p, w, i ? j1 : j0, win_start, st, buf);
        }
    }
    auto store = [&](u32 j, double V, double wv, float gx, float dgx, float gi, float dgi, float isic, float isic_in,
                     int refr, int refr_in, u32 word) {
        p.V[j] = V;
        p.w[j] = wv;
        p.g_ex[j] = gx;
        p.dg_ex[j] = dgx;
        p.g_in[j] = gi;
        p.dg_in[j] = dgi;
        if (isic != isic_in) p.I_sic[j] = isic;
        if (refr != refr_in) p.refr[j] = refr;
        u32* sw = w.spk_word + static_cast<u64>(buf) * nN + j;
        *sw = s_begin == 0 ? word : (*sw | word);
    };
    store(j0, V0, w0, lo2(g_ex), lo2(dg_ex), lo2(g_in), lo2(dg_in), lo2(I_sic), lo2(I_sic0), refr0, refr0_in, word0);
    if (have1)
        store(j1, V1, w1, hi2(g_ex), hi2(dg_ex), hi2(g_in), hi2(dg_in), hi2(I_sic), hi2(I_sic0), refr1, refr1_in,
              word1);
}

// ------------------------------------------------------------------ astrocytes
// astro_rhs_fast of both cells, with the gating variable held as nh = -h: a product or a
// fused operation with one sign turned gives exactly the negative, so that every minus
// sign of the formula sits in a constant and costs nothing.
struct AstroPair {
    f32x2 neg_1p_inv_ratio, Kd1, Kd_act, rate_Km2, Km2, neg_rate_SERCA, neg_channel, leak, neg_k_Kd_inh, Kd2, neg_k_IP3R;
    f32x2 Ct_ratio, neg_inv_tI, I0_tau;  // per cell: Ca_tot / ratio, -1 / tau_IP3, IP3_0 / tau_IP3
    __device__ __forceinline__ AstroPair(const AstroK& c, f32x2 Ct, f32x2 I0, f32x2 inv_tI)
        : neg_1p_inv_ratio(both(-c.f_1p_inv_ratio)), Kd1(both(c.f_Kd_IP3_1)), Kd_act(both(c.f_Kd_act)),
          rate_Km2(both(c.f_rate_Km2)), Km2(both(c.f_Km2)), neg_rate_SERCA(both(-c.f_rate_SERCA)),
          neg_channel(both(-c.f_ratio_rate_IP3R)), leak(both(c.f_ratio_rate_L)), neg_k_Kd_inh(both(-c.f_k_Kd_inh)),
          Kd2(both(c.f_Kd_IP3_2)), neg_k_IP3R(both(-c.f_k_IP3R)),
          Ct_ratio(mul2(Ct, both(c.f_inv_ratio))), neg_inv_tI(mul2(both(-1.0f), inv_tI)), I0_tau(mul2(I0, inv_tI)) {}
    __device__ __forceinline__ void operator()(f32x2 Ca, f32x2 IP3, f32x2 nh, f32x2 noise, f32x2& dCa, f32x2& dIP3,
                                               f32x2& dnh) const {
        const f32x2 d = fma2(Ca, neg_1p_inv_ratio, Ct_ratio);
        const f32x2 ip_k1 = add2(IP3, Kd1);
        const f32x2 mn = mul2(mul2(IP3, Ca), rcp2(mul2(ip_k1, add2(Ca, Kd_act))));
        const f32x2 mn3 = mul2(mul2(mn, mn), mn);
        const f32x2 nh3 = mul2(mul2(nh, nh), nh);
        const f32x2 neg_pump = fma2(rate_Km2, rcp2(fma2(Ca, Ca, Km2)), neg_rate_SERCA);
        dCa = fma2(d, fma2(mul2(neg_channel, mn3), nh3, leak), add2(noise, neg_pump));
        const f32x2 neg_alpha = mul2(mul2(neg_k_Kd_inh, ip_k1), rcp2(add2(IP3, Kd2)));
        dIP3 = fma2(IP3, neg_inv_tI, I0_tau);
        dnh = fma2(nh, fma2(neg_k_IP3R, Ca, neg_alpha), neg_alpha);
    }
};

// Astrocytes a0 and a1 = a0 + blockDim.x through steps [s_begin, s_end); active0/1
// receive whether their SIC factors were positive at any of them.
template <typename R>
__device__ __forceinline__ void astro_pair_window(const RunConsts& rc, const NetScalars& ns, const StepPtrs<R>& p,
                                                  const WinPtrs<R>& w, u32 a0, bool have1, i64 win_start, int s_begin,
                                                  int s_end, int buf, i64 mark, bool window_done,
                                                  bool& active0, bool& active1) {
    static_assert(std::is_same<R, float>::value, "FP32 form");
    const u32 a1 = have1 ? a0 + blockDim.x : a0;
    const u32* deposits = w.ain_cnt + static_cast<u64>(buf) * ns.n_astro;
    const u32 deposits0 = deposits[a0], deposits1 = deposits[a1];
    const int pull = w.mode[buf];
    AstroRegs<float> s0 = load_astro<float>(p.Ca[a0], p.IP3[a0], p.h[a0], p.Ca_tot[a0], p.IP3_0[a0], p.tau_IP3[a0],
                                            p.delta_IP3[a0]);
    AstroRegs<float> s1 = load_astro<float>(p.Ca[a1], p.IP3[a1], p.h[a1], p.Ca_tot[a1], p.IP3_0[a1], p.tau_IP3[a1],
                                            p.delta_IP3[a1]);
    const AstroPair f(rc.ak, pack2(s0.Ct, s1.Ct), pack2(s0.I0, s1.I0), pack2(s0.inv_tI, s1.inv_tI));
    f32x2 nh = pack2(-s0.h, -s1.h);
    AstroInput<float> x[2];
    x[1].mask = 0;
    // a weight that is not finite makes even an empty sum's input NaN at every step
    u32 input = rc.f_w_n2a * 0.0f == 0.0f ? 0u : 0xFFFFFFFFu;
#pragma unroll 1
    for (int i = 0; i < (have1 ? 2 : 1); ++i) {
        astro_input<float>(ns, p, w, i ? a1 : a0, i ? deposits1 : deposits0, s_begin, s_end, buf, pull != 0,
                           window_done, x[i]);
        input |= x[i].mask;
    }
    SicWriter<float> out0(p, w, ns, a0, buf, s_begin), out1(p, w, ns, a1, buf, s_begin);
    const u64 gap = static_cast<u64>(a1 - a0) * kStreamMul;
    u64 pbase = step_base(ns.seed, kAstroPoissonKey, win_start + s_begin, a0);
    u64 nbase = step_base(ns.seed, kAstroNoiseKey, win_start + s_begin, a0);
    const bool drive = ns.lambda_astro > 0.0;
    // an event needs a first draw above the limit (rng_poisson_at settles an equal upper part)
    const u32 lim_hi = static_cast<u32>(ns.lim53_astro >> 21);
    const bool has_noise = rc.noise_astro > 0.0;
    i64 rphase = p.ca_rec ? (win_start + s_begin + 1) % p.rec_every : 1;
    const f32x2 hs = both(rc.f_h_step), half_hs = both(0.5f * rc.f_h_step), h6 = both(rc.f_h6);
    for (int st = s_begin; st < s_end; ++st) {
        const i64 t = win_start + st;
        const bool ev0 = drive && rng_mix_hi(pbase) >= lim_hi, ev1 = drive && rng_mix_hi(pbase + gap) >= lim_hi;
        if (ev0 || ev1 || ((input >> st) & 1u)) {
            float in[2];
#pragma unroll 1
            for (int i = 0; i < 2; ++i)
                in[i] = astro_kick<float>(rc, ns, ((x[i].mask >> st) & 1u) ? x[i].sum[st] : 0.0f, pbase + (i ? gap : 0));
            if (in[0] != 0.0f) s0.IP3 += s0.delta_IP3 * static_cast<double>(in[0]);
            if (in[1] != 0.0f) s1.IP3 += s1.delta_IP3 * static_cast<double>(in[1]);
        }
        f32x2 noise = both(0.0f);
        if (has_noise) {  // normal_fast of both cells
            u64 b0 = nbase, b1 = nbase + gap;
            if (!rc.independent_noise)
                b0 = b1 = rng_base(ns.seed ^ kAstroNoiseKey, static_cast<u64>(t / rc.steps_per_noise));
            const f32x2 unit = both(1.0f / 16777216.0f);
            const f32x2 u1 = mul2(add2(pack2(static_cast<float>(rng_mix_hi(b0) >> 8),
                                             static_cast<float>(rng_mix_hi(b1) >> 8)), both(0.5f)), unit);
            const f32x2 u2 = mul2(pack2(static_cast<float>(rng_mix_hi(b0 + kCounterMul) >> 8),
                                        static_cast<float>(rng_mix_hi(b1 + kCounterMul) >> 8)), unit);
            const f32x2 l = mul2(both(-2.0f), mul2(pack2(lg2_ftz(lo2(u1)), lg2_ftz(hi2(u1))), both(kLn2)));
            const f32x2 th = mul2(both(static_cast<float>(kTwoPi)), u2);
            noise = mul2(both(rc.f_noise_astro), mul2(pack2(sqrt_ftz(lo2(l)), sqrt_ftz(hi2(l))),
                                                      pack2(cos_ftz(lo2(th)), cos_ftz(hi2(th)))));
        }
        pbase += kStepAdvance;
        nbase += kStepAdvance;
        for (int sub = 0; sub < rc.substeps; ++sub) {  // astro_advance (src/astrosim_fused.cu:255-278)
            const f32x2 ca = pack2(static_cast<float>(s0.Ca), static_cast<float>(s1.Ca));
            const f32x2 ip = pack2(static_cast<float>(s0.IP3), static_cast<float>(s1.IP3));
            f32x2 k1c, k1i, k1h, k2c, k2i, k2h, k3c, k3i, k3h, k4c, k4i, k4h;
            f(ca, ip, nh, noise, k1c, k1i, k1h);
            f(fma2(half_hs, k1c, ca), fma2(half_hs, k1i, ip), fma2(half_hs, k1h, nh), noise, k2c, k2i, k2h);
            f(fma2(half_hs, k2c, ca), fma2(half_hs, k2i, ip), fma2(half_hs, k2h, nh), noise, k3c, k3i, k3h);
            f(fma2(hs, k3c, ca), fma2(hs, k3i, ip), fma2(hs, k3h, nh), noise, k4c, k4i, k4h);
            const f32x2 dc = rk4_sum(h6, k1c, k2c, k3c, k4c), di = rk4_sum(h6, k1i, k2i, k3i, k4i);
            const f32x2 two = both(2.0f);
            const f32x2 hn = fma2(h6, add2(fma2(two, k3h, fma2(two, k2h, k1h)), k4h), nh);
            auto unit_clamp = [](float x) { return x > 0.0f ? 0.0f : (x < -1.0f ? -1.0f : x); };  // h in [0, 1]
            nh = pack2(unit_clamp(lo2(hn)), unit_clamp(hi2(hn)));
            auto settle = [](AstroRegs<float>& s, float dCa, float dIP3) {
                s.Ca += static_cast<double>(dCa);
                s.IP3 += static_cast<double>(dIP3);
                s.Ca = s.Ca < 0.0 ? 0.0 : (s.Ca > s.Ca_tot ? s.Ca_tot : s.Ca);
                s.IP3 = s.IP3 < 0.0 ? 0.0 : s.IP3;
            };
            settle(s0, lo2(dc), lo2(di));
            settle(s1, hi2(dc), hi2(di));
        }
        if (p.ca_rec) {
            record_ca<float>(p, a0, t, rphase == 0, s0.Ca);
            if (have1) record_ca<float>(p, a1, t, rphase == 0, s1.Ca);
            if (++rphase == p.rec_every) rphase = 0;
        }
        out0.step(st, sic_factor<float>(rc, s0.Ca), t == mark, true);
        out1.step(st, sic_factor<float>(rc, s1.Ca), t == mark, have1);
    }
    auto store = [&](u32 a, const AstroRegs<float>& s, float hv, const SicWriter<float>& o) {
        p.Ca[a] = s.Ca;
        p.IP3[a] = s.IP3;
        p.h[a] = hv;
        o.finish(p, a);
    };
    store(a0, s0, -lo2(nh), out0);
    if (have1) store(a1, s1, -hi2(nh), out1);
    active0 = out0.any;
    active1 = have1 && out1.any;
}

#endif  // ASTROSIM_FP32_IEEE

}  // namespace astrosim
