// window_kernels.cuh -- device bodies of the windowed engine, shared by the
// single-network kernels (window.cu) and the batched ensemble kernels (ensemble.cu).
#pragma once

#include "poisson_window.cuh"
#include "step_kernels.cuh"
#include "window.cuh"
#include "window_schedule.cuh"

namespace astrosim {

template <typename R>
struct WinPtrs {
    u32 *nin_cnt, *ain_cnt;          // [2][n]
    Deposit<R> *nin_ent, *ain_ent;   // [2][n][kInboxSlots]
    u32* spk_word;                   // [2][n_neurons]
    R* spk_val;                      // [2][W][n_neurons]
    u32* spk_list;                   // [2][cap]
    u32* spk_count;                  // [2]
    R* sic_win;                      // [2][n_astro][W]
    u32* astro_active;               // [2][astro_words]
    u32* sic_pos;                    // [2][n_neurons]
    int* mode;                       // [2]
    u64* events;                     // [n_neurons]
    const u32 *fe_rs, *fe_dst, *fi_rs, *fi_dst, *fa_rs, *fa_astro, *fa_pos, *fs_rs, *fs_dst;
    u32 cap, push_limit, astro_words;
    int W;
};

template <typename R>
inline WinPtrs<R> win_ptrs(WindowState& ws, const RunConsts& rc) {
    WinPtrs<R> w{};
    w.nin_cnt = ws.nin_cnt.get();
    w.ain_cnt = ws.ain_cnt.get();
    w.nin_ent = reinterpret_cast<Deposit<R>*>(ws.nin_ent.get());
    w.ain_ent = reinterpret_cast<Deposit<R>*>(ws.ain_ent.get());
    w.spk_word = ws.spk_word.get();
    w.spk_val = reinterpret_cast<R*>(ws.spk_val.get());
    w.spk_list = ws.spk_list.get();
    w.spk_count = ws.spk_count.get();
    w.sic_win = reinterpret_cast<R*>(ws.sic_win.get());
    w.astro_active = ws.astro_active.get();
    w.sic_pos = ws.sic_pos.get();
    w.mode = ws.mode.get();
    w.events = ws.events.get();
    w.fe_rs = ws.fwd.exc_rs.get();
    w.fe_dst = ws.fwd.exc_dst.get();
    w.fi_rs = ws.fwd.inh_rs.get();
    w.fi_dst = ws.fwd.inh_dst.get();
    w.fa_rs = ws.fwd.e2a_rs.get();
    w.fa_astro = ws.fwd.e2a_astro.get();
    w.fa_pos = ws.fwd.e2a_pos.get();
    w.fs_rs = ws.fwd.sic_rs.get();
    w.fs_dst = ws.fwd.sic_dst.get();
    w.cap = ws.push_limit + 1;
    w.push_limit = ws.push_limit;
    w.astro_words = (rc.n_astro + 31) / 32;
    w.W = ws.W;
    return w;
}

// Sorts deposits by (step, kind, key): the order in which the reference's dense
// gather meets them (row order within one step and kind).
template <typename R>
__device__ __forceinline__ void sort_deposits(Deposit<R>* d, int n) {
    for (int i = 1; i < n; ++i) {
        const Deposit<R> x = d[i];
        const unsigned long long kx = (static_cast<unsigned long long>(x.meta) << 32) | x.key;
        int k = i - 1;
        while (k >= 0 && ((static_cast<unsigned long long>(d[k].meta) << 32) | d[k].key) > kx) {
            d[k + 1] = d[k];
            --k;
        }
        d[k + 1] = x;
    }
}

// Per-step sums of one CSR row against the previous window's spike words, in row
// order (the exact fallback when deposits are not available).
template <typename R>
__device__ __forceinline__ void pull_row(const u32* __restrict__ rs, const u32* __restrict__ src, u32 row,
                                         const u32* __restrict__ words, const R* __restrict__ vals, u64 n_neurons,
                                         int s0, int s1, R* acc) {
    const u32 k1 = rs[row + 1];
    for (u32 k = rs[row]; k < k1; ++k) {
        const u32 s = src[k];
        u32 wd = words[s];
        if (!wd) continue;
        wd &= ((s1 >= 32 ? 0xFFFFFFFFu : ((1u << s1) - 1u)) & ~((1u << s0) - 1u));
        while (wd) {
            const int b = __ffs(wd) - 1;
            wd &= wd - 1;
            acc[b] += vals[static_cast<u64>(b) * n_neurons + s];
        }
    }
}

__device__ __forceinline__ WindowSchedule window_schedule(const RunConsts& rc, i64 win_start, int s_begin, int s_end) {
    return window_schedule(rc.d_a2n, rc.sic_interval, rc.steps_per_noise, win_start, s_begin, s_end);
}

// The synaptic input of one neuron over a window: excitatory and inhibitory sums of the
// steps whose bit is set in `mask` (the others have none).
template <typename R>
struct WindowInput {
    R ex[kMaxWindow], in[kMaxWindow];
    u32 mask;
};

// What says whether a neuron has any input at all.  It is loaded with the state at the
// window's start and the first deposit (the usual neuron with input has one) right after
// the noise draw, so that neither load is waited for on its own.
struct InboxState {
    u32 count, sic;  // deposits; positions of active astrocytes in its a2n row (sic_pos)
};
template <typename R>
__device__ __forceinline__ InboxState inbox_state(const NetScalars& ns, const WinPtrs<R>& w, u32 j, int buf) {
    return InboxState{w.nin_cnt[static_cast<u64>(buf) * ns.n_neurons + j],
                      w.sic_pos[static_cast<u64>(buf) * ns.n_neurons + j]};
}
template <typename R>
__device__ __forceinline__ Deposit<R> first_deposit(const NetScalars& ns, const WinPtrs<R>& w, u32 j, int buf,
                                                    const InboxState& inbox) {
    Deposit<R> d{0, 0, static_cast<R>(0.0)};
    if (inbox.count) d = w.nin_ent[(static_cast<u64>(buf) * ns.n_neurons + j) * kInboxSlots];
    return d;
}

template <typename R>
__device__ __forceinline__ void window_input(const NetScalars& ns, const StepPtrs<R>& p, const WinPtrs<R>& w, u32 j,
                                             const InboxState& inbox, const Deposit<R>& first, int s_begin, int s_end,
                                             int buf, bool pull, bool window_done, WindowInput<R>& x) {
    const int prev = buf ^ 1;
    const int W = w.W;
    const u64 nN = ns.n_neurons;
    x.mask = 0;
    // deposits (push) or the row walk (pull)
    const u64 slot_base = static_cast<u64>(buf) * nN + j;
    const u32 c = inbox.count;
    if (pull || c > kInboxSlots) {
        for (int i = 0; i < W; ++i) x.ex[i] = x.in[i] = static_cast<R>(0.0);
        x.mask = (1u << W) - 1u;
        const u32* words = w.spk_word + static_cast<u64>(prev) * nN;
        const R* vals = w.spk_val + static_cast<u64>(prev) * W * nN;
        pull_row<R>(p.exc_rs, p.exc_src, j, words, vals, nN, s_begin, s_end, x.ex);
        pull_row<R>(p.inh_rs, p.inh_src, j, words, vals, nN, s_begin, s_end, x.in);
    } else if (c == 1) {  // the usual case: nothing to sort or sum
        const int st = static_cast<int>(first.meta & 0xFFu);
        if (st >= s_begin && st < s_end) {
            x.ex[st] = (first.meta >> 8) == 0 ? first.val : static_cast<R>(0.0);
            x.in[st] = (first.meta >> 8) == 0 ? static_cast<R>(0.0) : first.val;
            x.mask = 1u << st;
        }
    } else if (c > 0) {
        Deposit<R> d[kInboxSlots];
        for (u32 i = 0; i < c; ++i) d[i] = w.nin_ent[slot_base * kInboxSlots + i];
        sort_deposits<R>(d, static_cast<int>(c));
        for (u32 i = 0; i < c; ++i) {
            const int st = static_cast<int>(d[i].meta & 0xFFu);
            if (st < s_begin || st >= s_end) continue;
            const u32 bit = 1u << st;
            if (!(x.mask & bit)) {
                x.ex[st] = x.in[st] = static_cast<R>(0.0);
                x.mask |= bit;
            }
            if ((d[i].meta >> 8) == 0) x.ex[st] += d[i].val;
            else x.in[st] += d[i].val;
        }
    }
    if (window_done && c) w.nin_cnt[slot_base] = 0;
    if (window_done && inbox.sic) w.sic_pos[slot_base] = 0;  // clean for the window after next
}

// SIC sums of a warp's 32 neurons over a window, by step: [W][kSicStride] of shared memory.
constexpr int kSicStride = 33;  // an odd stride: lanes of one neuron (by step) and of one step fall in different banks
template <typename R>
inline size_t sic_bytes(int W, int block) {
    return static_cast<size_t>(block / 32) * (static_cast<size_t>(W) * kSicStride * sizeof(R) + 32 * sizeof(u32));
}
template <typename R>
struct SicRows {
    R* sums;
    u32* list;  // 32 words of scratch
    __device__ __forceinline__ R at(int st) const { return sums[st * kSicStride + static_cast<int>(threadIdx.x & 31)]; }
};
template <typename R>
__device__ __forceinline__ SicRows<R> sic_rows(unsigned char* shared, int W) {
    const u32 sum_bytes = static_cast<u32>(W * kSicStride) * sizeof(R);
    unsigned char* mine = shared + (threadIdx.x >> 5) * (sum_bytes + 32 * static_cast<u32>(sizeof(u32)));
    return SicRows<R>{reinterpret_cast<R*>(mine), reinterpret_cast<u32*>(mine + sum_bytes)};
}

// Two adjacent factors, read with one load.
template <typename R>
struct alignas(2 * sizeof(R)) Factors2 {
    R a, b;
};

// Sums the previous window's SIC factors of lane l's neuron j, whose marked
// row positions are `marks` (0: nothing to sum, its sums stay unwritten).  Every lane of
// the warp takes part.  A group of lanes sums one neuron, each lane two steps (one where W
// is odd), so that an astrocyte's factors (W adjacent values) are read by adjacent lanes;
// a thread per neuron read them one by one and kept its sums in local memory (N = 1e6 FP32
// with 97 % of the astrocytes active: 440 of 568 us per window).  Each sum adds its row's
// factors in row order; the unmarked ones are 0.
template <typename R, int V>
__device__ __forceinline__ void sic_gather_by(const NetScalars& ns, const StepPtrs<R>& p, const WinPtrs<R>& w, u32 j,
                                              u32 marks, u32 flagged, int prev, const SicRows<R>& rows) {
    constexpr u32 kAll = 0xffffffffu;
    constexpr u32 kIds = 2;  // positions whose astrocytes a lane fetches at a time
    const u32 lane = threadIdx.x & 31;
    const u32 W = static_cast<u32>(w.W), width = W / V;  // lanes per neuron
    const R* fac = w.sic_win + static_cast<u64>(prev) * ns.n_astro * W;
    const u32* act = w.astro_active + static_cast<u64>(prev) * w.astro_words;
    const u32 row = marks ? p.sic_rs[j] : 0;
    if (marks) rows.list[__popc(flagged & ((1u << lane) - 1u))] = lane;
    __syncwarp();
    const u32 n = __popc(flagged), groups = 32 / width;
    const u32 g = lane / width, s = lane - g * width, base = g * width;
    for (u32 first = 0; first < n; first += groups) {
        const bool mine = g < groups && first + g < n;
        const u32 owner = mine ? rows.list[first + g] : 0;
        const u32 r0 = __shfl_sync(kAll, row, owner);
        const u32 m = __shfl_sync(kAll, marks, owner), owner_j = __shfl_sync(kAll, j, owner);
        u32 left = mine ? m & 0x7FFFFFFFu : 0u;
        R sum[2] = {static_cast<R>(0.0), static_cast<R>(0.0)};
        auto add = [&](u32 a, bool have) {  // astrocyte a's factors of this lane's steps
            Factors2<R> f{static_cast<R>(0.0), static_cast<R>(0.0)};
            if (have) {
                const R* at = fac + static_cast<u64>(a) * W + V * s;
                if (V == 2) f = *reinterpret_cast<const Factors2<R>*>(at);
                else f.a = *at;
            }
            return f;
        };
        const u32 chunk = width * kIds;
        for (u32 at = 0; __any_sync(kAll, left != 0); at += chunk, left = chunk < 32 ? left >> chunk : 0) {
            // the lanes of the group fetch the chunk's marked astrocytes (kNone elsewhere)
            constexpr u32 kNone = 0xFFFFFFFFu;
            const u32 now = chunk < 32 ? left & ((1u << chunk) - 1u) : left;
            u32 id[kIds];
#pragma unroll
            for (u32 q = 0; q < kIds; ++q) {
                const u32 pos = q * width + s;
                id[q] = (now >> pos) & 1u ? p.sic_src[r0 + at + pos] : kNone;
            }
            const u32 most = __reduce_max_sync(kAll, static_cast<u32>(__popc(now)));
            if (4 * most > chunk) {  // dense: every position in turn
#pragma unroll
                for (u32 q = 0; q < kIds; ++q)
                    for (u32 pos = 0; pos < width; pos += 5) {
                        Factors2<R> f[5];
#pragma unroll
                        for (u32 u = 0; u < 5; ++u) {
                            const u32 a = __shfl_sync(kAll, id[q], base + pos + u);
                            f[u] = add(a, a != kNone && pos + u < width);
                        }
#pragma unroll
                        for (u32 u = 0; u < 5; ++u) {
                            sum[0] += f[u].a;
                            if (V == 2) sum[1] += f[u].b;
                        }
                    }
            } else {  // sparse: the marked positions
                u32 rest = now;
                for (u32 k = 0; k < most; k += 2) {
                    Factors2<R> f[2];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const u32 pos = rest ? static_cast<u32>(__ffs(rest) - 1) : 0;
                        const bool upper = pos >= width;
                        const u32 from = base + (upper ? pos - width : pos);
                        const u32 a0 = __shfl_sync(kAll, id[0], from), a1 = __shfl_sync(kAll, id[1], from);
                        f[u] = add(upper ? a1 : a0, rest != 0);
                        rest &= rest - 1;
                    }
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        sum[0] += f[u].a;
                        if (V == 2) sum[1] += f[u].b;
                    }
                }
            }
        }
        if (mine && (m >> 31)) {  // positions from 31 on share the last mark
            const u32 end = p.sic_rs[owner_j + 1];
            for (u32 k = r0 + 31; k < end; ++k) {
                const u32 a = p.sic_src[k];
                const Factors2<R> f = add(a, (act[a >> 5] >> (a & 31)) & 1u);
                sum[0] += f.a;
                if (V == 2) sum[1] += f.b;
            }
        }
        if (mine)
#pragma unroll
            for (int v = 0; v < V; ++v)
                rows.sums[(V * s + v) * kSicStride + owner] = sum[v];
        __syncwarp();
    }
}
template <typename R>
__device__ __forceinline__ void sic_gather(const NetScalars& ns, const StepPtrs<R>& p, const WinPtrs<R>& w, u32 j,
                                           u32 marks, int prev, const SicRows<R>& rows) {
    const u32 flagged = __ballot_sync(0xffffffffu, marks != 0);
    if (!flagged) return;
    if (w.W % 2 == 0) sic_gather_by<R, 2>(ns, p, w, j, marks, flagged, prev, rows);
    else sic_gather_by<R, 1>(ns, p, w, j, marks, flagged, prev, rows);
}

// What a spike of neuron j at window step st leaves behind: its synaptic multiplier, a
// spike-list entry, its step's count and its raster bit.
template <typename R>
__device__ __forceinline__ void record_spike(const RunConsts& rc, const NetScalars& ns, const StepPtrs<R>& p,
                                             const WinPtrs<R>& w, u32 j, i64 win_start, int st, int buf) {
    const u64 nN = ns.n_neurons;
    const i64 t = win_start + st;
    const R out = stp_on_spike<R>(rc, p.stp_x[j], p.stp_u[j], p.stp_t[j], t);
    w.spk_val[(static_cast<u64>(buf) * w.W + st) * nN + j] = out;
    const u32 slot = atomicAdd(&w.spk_count[buf], 1u);
    if (slot < w.cap) w.spk_list[static_cast<u64>(buf) * w.cap + slot] = (j << 5) | static_cast<u32>(st);
    atomicAdd(&p.counts[t], 1u);
    if (t < p.raster_steps) atomicOr(&p.raster[static_cast<u64>(t) * ns.words + (j >> 5)], 1u << (j & 31));
}

// A neuron's registers over a window: neuron_ode_step on NeuronRegs, or in the FP32 form
// neuron_ode_step2 on NeuronRegs2.
template <typename R>
struct NeuronCore {
    NeuronRegs<R> n;
    R I_ext;
    __device__ __forceinline__ NeuronCore(const StepPtrs<R>& p, u32 j)
        : n{p.V[j],     p.w[j],     p.V_reset + j, p.b + j, p.g_ex[j],
            p.dg_ex[j], p.g_in[j], p.dg_in[j],    static_cast<R>(0.0), p.refr[j]},
          I_ext(static_cast<R>(0.0)) {}
    __device__ __forceinline__ void external(const NeuronK&, R I) { I_ext = I; }
    __device__ __forceinline__ bool step(const RunConsts& rc, const NeuronK& pk, R exc_input, R inh_input) {
        return neuron_ode_step<R>(rc, pk, n, exc_input, inh_input, I_ext, as_r<R>(pk.ex_decay, pk.f_ex_decay),
                                  as_r<R>(pk.in_decay, pk.f_in_decay));
    }
    __device__ __forceinline__ int refr() const { return n.refr; }
    __device__ __forceinline__ void store(const StepPtrs<R>& p, u32 j) const {
        p.V[j] = n.V;
        p.w[j] = n.w;
        p.g_ex[j] = n.g_ex;
        p.dg_ex[j] = n.dg_ex;
        p.g_in[j] = n.g_in;
        p.dg_in[j] = n.dg_in;
    }
};
#ifndef ASTROSIM_FP32_IEEE
template <>
struct NeuronCore<float> {
    NeuronRegs2 n;
    const double *V_reset, *b;
    float iext_c;
    __device__ __forceinline__ NeuronCore(const StepPtrs<float>& p, u32 j)
        : n{p.V[j], p.w[j], pack2(p.g_ex[j], p.g_in[j]), pack2(p.dg_ex[j], p.dg_in[j]), p.refr[j]},
          V_reset(p.V_reset + j), b(p.b + j), iext_c(0.0f) {}
    __device__ __forceinline__ void external(const NeuronK& pk, float I) { iext_c = fmaf(I, pk.f_inv_Cm, pk.f_C0); }
    __device__ __forceinline__ bool step(const RunConsts& rc, const NeuronK& pk, float exc_input, float inh_input) {
        return neuron_ode_step2(rc, pk, n, V_reset, b, pack2(exc_input, inh_input), iext_c);
    }
    __device__ __forceinline__ int refr() const { return n.refr; }
    __device__ __forceinline__ void store(const StepPtrs<float>& p, u32 j) const {
        p.V[j] = n.V;
        p.w[j] = n.w;
        p.g_ex[j] = lo2(n.g);
        p.dg_ex[j] = lo2(n.dg);
        p.g_in[j] = hi2(n.g);
        p.dg_in[j] = hi2(n.dg);
    }
};
#endif

// Neuron j through steps [s_begin, s_end) of the window starting at win_start.  Every lane
// of the warp calls it; those without a cell (!have) name any valid one.  Steps at which
// anything but the cell's own dynamics, its background events and its SIC input happens (a
// deposit, new noise, an exact Poisson draw) are rare and marked in `special`, so that the
// common step reads its event count and integrates.
template <typename R, bool EXC>
__device__ __forceinline__ void neuron_window(const RunConsts& rc, const NetScalars& ns, const NeuronK& pk,
                                              const StepPtrs<R>& p, const WinPtrs<R>& w, u32 j, bool have,
                                              i64 win_start, int s_begin, int s_end, int buf, bool window_done,
                                              const SicRows<R>& sic) {
    const u64 nN = ns.n_neurons;
    const InboxState inbox = inbox_state<R>(ns, w, j, buf);
    const int pull = w.mode[buf];
    u64 counts = w.events[j] >> (4 * s_begin);  // four bits per step, this step's lowest
    NeuronCore<R> n(p, j);
    R I_sic = p.I_sic[j];
    const R I_sic_in = I_sic;
    const int refr_in = n.refr();
    const double nstd = EXC ? rc.noise_exc : rc.noise_inh;
    const bool has_noise = nstd > 0.0 && rc.independent_noise;
    WindowSchedule sched = window_schedule(rc, win_start, s_begin, s_end);
    R noise = static_cast<R>(0.0);
    if (has_noise) noise = static_cast<R>(neuron_noise<R>(ns, nstd, sched.noise_idx, j));
    const Deposit<R> first = first_deposit<R>(ns, w, j, buf, inbox);
    const u32 exact = exact_steps(counts) << s_begin;
    sic_gather<R>(ns, p, w, j, have ? inbox.sic : 0u, buf ^ 1, sic);
    if (!have) return;
    WindowInput<R> x;
    window_input<R>(ns, p, w, j, inbox, first, s_begin, s_end, buf, pull != 0, window_done, x);
    u32 special = x.mask | exact | (has_noise ? sched.noise : 0u);
    // a weight that is not finite makes even an empty sum's input NaN at every step
    const R zero = static_cast<R>(0.0);
    const R weight = EXC ? as_r<R>(rc.weight_exc, rc.f_weight_exc) : as_r<R>(rc.weight_inh, rc.f_weight_inh);
    const R neg_w_i = as_r<R>(-rc.w_i, rc.f_neg_w_i);
    if (!(as_r<R>(rc.w_e, rc.f_w_e) * zero == zero && neg_w_i * zero == zero && weight * zero == zero))
        special = 0xFFFFFFFFu;
    // a refresh without SIC input sets the current to w_a2n * 0
    const R w_a2n = as_r<R>(ns.w_a2n, ns.f_w_a2n);
    const u32 refresh = inbox.sic || I_sic != w_a2n * zero ? sched.refresh : 0u;
    auto external = [&] { n.external(pk, has_noise ? I_sic + noise : I_sic); };
    external();
    u32 word = 0;
    for (int st = s_begin; st < s_end; ++st) {
        const int events = static_cast<int>(static_cast<u32>(counts) & kExactCount);
        counts >>= 4;
        R exc_input = weight * static_cast<R>(events), inh_input = zero;
        if (((special | refresh) >> st) & 1u) {
            if ((refresh >> st) & 1u) {
                I_sic = w_a2n * (inbox.sic ? sic.at(st) : zero);
                external();
            }
            if ((special >> st) & 1u) {
                const bool has = (x.mask >> st) & 1u;
                int drawn = events;
                if (events == static_cast<int>(kExactCount))
                    drawn = poisson_exact(step_base(ns.seed, kNeuronPoissonKey, win_start + st, j),
                                          EXC ? ns.lambda_exc : ns.lambda_inh, EXC ? ns.limit_exc : ns.limit_inh,
                                          EXC ? ns.lim53_exc : ns.lim53_inh);
                exc_input = exc_input_of<R>(rc, EXC, has ? x.ex[st] : zero, drawn);
                inh_input = neg_w_i * (has ? x.in[st] : zero);
                if (has_noise && ((sched.noise >> st) & 1u)) {
                    noise = static_cast<R>(neuron_noise<R>(ns, nstd, ++sched.noise_idx, j));
                    external();
                }
            }
        }
        if (n.step(rc, pk, exc_input, inh_input)) {
            record_spike<R>(rc, ns, p, w, j, win_start, st, buf);
            word |= 1u << st;
        }
    }
    n.store(p, j);
    if (I_sic != I_sic_in) p.I_sic[j] = I_sic;
    if (n.refr() != refr_in) p.refr[j] = n.refr();
    u32* sw = w.spk_word + static_cast<u64>(buf) * nN + j;
    *sw = s_begin == 0 ? word : (*sw | word);
}

// A block advances a tile of cells of one population, so that the population's constants
// are the same for the whole block.  The tiles of a cell range: astrocytes first (their
// steps are the longest), then the excitatory, then the inhibitory neurons.
enum CellKind : int { kExcCells = 0, kInhCells = 1, kAstroCells = 2 };
struct CellTiles {
    u32 lo[3], hi[3], tiles[3];  // by CellKind
    u32 tile;
};
inline CellTiles cell_tiles(u32 n_exc, u32 n_lo, u32 n_hi, u32 a_lo, u32 a_hi, u32 tile) {
    CellTiles t{};
    t.tile = tile;
    t.lo[kExcCells] = n_lo;
    t.hi[kExcCells] = n_hi < n_exc ? n_hi : n_exc;
    t.lo[kInhCells] = n_lo > n_exc ? n_lo : n_exc;
    t.hi[kInhCells] = n_hi;
    t.lo[kAstroCells] = a_lo;
    t.hi[kAstroCells] = a_hi;
    for (int k = 0; k < 3; ++k) t.tiles[k] = t.hi[k] > t.lo[k] ? ceil_div(t.hi[k] - t.lo[k], tile) : 0;
    return t;
}
inline u32 total_tiles(const CellTiles& t) { return t.tiles[0] + t.tiles[1] + t.tiles[2]; }

struct Tile {
    int kind;
    u32 base, end;  // cells [base, min(base + tile, end))
};
__device__ __forceinline__ Tile tile_of(const CellTiles& t, u32 blk) {
    int kind = kAstroCells;
    if (blk >= t.tiles[kAstroCells]) {
        blk -= t.tiles[kAstroCells];
        kind = kExcCells;
        if (blk >= t.tiles[kExcCells]) {
            blk -= t.tiles[kExcCells];
            kind = kInhCells;
        }
    }
    return Tile{kind, t.lo[kind] + blk * t.tile, t.hi[kind]};
}

// The IP3 input of one astrocyte over a window: the spike sums of the steps whose bit is
// set in `mask` (the others have none), from its `c` deposits.
template <typename R>
struct AstroInput {
    R sum[kMaxWindow];
    u32 mask;
};
template <typename R>
__device__ __forceinline__ void astro_input(const NetScalars& ns, const StepPtrs<R>& p, const WinPtrs<R>& w, u32 a, u32 c,
                                            int s_begin, int s_end, int buf, bool pull, bool window_done,
                                            AstroInput<R>& x) {
    const int prev = buf ^ 1;
    const int W = w.W;
    x.mask = 0;
    const u64 slot_base = (static_cast<u64>(buf) * ns.n_astro + a);
    if (pull || c > kInboxSlots) {
        for (int i = 0; i < W; ++i) x.sum[i] = static_cast<R>(0.0);
        x.mask = (1u << W) - 1u;
        pull_row<R>(p.e2a_rs, p.e2a_src, a, w.spk_word + static_cast<u64>(prev) * ns.n_neurons,
                    w.spk_val + static_cast<u64>(prev) * W * ns.n_neurons, ns.n_neurons, s_begin, s_end, x.sum);
    } else if (c > 0) {
        Deposit<R> d[kInboxSlots];
        for (u32 i = 0; i < c; ++i) d[i] = w.ain_ent[slot_base * kInboxSlots + i];
        sort_deposits<R>(d, static_cast<int>(c));
        for (u32 i = 0; i < c; ++i) {
            const int st = static_cast<int>(d[i].meta & 0xFFu);
            if (st < s_begin || st >= s_end) continue;
            const u32 bit = 1u << st;
            x.sum[st] = ((x.mask & bit) ? x.sum[st] : static_cast<R>(0.0)) + d[i].val;
            x.mask |= bit;
        }
    }
    if (window_done && c) w.ain_cnt[slot_base] = 0;
}

// The SIC factors of one astrocyte over a window.  A window's factors are read only for
// astrocytes marked active in it, so they are written only from the first positive one
// on (the steps before it as zeros); the second part of a split window continues what
// the first part marked.
template <typename R>
struct SicWriter {
    R* out;
    R last;
    unsigned char ever, ever_in;
    bool writing, any;
    __device__ __forceinline__ SicWriter(const StepPtrs<R>& p, const WinPtrs<R>& w, const NetScalars& ns, u32 a,
                                         int buf, int s_begin)
        : out(w.sic_win + (static_cast<u64>(buf) * ns.n_astro + a) * w.W), last(static_cast<R>(0.0)),
          ever(p.ever_active[a]), ever_in(ever), writing(false), any(false) {
        if (s_begin > 0)
            writing = (w.astro_active[static_cast<u64>(buf) * w.astro_words + (a >> 5)] >> (a & 31)) & 1u;
    }
    // Step st's factor; `mark`: the pre-run ends here (src/astrosim_fused.cu:1075).
    __device__ __forceinline__ void step(int st, R factor, bool mark) {
        last = factor;
        if (factor > static_cast<R>(0.0)) {
            ever = 1;
            any = true;
            if (!writing)
                for (int i = 0; i < st; ++i) out[i] = static_cast<R>(0.0);
            writing = true;
        }
        if (writing) out[st] = factor;
        if (mark) ever = 0;
    }
    __device__ __forceinline__ void finish(const StepPtrs<R>& p, u32 a) const {
        if (ever != ever_in) p.ever_active[a] = ever;
        p.sic_last[a] = last;
    }
};

// Astrocyte a through steps [s_begin, s_end) of the window; returns whether its SIC
// factor was positive at any of them.
template <typename R>
__device__ __forceinline__ bool astro_window(const RunConsts& rc, const NetScalars& ns, const StepPtrs<R>& p,
                                             const WinPtrs<R>& w, u32 a, i64 win_start, int s_begin, int s_end,
                                             int buf, i64 mark, bool window_done) {
    const u32 deposits = w.ain_cnt[static_cast<u64>(buf) * ns.n_astro + a];
    const int pull = w.mode[buf];
    AstroRegs<R> s =
        load_astro<R>(p.Ca[a], p.IP3[a], p.h[a], p.Ca_tot[a], p.IP3_0[a], p.tau_IP3[a], p.delta_IP3[a]);
    SicWriter<R> out(p, w, ns, a, buf, s_begin);
    AstroInput<R> x;
    astro_input<R>(ns, p, w, a, deposits, s_begin, s_end, buf, pull != 0, window_done, x);
    u64 pbase = step_base(ns.seed, kAstroPoissonKey, win_start + s_begin, a);
    u64 nbase = step_base(ns.seed, kAstroNoiseKey, win_start + s_begin, a);
    // recording phase (t + 1) % rec_every, advanced by a counter
    i64 rphase = p.ca_rec ? (win_start + s_begin + 1) % p.rec_every : 1;
    for (int st = s_begin; st < s_end; ++st) {
        const i64 t = win_start + st;
        const R factor = astro_advance_step<R>(rc, ns, s, ((x.mask >> st) & 1u) ? x.sum[st] : static_cast<R>(0.0), a,
                                               t, pbase, nbase);
        pbase += kStepAdvance;
        nbase += kStepAdvance;
        if (p.ca_rec) {
            record_ca<R>(p, a, t, rphase == 0, s.Ca);
            if (++rphase == p.rec_every) rphase = 0;
        }
        out.step(st, factor, t == mark);
    }
    p.Ca[a] = s.Ca;
    p.IP3[a] = s.IP3;
    p.h[a] = s.h;
    out.finish(p, a);
    return out.any;
}

// One block's tile through steps [s_begin, s_end) of the window that starts at step
// win_start (buffer parity buf), one cell per thread.  `shared`: sic_bytes of shared memory.
template <typename R>
__device__ __forceinline__ void window_cells(const RunConsts& rc, const NetScalars& ns, const StepPtrs<R>& p,
                                             const WinPtrs<R>& w, i64 win_start, int s_begin, int s_end, int buf,
                                             i64 mark, const Tile& tile, unsigned char* shared) {
    const bool window_done = s_end == w.W;
    const u32 cell = tile.base + threadIdx.x;
    const bool have = cell < tile.end;
    if (tile.kind == kAstroCells) {
        const bool active =
            have && astro_window<R>(rc, ns, p, w, cell, win_start, s_begin, s_end, buf, mark, window_done);
        // one word of the active mask per warp (tiles and blocks start at multiples of 32)
        const unsigned ballot = __ballot_sync(0xffffffffu, active);
        if ((threadIdx.x & 31) == 0 && have) {
            u32* word = w.astro_active + static_cast<u64>(buf) * w.astro_words + (cell >> 5);
            if (s_begin == 0) *word = ballot; else if (ballot) atomicOr(word, ballot);
        }
        return;
    }
    if (!__any_sync(0xffffffffu, have)) return;
    const SicRows<R> sic = sic_rows<R>(shared, w.W);
    const u32 j = have ? cell : tile.base;  // a lane without a cell still sums SIC factors for the others
    // one instantiation per population, so its constants are compile-time operands
    if (tile.kind == kExcCells)
        neuron_window<R, true>(rc, ns, rc.pe, p, w, j, have, win_start, s_begin, s_end, buf, window_done, sic);
    else
        neuron_window<R, false>(rc, ns, rc.pi, p, w, j, have, win_start, s_begin, s_end, buf, window_done, sic);
}

// After window `buf` completes: mark the astrocytes that were active in it in the a2n rows
// that hold them, and deliver its spikes into the inboxes of the next
// window (buffer buf ^ 1), or switch the next window to pull when it was busy.
// Blocks 0 .. n_blk-1 share the spike list and the active-astrocyte words.
// Targets outside [t_lo, t_hi) (neurons) and [a_lo, a_hi) (astrocytes) are skipped:
// a rank of a sharded network delivers only into the cells it owns.
template <typename R>
__device__ __forceinline__ void push_cells(const WinPtrs<R>& w, u32 n_exc, u32 n_inh, u64 n_neurons, u64 n_astro,
                                           int buf, u32 blk, u32 n_blk, u32 t_lo = 0, u32 t_hi = 0xFFFFFFFFu,
                                           u32 a_lo = 0, u32 a_hi = 0xFFFFFFFFu) {
    const int nxt = buf ^ 1;
    const u32 n = w.spk_count[buf];
    const bool busy = n > w.push_limit;
    if (blk == 0 && threadIdx.x == 0) {
        w.mode[nxt] = busy ? 1 : 0;
        w.spk_count[nxt] = 0;  // the next window appends its spikes there
    }
    const u32 lane = threadIdx.x & 31;
    const u64 warp = (static_cast<u64>(blk) * blockDim.x + threadIdx.x) >> 5;
    const u64 n_warps = (static_cast<u64>(n_blk) * blockDim.x) >> 5;
    // A warp takes one item at a time: first the active astrocytes, then each
    // spike's excitatory, n2a and inhibitory targets as three items.  The items of a
    // spike go to different warps, because each is a chain of four dependent accesses and
    // a small network has warps to spare (N = 500: one warp for all three took 7.8k
    // cycles).
    const u32* act = w.astro_active + static_cast<u64>(buf) * w.astro_words;
    u32* marks = w.sic_pos + static_cast<u64>(nxt) * n_neurons;
    const R* vals = w.spk_val + static_cast<u64>(buf) * w.W * n_neurons;
    // An item of active astrocytes is a word's 32, or fewer when there are warps to spare.
    u32 span = 32;
    while (span > 1 && n_astro / (span / 2) <= n_warps) span /= 2;
    const u32 spans = (static_cast<u32>(n_astro) + span - 1) / span;
    const u64 items = spans + (busy ? 0 : 3 * static_cast<u64>(n));
    for (u64 item = warp; item < items; item += n_warps) {
        if (item < spans) {
            // mark the active astrocytes in their targets' a2n rows for the next window: the
            // lanes read the rows' ends together, then the warp walks one row after the other
            // with three loads in flight (a row has 80 targets on average)
            const u32 a0 = static_cast<u32>(item) * span;
            u32 bits = (act[a0 >> 5] >> (a0 & 31)) & (span == 32 ? 0xFFFFFFFFu : (1u << span) - 1u);
            if (!bits) continue;
            const bool mine = (bits >> lane) & 1u;
            const u32 r0 = mine ? w.fs_rs[a0 + lane] : 0, r1 = mine ? w.fs_rs[a0 + lane + 1] : 0;
            auto mark = [&](u32 entry, bool have) {
                const u32 t = entry >> 5;
                if (have && t >= t_lo && t < t_hi) atomicOr(&marks[t], 1u << (entry & 31));
            };
            while (bits) {
                const int b = __ffs(bits) - 1;
                bits &= bits - 1;
                const u32 end = __shfl_sync(0xffffffffu, r1, b);
                for (u32 k = __shfl_sync(0xffffffffu, r0, b) + lane; k < end + lane; k += 96) {
                    const bool h0 = k < end, h1 = k + 32 < end, h2 = k + 64 < end;
                    const u32 e0 = h0 ? w.fs_dst[k] : 0, e1 = h1 ? w.fs_dst[k + 32] : 0, e2 = h2 ? w.fs_dst[k + 64] : 0;
                    mark(e0, h0);
                    mark(e1, h1);
                    mark(e2, h2);
                }
            }
            continue;
        }
        const u32 e = static_cast<u32>(item - spans), kind = e % 3;
        const u32 packed = w.spk_list[static_cast<u64>(buf) * w.cap + e / 3];
        const u32 j = packed >> 5, st = packed & 31u;
        const R v = vals[static_cast<u64>(st) * n_neurons + j];
        if (kind == 1) {
            if (j >= n_exc) continue;
            for (u32 k = w.fa_rs[j] + lane; k < w.fa_rs[j + 1]; k += 32) {
                const u32 a = w.fa_astro[k];
                if (a < a_lo || a >= a_hi) continue;
                const u64 sb = static_cast<u64>(nxt) * n_astro + a;
                const u32 slot = atomicAdd(&w.ain_cnt[sb], 1u);
                if (slot < kInboxSlots) w.ain_ent[sb * kInboxSlots + slot] = Deposit<R>{w.fa_pos[k], st, v};
            }
            continue;
        }
        // the inhibitory rows hold local inhibitory ids and read the spike ring by
        // global id (src/astrosim_fused.cu:458-463): neuron j feeds them when j < n_inh
        const bool inh = kind == 2;
        if (j >= (inh ? n_inh : n_exc)) continue;
        const u32* rs = inh ? w.fi_rs : w.fe_rs;
        const u32* dst = inh ? w.fi_dst : w.fe_dst;
        const u32 meta = inh ? st | (1u << 8) : st;
        for (u32 k = rs[j] + lane; k < rs[j + 1]; k += 32) {
            const u32 t = dst[k];
            if (t < t_lo || t >= t_hi) continue;
            const u64 sb = static_cast<u64>(nxt) * n_neurons + t;
            const u32 slot = atomicAdd(&w.nin_cnt[sb], 1u);
            if (slot < kInboxSlots) w.nin_ent[sb * kInboxSlots + slot] = Deposit<R>{j, meta, v};
        }
    }
}

// One block's tile of neurons: the background events of the window that starts at
// win_start.  `shared`: poisson_bytes of shared memory.
template <int CELLS>
__device__ __forceinline__ void draw_events(const NetScalars& ns, u64* events, i64 win_start, int W, const Tile& tile,
                                            u32* shared) {
    const u32 j = tile.base + threadIdx.x;
    if (j >= tile.end) return;
    const bool exc = tile.kind == kExcCells;
    poisson_window<CELLS>(ns.seed, win_start, W, j, CELLS == 2 && tile.end - j > blockDim.x,
                          exc ? ns.lambda_exc : ns.lambda_inh,
                          exc ? ns.lim53_exc : ns.lim53_inh, shared, threadIdx.x, blockDim.x, events + j);
}
// The tiles of the neurons [n_lo, n_hi) for it.
inline CellTiles event_tiles(u32 n_exc, u32 n_lo, u32 n_hi, int block, int cells) {
    return cell_tiles(n_exc, n_lo, n_hi, 0, 0, static_cast<u32>(block * cells));
}

}  // namespace astrosim
