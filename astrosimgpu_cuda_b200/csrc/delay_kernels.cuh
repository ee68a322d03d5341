// delay_kernels.cuh -- stepping with delays that the windowed engine does not take
// (unequal ones, one step, or more than 16 steps).
//
// A cell's step reads only spikes and SIC factors that are at least min(d) steps old, so
// one launch advances every cell by a window of up to min(d) steps (at most 16) without any
// cell waiting for another; the state stays in registers.  What bounds it is latency: the
// chain of a cell's steps (about 3 us each in FP64), and before it the walk of its rows.  A
// launch per step, with a thread walking each row, took 20.5 us a step at N = 20011 and 92
// at N = 2e5 (FP64); a launch per step with rows walked by warps 14.4 and 65; windows of six
// steps take 5.3 and 23 (6.8 at N = 20011 with every astrocyte active).
//
// A window's spikes are one word per neuron (bit s: a spike at its step s), kept for
// as many windows as the longest delay reaches back, so one load of a source tells its
// spikes at all delayed steps of the window, and one bit per neuron (any spike in the
// window) spares most of those loads (N = 2e5: 41 us a step without it).  The values that spikes carry and the SIC
// factors are in rings by step; the words say which entries mean something.
#pragma once

#include "window_kernels.cuh"

namespace astrosim {

// Where the delayed steps of a window lie, for one delay d = q W + shift: step s of window
// k sees step s - shift of window k - q, or for s < shift step s - shift + W of window
// k - q - 1.
struct Delayed {
    u32 row, row_before;  // their rows in the rings of words
    u32 shift;
    u32 slot, bit_slot;   // ring slots that step 0 of the window sees
};

// One launch: steps [s_begin, s_end) of the window that starts at step `start`.
struct DelayWindow {
    i64 start, mark;  // mark: the step at which the pre-run ends
    int W, s_begin, s_end;
    u32 row, row_next;     // the window's and the next one's rows of words
    u32 slot, slots;       // step 0's ring slot, slots of the ring
    u32 bit_slot, bit_slots;  // the same of the ring of bits by step
    Delayed e, i, a2n;
};
// A launch of one step (a caller that steps one at a time, or a shortest delay of one step)
// reads the bits of the step it sees, where a set one is that step's spike; the window's bits
// would send it to the words of every source that spiked at any of the window's steps.  A
// call of one step at N = 200003 FP32 with delays of 20 steps: 340 us with a window's draws
// and bits, 75 so; 90 with a thread per row and a launch per step.  Such launches have their own
// instantiation (`Short`), since the branch alone cost the longer ones 2 to 5 % in FP64.
__host__ __device__ __forceinline__ bool one_step(const DelayWindow& w) { return w.s_end - w.s_begin == 1; }

// Shared memory of a warp: per step and lane three sums (excitatory or IP3, inhibitory, SIC),
// and before them, in the same place, its background draws.  A launch of at most half a
// window takes its own steps' share, which leaves the rest to the cache of the walks'
// look-ups (N = 200003 FP32, delays of 20 steps, 3 steps: 141 us instead of 312).  A longer
// one takes a whole window's: with the share of 11 to 14 steps in FP64 one more block fits
// on a multiprocessor and all of them lose their look-ups' cache (448 us instead of 242).
__host__ __device__ __forceinline__ int shared_steps(const DelayWindow& w) {
    const int steps = w.s_end - w.s_begin;
    return 2 * steps <= w.W ? steps : w.W;
}
template <typename R>
__host__ __device__ __forceinline__ u32 delay_warp_bytes(int steps) {
    const u32 sums = 32 * 3 * static_cast<u32>(steps) * static_cast<u32>(sizeof(R));
    const u32 draws = 32 * (static_cast<u32>(steps) * static_cast<u32>(sizeof(u32)) + count_bytes(1));
    return sums > draws ? sums : draws;
}
template <typename R>
inline size_t delay_shared_bytes(int steps, int block) {
    return static_cast<size_t>(block / 32) * delay_warp_bytes<R>(steps);
}
// A lane's sums of one kind, by step of the window.
template <typename R>
struct StepSums {
    R* warp_sums;
    int at;
    __device__ __forceinline__ StepSums(R* sums, const DelayWindow& w, int kind)
        : warp_sums(sums), at(32 * (kind * shared_steps(w) - w.s_begin) + static_cast<int>(threadIdx.x & 31)) {}
    __device__ __forceinline__ R& operator[](int step) const { return warp_sums[at + 32 * step]; }
};

__device__ __forceinline__ u32 delayed_steps(const u32* __restrict__ words, u64 n, const Delayed& d, int W, u32 src) {
    u32 m = words[d.row * n + src] << d.shift;
    if (d.shift) m |= words[d.row_before * n + src] >> (W - static_cast<int>(d.shift));
    return m;
}
__device__ __forceinline__ u32 delayed_slot(const DelayWindow& w, const Delayed& d, int s) {
    const u32 slot = d.slot + static_cast<u32>(s);
    return slot >= w.slots ? slot - w.slots : slot;
}

__device__ __forceinline__ u32 delayed_bit_slot(const DelayWindow& w, const Delayed& d) {  // of a launch of one step
    const u32 slot = d.bit_slot + static_cast<u32>(w.s_begin);
    return slot >= w.bit_slots ? slot - w.bit_slots : slot;
}

// Sums, for every step in `steps`, the delayed spike values of lane i's CSR row in row
// order, for the warp's 32 consecutive rows (those from `end_row` on are empty; every lane
// calls).  Skipped terms are +0.0 in the reference's dense ring, so the sums are
// bit-identical.  The rows lie one behind the other, so the warp reads their entries as
// one coalesced run, kGatherRun of them in flight per lane since latency bounds the walk;
// the values of the few that spiked go to their rows' lanes one by one, in order.
constexpr int kGatherRun = 8;
template <typename R, bool Short>
__device__ __forceinline__ void gather_spikes(const DelayWindow& w, const Delayed& d, const StepPtrs<R>& p, u64 n_src, u64 words,
                                              const u32* __restrict__ rs, const u32* __restrict__ src, u32 row,
                                              u32 end_row, u32 steps, const StepSums<R>& sums) {
    constexpr unsigned kAll = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31;
    for (int s = w.s_begin; s < w.s_end; ++s) sums[s] = static_cast<R>(0.0);
    const bool single = Short && one_step(w);
    const u32* bits = single && p.step_bits ? p.step_bits + delayed_bit_slot(w, d) * words : p.spk_bits + d.row * words;
    const u32* bits_before = p.spk_bits + d.row_before * words;
    const bool both_rows = !single && d.shift != 0;
    const u32 lo = rs[min(row, end_row)];
    const u32 end = __shfl_sync(kAll, rs[min(row + 1, end_row)], 31);
    for (u64 k0 = __shfl_sync(kAll, lo, 0); k0 < end; k0 += 32 * kGatherRun) {
        u32 id[kGatherRun], hit[kGatherRun];
#pragma unroll
        for (int i = 0; i < kGatherRun; ++i) {
            const u64 k = k0 + 32 * i + lane;
            id[i] = k < end ? src[k] : ~0u;
        }
        u32 any = 0;
#pragma unroll
        for (int i = 0; i < kGatherRun; ++i) {
            hit[i] = 0;
            if (id[i] != ~0u) {
                hit[i] = bits[id[i] >> 5];
                if (both_rows) hit[i] |= bits_before[id[i] >> 5];
                hit[i] &= 1u << (id[i] & 31);
            }
            any |= hit[i];
        }
        if (!__any_sync(kAll, any != 0)) continue;
#pragma unroll
        for (int i = 0; i < kGatherRun; ++i)
            if (hit[i]) hit[i] = single ? steps : delayed_steps(p.spk_word, n_src, d, w.W, id[i]) & steps;
#pragma unroll
        for (int i = 0; i < kGatherRun; ++i) {
            auto value = [&](u32 m, u32 source) {  // of the first step in m
                return p.val[delayed_slot(w, d, __ffs(static_cast<int>(m)) - 1) * n_src + source];
            };
            const R v = hit[i] ? value(hit[i], id[i]) : static_cast<R>(0.0);
            for (unsigned left = __ballot_sync(kAll, hit[i] != 0); left; left &= left - 1) {
                const int from = __ffs(static_cast<int>(left)) - 1;
                const R first = __shfl_sync(kAll, v, from);
                u32 m = __shfl_sync(kAll, hit[i], from);
                const u32 source = __shfl_sync(kAll, id[i], from);
                // the entry's row: the last one that starts at it or before
                const unsigned owner = __popc(__ballot_sync(kAll, lo <= k0 + 32 * i + from)) - 1;
                if (lane != owner) continue;
                sums[__ffs(static_cast<int>(m)) - 1] += first;
                while (m &= m - 1) sums[__ffs(static_cast<int>(m)) - 1] += value(m, source);
            }
        }
    }
}

// Sums the delayed SIC factors of neuron j's a2n row for the steps in `steps`, in row
// order (a factor of 0 adds nothing and is not read).  A thread walks its own row, four
// steps and four entries at a time, so that sixteen loads are in flight where every
// astrocyte is active (one value after the other: 10 us more per window at N = 20011).  A
// first walk, over the words alone, is all there is while none is.  A launch of one step
// walks once (a shortest delay of one step, every astrocyte active, N = 200003 FP32: 84 us a
// step with both walks, 68 so).
template <typename R, bool Short>
__device__ __forceinline__ void gather_sic(const DelayWindow& w, const StepPtrs<R>& p, u64 n_astro, u32 j, u32 steps,
                                           const StepSums<R>& sums) {
    constexpr int kSteps = 4;
    if (!steps) return;  // no refresh: the sums are not read
    const u32 k0 = p.sic_rs[j], k1 = p.sic_rs[j + 1];
    if (Short && one_step(w)) {
        const int s = w.s_begin, from = s - static_cast<int>(w.a2n.shift);
        const u32* words = p.act_word + (from >= 0 ? w.a2n.row : w.a2n.row_before) * n_astro;
        const int bit = from >= 0 ? from : from + w.W;
        const u32 slot = delayed_slot(w, w.a2n, s);
        R sum = static_cast<R>(0.0);
#pragma unroll 8
        for (u32 k = k0; k < k1; ++k) {
            const u32 a = p.sic_src[k];
            if ((words[a] >> bit) & 1u) sum += p.sic_ring[static_cast<u64>(a) * w.slots + slot];
        }
        sums[s] = sum;
        return;
    }
    u32 any = 0;
#pragma unroll 8
    for (u32 k = k0; k < k1; ++k) any |= delayed_steps(p.act_word, n_astro, w.a2n, w.W, p.sic_src[k]);
    steps &= any;
    for (int s0 = w.s_begin; s0 < w.s_end; s0 += kSteps) {
        const u32 now = (steps >> s0) & ((1u << kSteps) - 1u);
        R sum[kSteps] = {};
        if (now)
#pragma unroll 4
            for (u32 k = k0; k < k1; ++k) {
                const u32 a = p.sic_src[k];
                const u32 m = (delayed_steps(p.act_word, n_astro, w.a2n, w.W, a) >> s0) & now;
                const R* factors = p.sic_ring + static_cast<u64>(a) * w.slots;
#pragma unroll
                for (int i = 0; i < kSteps; ++i)
                    if ((m >> i) & 1u) sum[i] += factors[delayed_slot(w, w.a2n, s0 + i)];
            }
#pragma unroll
        for (int i = 0; i < kSteps; ++i)
            if (s0 + i < w.s_end) sums[s0 + i] = sum[i];
    }
}

// One astrocyte through the launch's steps (src/astrosim_fused.cu:374-427); called by whole warps.
template <typename R, bool Short>
__device__ __forceinline__ void astro_delay_window(const RunConsts& rc, const NetScalars& ns, const StepPtrs<R>& p,
                                                   const DelayWindow& w, u32 a, u32 end, u32 steps, R* warp_sums) {
    const StepSums<R> sums(warp_sums, w, 0);
    // the e2a delay is d_e (src/astrosim_fused.cu:384)
    gather_spikes<R, Short>(w, w.e, p, ns.n_neurons, ns.words, p.e2a_rs, p.e2a_src, a, end, steps, sums);
    __syncwarp();
    if (a >= end) return;
    AstroRegs<R> s = load_astro<R>(p.Ca[a], p.IP3[a], p.h[a], p.Ca_tot[a], p.IP3_0[a], p.tau_IP3[a], p.delta_IP3[a]);
    const unsigned char ever_in = p.ever_active[a];
    unsigned char ever = ever_in;
    u64 pbase = step_base(ns.seed, kAstroPoissonKey, w.start + w.s_begin, a);
    u64 nbase = step_base(ns.seed, kAstroNoiseKey, w.start + w.s_begin, a);
    i64 rphase = p.ca_rec ? (w.start + w.s_begin + 1) % p.rec_every : 1;
    u32 active = 0;
    R factor = static_cast<R>(0.0);
    for (int st = w.s_begin; st < w.s_end; ++st) {
        const i64 t = w.start + st;
        factor = astro_advance_step<R>(rc, ns, s, sums[st], a, t, pbase, nbase);
        pbase += kStepAdvance;
        nbase += kStepAdvance;
        if (p.ca_rec) {
            record_ca<R>(p, a, t, rphase == 0, s.Ca);
            if (++rphase == p.rec_every) rphase = 0;
        }
        if (factor > static_cast<R>(0.0)) ever = 1;
        if (t == w.mark) ever = 0;
        if (factor != static_cast<R>(0.0)) {
            const u32 slot = w.slot + static_cast<u32>(st);
            p.sic_ring[static_cast<u64>(a) * w.slots + (slot >= w.slots ? slot - w.slots : slot)] = factor;
            active |= 1u << st;
        }
    }
    p.Ca[a] = s.Ca;
    p.IP3[a] = s.IP3;
    p.h[a] = s.h;
    if (ever != ever_in) p.ever_active[a] = ever;
    p.sic_last[a] = factor;
    u32* word = p.act_word + static_cast<u64>(w.row) * ns.n_astro + a;
    if (w.s_begin == 0) *word = active;
    else if (active) *word |= active;  // mostly nothing to add, and no word to wait for
}

// One neuron through the launch's steps (src/astrosim_fused.cu:433-587); called by whole warps.
template <typename R, bool Short, bool EXC>
__device__ __forceinline__ void neuron_delay_window(const RunConsts& rc, const NetScalars& ns, const NeuronK& pk,
                                                    const StepPtrs<R>& p, const DelayWindow& w, u32 j, u32 end,
                                                    u32 steps, R* sums) {
    const unsigned lane = threadIdx.x & 31;
    const u64 nN = ns.n_neurons;
    const StepSums<R> ex(sums, w, 0), in(sums, w, 1), sic(sums, w, 2);
    const double lambda = EXC ? ns.lambda_exc : ns.lambda_inh;
    const u64 lim53 = EXC ? ns.lim53_exc : ns.lim53_inh;
    u64 counts;
    // four bits per step of the launch, the first step's lowest
    poisson_window<1>(ns.seed, w.start + w.s_begin, w.s_end - w.s_begin, j, false, lambda, lim53,
                      reinterpret_cast<u32*>(sums), lane, 32, &counts);
    __syncwarp();
    gather_spikes<R, Short>(w, w.e, p, nN, ns.words, p.exc_rs, p.exc_src, j, end, steps, ex);
    // inh sources are local inhibitory indices that index the ring by global id (458-463)
    gather_spikes<R, Short>(w, w.i, p, nN, ns.words, p.inh_rs, p.inh_src, j, end, steps, in);
    __syncwarp();
    if (j >= end) return;
    WindowSchedule sched = window_schedule(rc, w.start, w.s_begin, w.s_end);
    gather_sic<R, Short>(w, p, ns.n_astro, j, sched.refresh, sic);
    NeuronCore<R> n(p, j);
    R I_sic = p.I_sic[j];
    const double nstd = EXC ? rc.noise_exc : rc.noise_inh;
    const bool has_noise = nstd > 0.0 && rc.independent_noise;
    R noise = static_cast<R>(0.0);
    if (has_noise) noise = static_cast<R>(neuron_noise<R>(ns, nstd, sched.noise_idx, j));
    const R w_a2n = as_r<R>(ns.w_a2n, ns.f_w_a2n), neg_w_i = as_r<R>(-rc.w_i, rc.f_neg_w_i);
    u32 spikes = 0;
    for (int st = w.s_begin; st < w.s_end; ++st) {
        int events = static_cast<int>(static_cast<u32>(counts) & kExactCount);
        counts >>= 4;
        if (events == static_cast<int>(kExactCount))
            events = poisson_exact(step_base(ns.seed, kNeuronPoissonKey, w.start + st, j), lambda,
                                   EXC ? ns.limit_exc : ns.limit_inh, lim53);
        if ((sched.refresh >> st) & 1u) I_sic = w_a2n * sic[st];
        if (has_noise && ((sched.noise >> st) & 1u))
            noise = static_cast<R>(neuron_noise<R>(ns, nstd, ++sched.noise_idx, j));
        n.external(pk, has_noise ? I_sic + noise : I_sic);
        if (!n.step(rc, pk, exc_input_of<R>(rc, EXC, ex[st], events), neg_w_i * in[st])) continue;
        const i64 t = w.start + st;
        const u32 slot = w.slot + static_cast<u32>(st);
        p.val[static_cast<u64>(slot >= w.slots ? slot - w.slots : slot) * nN + j] =
            stp_on_spike<R>(rc, p.stp_x[j], p.stp_u[j], p.stp_t[j], t);
        atomicAdd(&p.counts[t], 1u);
        if (t < p.raster_steps) atomicOr(&p.raster[static_cast<u64>(t) * ns.words + (j >> 5)], 1u << (j & 31));
        if (p.step_bits) {
            const u32 row = w.bit_slot + static_cast<u32>(st);
            atomicOr(&p.step_bits[static_cast<u64>(row >= w.bit_slots ? row - w.bit_slots : row) * ns.words + (j >> 5)],
                     1u << (j & 31));
        }
        spikes |= 1u << st;
    }
    n.store(p, j);
    p.I_sic[j] = I_sic;
    p.refr[j] = n.refr();
    u32* word = p.spk_word + static_cast<u64>(w.row) * nN + j;
    if (w.s_begin == 0) *word = spikes;
    else if (spikes) *word |= spikes;
    if (spikes) atomicOr(&p.spk_bits[static_cast<u64>(w.row) * ns.words + (j >> 5)], 1u << (j & 31));
}

// Threads of a block: FP64 needs more registers than 1024 threads leave it (88 with 736).  A
// larger block size of the configuration runs as blocks of this one, to the same results.
template <typename R>
constexpr int kDelayThreads = sizeof(R) == 4 ? 1024 : 736;

template <typename R, bool Short>
__global__ void __launch_bounds__(kDelayThreads<R>)
    delay_kernel(RunConsts rc, StepPtrs<R> p, DelayWindow w, CellTiles tiles) {
    extern __shared__ __align__(16) unsigned char shared[];
    const NetScalars ns = net_scalars(rc);
    const Tile tile = tile_of(tiles, blockIdx.x);
    const u32 cell = tile.base + threadIdx.x, end = tile.end;
    R* sums = reinterpret_cast<R*>(shared + (threadIdx.x >> 5) * delay_warp_bytes<R>(shared_steps(w)));
    if (w.s_begin == 0) {  // the next window's bits start clear; no one reads or sets them yet
        const u64 i = static_cast<u64>(blockIdx.x) * blockDim.x + threadIdx.x;
        if (i < ns.words) p.spk_bits[static_cast<u64>(w.row_next) * ns.words + i] = 0;
        // the next window's rows of the bits by step: at most 16 words for 32 neurons
        if (p.step_bits && i < static_cast<u64>(w.W) * ns.words) {
            const u32 step = static_cast<u32>(i) / ns.words;
            u32 slot = w.bit_slot + static_cast<u32>(w.W) + step;
            if (slot >= w.bit_slots) slot -= w.bit_slots;
            p.step_bits[static_cast<u64>(slot) * ns.words + (static_cast<u32>(i) - step * ns.words)] = 0;
        }
    }
    const u32 steps = (1u << w.s_end) - (1u << w.s_begin);
    if (tile.kind == kAstroCells) astro_delay_window<R, Short>(rc, ns, p, w, cell, end, steps, sums);
    else if (tile.kind == kExcCells) neuron_delay_window<R, Short, true>(rc, ns, rc.pe, p, w, cell, end, steps, sums);
    else neuron_delay_window<R, Short, false>(rc, ns, rc.pi, p, w, cell, end, steps, sums);
}

}  // namespace astrosim
