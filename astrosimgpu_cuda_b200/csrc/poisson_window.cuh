// poisson_window.cuh -- the background events of a whole window, drawn before its steps.
//
// A neuron's Poisson count (src/astrosim_fused.cu:154-175, Knuth's product) needs one
// draw when it is zero and count + 1 otherwise.  Drawn step by step, every warp ran as
// many dependent draws per step as its unluckiest lane needed (about 3.5 at the default
// rate, where a lane needs 1.27 on average), and they sat in the step's serial chain:
// 30 % of the FP32 window at N = 1e7 and of the whole window at N = 500.  The draws
// depend on nothing but (seed, step, cell).  So the launch that delivers one window's
// spikes also draws the next window's counts, with its own (small) register budget and
// on the multiprocessors that the delivery leaves idle: all first draws of a window are
// made in one divergence-free pass of independent hashes; each lane lists its steps that
// go on, and every further pass makes one more draw for each listed step and keeps those
// that go on again.  A warp then runs as many second draws as its unluckiest lane lists
// over the whole window, and the count of a step is the number of the pass it ended in.
//
// The counts equal rng_poisson_at's.  The product is kept as a 32-bit fraction whose low
// 5 bits carry the step (kRowMask), formed from the upper 32 bits of each draw.  Every
// pass loses less than 2^5 + 2 units of 2^-32 from it (truncated bits of the product, of
// the draw and of their product, all factors being below 1), so after kExactCount passes
// it is at most 510 units low; a product within kPoissonSlack units of the limit
// e^-lambda is not decided here but leaves its step to the exact draw (about one step in
// 2e6).
#pragma once

#include "model.cuh"

namespace astrosim {

// A window's counts of one neuron: four bits per step, kExactCount where the window
// kernel draws the step itself (rng_poisson_at).
constexpr u32 kExactCount = 15;
constexpr double kPoissonWindowLambda = 4.0;  // larger rates leave every step to the exact draw
constexpr u32 kPoissonSlack = 1024;           // units of 2^-32

// A thread draws CELLS (1 or 2) cells, kRowSteps rows apart.
constexpr int kRowSteps = 16;
constexpr u32 kRowMask = 2 * kRowSteps - 1;

// Shared memory of one thread: its column of the list ([rows][threads]) and one count
// byte per row.  The bytes of a thread are an odd number of words, so the same row of a
// warp's lanes lies in 32 different banks.
constexpr u32 count_bytes(int cells) { return static_cast<u32>(cells * kRowSteps + 4); }
inline size_t poisson_bytes(int cells, int W, int block) {
    return static_cast<size_t>(block) * (static_cast<size_t>(W * cells) * sizeof(u32) + count_bytes(cells));
}

// Sixteen count bytes of one cell as four-bit counts.
__device__ __forceinline__ u64 pack_counts(const u32* words) {
    u32 half[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const u32 a = words[2 * i], b = words[2 * i + 1];
        half[i] = __byte_perm(a | a >> 4, b | b >> 4, 0x6420);
    }
    return static_cast<u64>(half[1]) << 32 | half[0];
}

// Draws the counts of cells j and (when have1) j + threads over the window of W steps that
// starts at step win_start, into counts[0] and counts[threads].  `shared`: poisson_bytes
// for `threads` threads, of which the caller is number `thread`.
template <int CELLS>
__device__ __forceinline__ void poisson_window(u64 seed, i64 win_start, int W, u32 j, bool have1, double lambda,
                                               u64 lim53, u32* shared, u32 thread, u32 threads, u64* counts) {
    const u32 gap = have1 ? threads : 0;
    if (!(lambda > 0.0) || !(lambda <= kPoissonWindowLambda)) {
        const u64 all = lambda > 0.0 ? ~u64(0) : u64(0);
        counts[0] = all;
        if (have1) counts[gap] = all;
        return;
    }
    u32* const list = shared + thread;
    u8* const bytes = reinterpret_cast<u8*>(shared + static_cast<u32>(W) * CELLS * threads) +
                      thread * count_bytes(CELLS);
    u32* const words = reinterpret_cast<u32*>(bytes);
#pragma unroll
    for (int i = 0; i < CELLS * kRowSteps / 4; ++i) words[i] = 0;
    // u0 > limit exactly when its 53 bits exceed lim53; an equal upper part is listed and
    // then falls within the slack
    const u32 lim_hi = poisson_limit_hi(lim53);
    const u32 sure_more = lim_hi < 0xFFFFFFFFu - kPoissonSlack ? lim_hi + kPoissonSlack : 0xFFFFFFFFu;
    const u32 sure_done = lim_hi > kPoissonSlack ? lim_hi - kPoissonSlack : 0;
    const u64 base = rng_base(seed ^ kNeuronPoissonKey, static_cast<u64>(win_start) * kCellStride + j);
    u32 undecided = 0;
    u32* end = list;
    {
        u64 z = base;
        const u64 z_gap = gap * kStreamMul;
#pragma unroll 5
        for (int st = 0; st < W; ++st) {
#pragma unroll
            for (int i = 0; i < CELLS; ++i) {
                const u32 hi = rng_mix_hi(i == 0 ? z : z + z_gap);
                if (hi >= lim_hi) {
                    *end = (hi & ~kRowMask) | static_cast<u32>(st + i * kRowSteps);
                    end += threads;
                    if (hi <= sure_more) undecided |= 1u << (st + i * kRowSteps);
                }
            }
            z += kCellStride * kStreamMul;
        }
    }
    u64 zb = base;
    for (u32 pass = 1; end != list; ++pass) {
        zb += kCounterMul;
        const u32* const last = end;
        end = list;
        for (const u32* k = list; k != last; k += threads) {
            const u32 entry = *k;
            const u32 row = entry & kRowMask;
            const u32 ahead = (row & (kRowSteps - 1)) * static_cast<u32>(kCellStride) + (CELLS == 2 && row >= kRowSteps ? gap : 0u);
            const u32 product = __umulhi(entry, rng_mix_hi(zb + ahead * kStreamMul));
            if (product > sure_more) {
                *end = (product & ~kRowMask) | row;
                end += threads;
            } else {
                bytes[row] = static_cast<u8>(pass);
                if (product >= sure_done) undecided |= 1u << row;
            }
        }
        if (pass == kExactCount - 1) {  // whatever is left has more events than a count holds
            for (const u32* k = list; k != end; k += threads) undecided |= 1u << (*k & kRowMask);
            break;
        }
    }
    for (; undecided; undecided &= undecided - 1) bytes[__ffs(undecided) - 1] = static_cast<u8>(kExactCount);
    counts[0] = pack_counts(words);
    if (CELLS == 2 && have1) counts[gap] = pack_counts(words + kRowSteps / 4);
}

// The steps of a window's counts that are left to the exact draw.
__device__ __forceinline__ u32 exact_steps(u64 counts) {
    u64 m = counts & (counts >> 1);
    m &= m >> 2;
    m &= 0x1111111111111111ull;
    u32 steps = 0;
    for (; m; m &= m - 1) steps |= 1u << ((__ffsll(static_cast<long long>(m)) - 1) >> 2);
    return steps;
}

}  // namespace astrosim
