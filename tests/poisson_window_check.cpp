// Host check of the window-wide background draw (astrosimgpu_cuda_b200/csrc/poisson_window.cuh),
// compiled with g++ by test_poisson_window.py: every count equals the neuron's own draw
// of that step (rng_poisson_at; src/astrosim_fused.cu:154-175), or leaves the step to it.
// One and two cells per thread, with and without the second cell, windows of 1 to 16
// steps, and rates from none to past the limit of the window-wide form.
// Test infrastructure.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

inline std::uint32_t __umulhi(std::uint32_t a, std::uint32_t b) {
    return static_cast<std::uint32_t>((static_cast<std::uint64_t>(a) * b) >> 32);
}
inline std::uint32_t __byte_perm(std::uint32_t a, std::uint32_t b, std::uint32_t sel) {
    const std::uint64_t both = static_cast<std::uint64_t>(b) << 32 | a;
    std::uint32_t r = 0;
    for (int i = 0; i < 4; ++i)
        r |= static_cast<std::uint32_t>((both >> (8 * ((sel >> (4 * i)) & 7u))) & 0xFFu) << (8 * i);
    return r;
}
inline int __ffs(int x) { return __builtin_ffs(x); }
inline int __ffsll(long long x) { return __builtin_ffsll(x); }

#include "../astrosimgpu_cuda_b200/csrc/poisson_window.cuh"

using namespace astrosim;

struct Tally {
    long checked = 0, wrong = 0, exact = 0, events = 0, past_nibble = 0;
};

template <int CELLS>
void check(u64 seed, i64 win_start, int W, u32 first, u32 threads, u32 have1_below, double lambda, Tally& t) {
    const double limit = std::exp(-lambda);
    const u64 lim53 = static_cast<u64>(std::floor(limit * 9007199254740992.0));
    std::vector<u32> shared(poisson_bytes(CELLS, W, static_cast<int>(threads)) / sizeof(u32) + 1, 0xDEADBEEFu);
    const u64 kUnset = 0x0123456789ABCDEFull;
    std::vector<u64> counts(2 * threads, kUnset);
    for (u32 i = 0; i < threads; ++i) {
        const bool have1 = CELLS == 2 && i < have1_below;
        poisson_window<CELLS>(seed, win_start, W, first + i, have1, lambda, lim53, shared.data(), i, threads,
                              counts.data() + i);
        for (int c = 0; c < 2; ++c) {
            const u64 got = counts[i + c * threads];
            if (c == 1 && !have1) {
                t.wrong += got != kUnset;
                continue;
            }
            u32 left_to_exact = 0;
            for (int s = 0; s < W; ++s) {
                const u64 base = rng_base(seed ^ kNeuronPoissonKey,
                                          static_cast<u64>(win_start + s) * kCellStride + first + i + c * threads);
                const int want = rng_poisson_at(base, lambda, limit, lim53);
                const u32 have = static_cast<u32>(got >> (4 * s)) & kExactCount;
                ++t.checked;
                t.events += want > 0;
                t.past_nibble += want >= static_cast<int>(kExactCount);
                if (have == kExactCount) {
                    ++t.exact;
                    left_to_exact |= 1u << s;
                } else if (static_cast<int>(have) != want) {
                    ++t.wrong;
                }
            }
            if ((exact_steps(got) & ((1u << W) - 1u)) != left_to_exact) ++t.wrong;
        }
    }
    if (shared.back() != 0xDEADBEEFu) ++t.wrong;  // past its shared memory
}

int main(int argc, char** argv) {
    if (argc < 3) return 2;
    const double lambda = std::strtod(argv[1], nullptr);
    const int rounds = std::atoi(argv[2]);
    std::mt19937_64 rng(5);
    Tally t;
    for (int k = 0; k < rounds; ++k)
        for (int W = 1; W <= 16; ++W) {
            const u64 seed = rng();
            const i64 start = static_cast<i64>(rng() % (k % 3 ? 100000 : (1ull << 40)));
            const u32 first = static_cast<u32>(rng() % (k % 2 ? 50 : 100000000));
            check<1>(seed, start, W, first, 32, 0, lambda, t);
            check<2>(seed, start, W, first, 96, static_cast<u32>(rng() % 97), lambda, t);
            check<2>(seed, start, W, first, 256, 256, lambda, t);
        }
    std::printf("checked %ld wrong %ld exact %ld events %ld past %ld\n", t.checked, t.wrong, t.exact, t.events,
                t.past_nibble);
    return t.wrong != 0;
}
