// Host check of a window's schedule (astrosimgpu_cuda_b200/csrc/window_schedule.cuh), compiled
// with g++ by test_window_schedule.py: the SIC refreshes, new noise indexes and first noise
// index of every part of a window are those of the loop over its steps
// (src/astrosim_fused.cu:1043-1050), for intervals and delays from 1 to the largest int and
// steps from 0 to past 2^31.
// Test infrastructure.
#include <climits>
#include <cstdint>
#include <cstdio>
#include <random>

#include "../astrosimgpu_cuda_b200/csrc/window_schedule.cuh"

using namespace astrosim;

int main() {
    std::mt19937_64 rng(3);
    const int edge[] = {1, 2, 3, 7, 10, 16, 17, 100, 1 << 20, INT_MAX - 17, INT_MAX - 16, INT_MAX - 2, INT_MAX - 1, INT_MAX};
    auto pick = [&] { return edge[rng() % (sizeof(edge) / sizeof(edge[0]))]; };
    long checked = 0, bad = 0, refreshes = 0, noises = 0;
    for (long k = 0; k < 400000; ++k) {
        const int W = 1 + static_cast<int>(rng() % 16);
        const int d = pick(), si = pick(), spn = pick();
        const i64 centres[] = {0, d, si, static_cast<i64>(d) + si, spn, i64(1) << 31, (i64(1) << 40) + 5};
        i64 start = centres[rng() % 7] + static_cast<i64>(rng() % 64) - 32;
        start = start < 0 ? 0 : start / W * W;
        const int s0 = static_cast<int>(rng() % W), s1 = s0 + 1 + static_cast<int>(rng() % (W - s0));
        u32 refresh = 0, noise = 0;
        for (int s = s0; s < s1; ++s) {
            const i64 t = start + s;
            if (t - d >= 0 && (t - d) % si == 0) refresh |= 1u << s;
            if (s != s0 && t % spn == 0) noise |= 1u << s;
        }
        const WindowSchedule w = window_schedule(d, si, spn, start, s0, s1);
        ++checked;
        refreshes += refresh != 0;
        noises += noise != 0;
        bad += w.refresh != refresh || w.noise != noise || w.noise_idx != static_cast<u64>((start + s0) / spn);
    }
    std::printf("checked %ld bad %ld refreshes %ld noises %ld\n", checked, bad, refreshes, noises);
    return bad != 0;
}
