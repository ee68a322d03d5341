// window_schedule.cuh -- the steps of a window at which something besides the cells' own
// dynamics happens.
//
// Device code, also compiled on the host by a CPU test (tests/window_schedule_check.cpp).
#pragma once

#include "model.cuh"

namespace astrosim {

// The steps of a window at which something besides the cells' own dynamics happens:
// bit s of `refresh` when the SIC current is refreshed ((t - d_a2n) >= 0 and
// (t - d_a2n) % sic_interval == 0), bit s of `noise` when a new noise index starts
// (t / steps_per_noise; src/astrosim_fused.cu:1046-1050), and the index at s_begin.
struct WindowSchedule {
    u32 refresh, noise;
    u64 noise_idx;
};

__device__ __forceinline__ WindowSchedule window_schedule(int d_a2n, int sic_interval, int steps_per_noise,
                                                          i64 win_start, int s_begin, int s_end) {
    WindowSchedule w{0, 0, 0};
    const i64 t0 = win_start + s_begin;
    const int si = sic_interval, spn = steps_per_noise, n = s_end - s_begin;
    // steps of the first refresh and of the first new noise index, counted from t0
    int first = 0, fresh;
    if (t0 < (i64(1) << 31)) {  // 32-bit division: a few instructions instead of a call
        const u32 t = static_cast<u32>(t0);
        w.noise_idx = t / static_cast<u32>(spn);
        fresh = spn - static_cast<int>(t % static_cast<u32>(spn));
        if (t0 < d_a2n) first = d_a2n - static_cast<int>(t0);
        else if (si > 1) first = (si - static_cast<int>((t - static_cast<u32>(d_a2n)) % static_cast<u32>(si))) % si;
    } else {
        w.noise_idx = static_cast<u64>(t0 / spn);
        fresh = spn - static_cast<int>(t0 % spn);
        if (si > 1) first = (si - static_cast<int>((t0 - d_a2n) % si)) % si;
    }
    // a step past the longest window ends the loops below, which an interval near the
    // largest int would overflow (added up unsigned: 1 % of the FP64 window at N = 1e6)
    constexpr int kPast = 16;
    if (si == 1) {
        if (first < n) w.refresh = (1u << n) - (1u << first);
    } else {
        for (int i = first; i < n; i += si < kPast ? si : kPast) w.refresh |= 1u << i;
    }
    for (int i = fresh; i < n; i += spn < kPast ? spn : kPast) w.noise |= 1u << i;
    w.refresh <<= s_begin;
    w.noise <<= s_begin;
    return w;
}

}  // namespace astrosim
