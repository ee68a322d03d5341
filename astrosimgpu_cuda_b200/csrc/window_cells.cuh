// window_cells.cuh -- one block of a window kernel, shared by the single-network
// (window.cu), batched (ensemble.cu) and sharded (shard.cu) launches.
#pragma once

#include "window_kernels.cuh"
#include "window_pair.cuh"

namespace astrosim {

// One block's tile through steps [s_begin, s_end) of the window that starts at step
// win_start (buffer parity buf).  A thread advances kCells cells: one, or in the FP32 form
// two (window_pair.cuh).
template <typename R, int kCells>
__device__ __forceinline__ void window_cells(const RunConsts& rc, const NetScalars& ns, const StepPtrs<R>& p,
                                             const WinPtrs<R>& w, i64 win_start, int s_begin, int s_end, int buf,
                                             i64 mark, const Tile& tile) {
    const bool window_done = s_end == w.W;
    const u32 cell = tile.base + threadIdx.x;
    const bool have0 = cell < tile.end;
    const bool have1 = kCells == 2 && have0 && tile.end - cell > blockDim.x;
    if (tile.kind == kAstroCells) {
        bool active[2] = {false, false};
        if (have0) {
            if constexpr (kCells == 2)
                astro_pair_window<R>(rc, ns, p, w, cell, have1, win_start, s_begin, s_end, buf, mark,
                                     window_done, active[0], active[1]);
            else
                active[0] = astro_window<R>(rc, ns, p, w, cell, win_start, s_begin, s_end, buf, mark,
                                            window_done);
        }
        // one word of the active mask per warp and cell row (tiles and blocks start at multiples of 32)
#pragma unroll
        for (int i = 0; i < kCells; ++i) {
            const unsigned ballot = __ballot_sync(0xffffffffu, active[i]);
            if ((threadIdx.x & 31) == 0 && (i == 0 ? have0 : have1)) {
                u32* word = w.astro_active + static_cast<u64>(buf) * w.astro_words + ((cell + i * blockDim.x) >> 5);
                if (s_begin == 0) *word = ballot; else if (ballot) atomicOr(word, ballot);
            }
        }
        return;
    }
    if (!have0) return;
    // one instantiation per population, so its constants are compile-time operands
    if constexpr (kCells == 2) {
        if (tile.kind == kExcCells)
            neuron_pair_window<R, true>(rc, ns, p, w, cell, have1, win_start, s_begin, s_end, buf, window_done);
        else
            neuron_pair_window<R, false>(rc, ns, p, w, cell, have1, win_start, s_begin, s_end, buf, window_done);
    } else if (tile.kind == kExcCells) {
        neuron_window<R, true>(rc, ns, rc.pe, p, w, cell, win_start, s_begin, s_end, buf, window_done);
    } else {
        neuron_window<R, false>(rc, ns, rc.pi, p, w, cell, win_start, s_begin, s_end, buf, window_done);
    }
}

}  // namespace astrosim
