// window.cu -- windowed stepping: one launch per window of D steps plus one push
// launch between windows (see window.cuh).

#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdlib>
#include <map>
#include <tuple>
#include <mutex>
#include <type_traits>
#include <utility>

#include "window_kernels.cuh"

namespace astrosim {

namespace {

// Block and MinBlocks are the block size and the launch-bounds occupancy target
// (resident blocks per SM): the autotuner (window_launch) times the instantiated
// pairs on the first windows of a run and keeps the fastest.  The per-cell
// arithmetic is the same in every instantiation; the kernel indexes cells by
// blockDim.x, so Block = 1024 with MinBlocks = 1 serves any other block size.
template <typename R, int Block, int MinBlocks>
__global__ void __launch_bounds__(Block, MinBlocks) window_kernel(RunConsts rc, StepPtrs<R> p, WinPtrs<R> w,
                                                                  i64 win_start, int s_begin, int s_end, int buf,
                                                                  i64 mark, CellTiles tiles) {
    extern __shared__ __align__(16) unsigned char shared[];
    window_cells<R>(rc, net_scalars(rc), p, w, win_start, s_begin, s_end, buf, mark, tile_of(tiles, blockIdx.x), shared);
}

// The first push_blocks blocks deliver window `buf`'s spikes; the others draw the
// background events of the window that starts at next_start (tiles), Cells neurons per
// thread.  Either part may be absent.  The two touch nothing in common.
template <typename R, int Block, int Cells>
__global__ void __launch_bounds__(Block) push_kernel(WinPtrs<R> w, NetScalars ns, int buf, u32 push_blocks,
                                                     i64 next_start, CellTiles tiles) {
    extern __shared__ u32 rows[];
    if (blockIdx.x < push_blocks)
        push_cells<R>(w, ns.n_exc, ns.n_neurons - ns.n_exc, ns.n_neurons, ns.n_astro, buf, blockIdx.x, push_blocks);
    else
        draw_events<Cells>(ns, w.events, next_start, w.W, tile_of(tiles, blockIdx.x - push_blocks), rows);
}

// Delivers window `buf` (push_warps > 0) and draws the window that starts at next_start
// (draw).  A network that leaves schedulers idle draws one cell per thread in blocks of
// two warps, which spreads the draws over more of them (N = 500: with two cells in blocks
// of eight warps the launch took 8.6 us, of which the draws 7.6); a larger one draws two,
// which shares a warp's unluckiest lane between more draws (67 instead of 74 warp
// instructions per warp of cells and step).
template <typename R>
cudaError_t launch_push(const WinPtrs<R>& w, const NetScalars& ns, int buf, u32 push_warps, bool draw, i64 next_start,
                        cudaStream_t st) {
    const bool spread = ns.n_neurons <= sm_count() * 4 * 32 * 2;
    const int block = spread ? 64 : 256, cells = spread ? 1 : 2;
    const CellTiles tiles = event_tiles(ns.n_exc, 0, ns.n_neurons, block, cells);
    const u32 push_blocks = ceil_div(push_warps * 32, block);
    const u32 grid = push_blocks + (draw ? total_tiles(tiles) : 0);
    if (grid == 0) return cudaSuccess;
    const size_t smem = draw ? poisson_bytes(cells, w.W, block) : 0;
    if (spread) push_kernel<R, 64, 1><<<grid, block, smem, st>>>(w, ns, buf, push_blocks, next_start, tiles);
    else push_kernel<R, 256, 2><<<grid, block, smem, st>>>(w, ns, buf, push_blocks, next_start, tiles);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ forward CSRs
// One warp per target row, so that a row's entries are written by adjacent lanes.
__global__ void edge_rows_kernel(const u32* rs, u32 n_rows, u32* row_of_edge) {
    const u64 r = (static_cast<u64>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (r >= n_rows) return;
    const u32 end = rs[r + 1];
    for (u32 k = rs[r] + (threadIdx.x & 31u); k < end; k += 32) row_of_edge[k] = static_cast<u32>(r);
}

// The same, each entry also naming its place in the row: (row + row0) << 5 | min(place, 31).
__global__ void edge_places_kernel(const u32* rs, u32 n_rows, u32 row0, u32* place_of_edge) {
    const u64 r = (static_cast<u64>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (r >= n_rows) return;
    const u32 start = rs[r], end = rs[r + 1];
    for (u32 k = start + (threadIdx.x & 31u); k < end; k += 32)
        place_of_edge[k] = (static_cast<u32>(r) + row0) << 5 | min(k - start, 31u);
}

__global__ void iota_kernel(u32* v, u64 n) {
    const u64 i = static_cast<u64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) v[i] = static_cast<u32>(i);
}

__global__ void lower_bound_rows_kernel(const u32* sorted_keys, u64 n, u32 n_rows, u32* rs) {
    const u64 t = static_cast<u64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t > n_rows) return;
    u64 lo = 0, hi = n;
    while (lo < hi) {
        const u64 mid = (lo + hi) >> 1;
        if (sorted_keys[mid] < t) lo = mid + 1; else hi = mid;
    }
    rs[t] = static_cast<u32>(lo);
}

__global__ void gather_fwd_kernel(const u32* edge_idx, u64 n, const u32* row_of_edge, const u32* tgt_rs, u32 row0,
                                  u32* dst, u32* pos) {
    const u64 i = static_cast<u64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const u32 e = edge_idx[i];
    const u32 r = row_of_edge[e];
    dst[i] = r + row0;
    if (pos) pos[i] = e - tgt_rs[r];
}

__global__ void add_offset_kernel(u32* v, u64 n, u32 off) {
    const u64 i = static_cast<u64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) v[i] += off;
}

// Inverts a target-keyed CSR into a source-keyed one.  Within one source the
// targets come out in increasing edge order (stable sort), which the push does not
// depend on; positions let e2a deposits name their place in the target row.  Row r
// of `c` is target row0 + r (a network that keeps only its owned cells' rows), and
// the forward lists hold target ids.
// With `places` an entry is target << 5 | min(place in the target's row, 31).
Status invert_csr(const DeviceCSR& c, u32 row0, u32 n_sources, DevBuf<u32>& rs, DevBuf<u32>& dst, DevBuf<u32>* pos,
                  bool places, cudaStream_t st) {
    const u64 n = c.n_edges;
    AS_TRY(rs.alloc(static_cast<size_t>(n_sources) + 1));
    AS_TRY(dst.alloc(n));
    if (pos) AS_TRY(pos->alloc(n));
    if (n == 0) {
        AS_CUDA(cudaMemsetAsync(rs.get(), 0, rs.bytes(), st));
        return Status::Ok();
    }
    DevBuf<u32> row_of, keys_out;
    AS_TRY(row_of.alloc(n));
    AS_TRY(keys_out.alloc(n));
    const u32 row_blocks = ceil_div(static_cast<u64>(c.n_targets) * 32, 256);
    if (places) edge_places_kernel<<<row_blocks, 256, 0, st>>>(c.row_start.get(), c.n_targets, row0, row_of.get());
    else edge_rows_kernel<<<row_blocks, 256, 0, st>>>(c.row_start.get(), c.n_targets, row_of.get());
    AS_CUDA(cudaGetLastError());
    int end_bit = 1;
    while (end_bit < 32 && (1ull << end_bit) < static_cast<u64>(n_sources) + 1) ++end_bit;
    size_t tb = 0;
    if (!pos) {
        // Sorting the target rows themselves by source gives the forward lists
        // directly (the same lists as the edge-index route below, without its index
        // arrays and gather pass).
        AS_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, c.src.get(), keys_out.get(), row_of.get(), dst.get(), n,
                                                0, end_bit, st));
        DevBuf<unsigned char> tmp;
        AS_TRY(tmp.alloc(tb));
        AS_CUDA(cub::DeviceRadixSort::SortPairs(tmp.get(), tb, c.src.get(), keys_out.get(), row_of.get(), dst.get(),
                                                n, 0, end_bit, st));
        lower_bound_rows_kernel<<<ceil_div(static_cast<u64>(n_sources) + 1, 256), 256, 0, st>>>(keys_out.get(), n,
                                                                                              n_sources, rs.get());
        if (row0 && !places) add_offset_kernel<<<ceil_div(n, 256), 256, 0, st>>>(dst.get(), n, row0);
        AS_CUDA(cudaGetLastError());
        AS_CUDA(cudaStreamSynchronize(st));
        return Status::Ok();
    }
    DevBuf<u32> idx_in, idx_out;
    AS_TRY(idx_in.alloc(n));
    AS_TRY(idx_out.alloc(n));
    iota_kernel<<<ceil_div(n, 256), 256, 0, st>>>(idx_in.get(), n);
    AS_CUDA(cudaGetLastError());
    AS_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, c.src.get(), keys_out.get(), idx_in.get(), idx_out.get(), n,
                                            0, end_bit, st));
    DevBuf<unsigned char> tmp;
    AS_TRY(tmp.alloc(tb));
    AS_CUDA(cub::DeviceRadixSort::SortPairs(tmp.get(), tb, c.src.get(), keys_out.get(), idx_in.get(), idx_out.get(), n,
                                            0, end_bit, st));
    lower_bound_rows_kernel<<<ceil_div(static_cast<u64>(n_sources) + 1, 256), 256, 0, st>>>(keys_out.get(), n,
                                                                                          n_sources, rs.get());
    gather_fwd_kernel<<<ceil_div(n, 256), 256, 0, st>>>(idx_out.get(), n, row_of.get(), c.row_start.get(), row0,
                                                        dst.get(), pos->get());
    AS_CUDA(cudaGetLastError());
    AS_CUDA(cudaStreamSynchronize(st));
    return Status::Ok();
}

}  // namespace

Status window_setup(const RunConsts& rc, Network& net, bool fp32, WindowState& ws, cudaStream_t st) {
    ws.W = rc.d_e;
    const u64 nN = rc.n_neurons, nA = rc.n_astro;
    const size_t rb = fp32 ? sizeof(float) : sizeof(double);
    const size_t db = fp32 ? sizeof(Deposit<float>) : sizeof(Deposit<double>);
    // a rank of a sharded network keeps its own cells' rows: its forward lists reach its own cells only
    if (net.has_fwd && net.fwd_exc_rs.size() == static_cast<size_t>(rc.n_exc) + 1 &&
        net.fwd_inh_rs.size() == static_cast<size_t>(net.sz.n_inh) + 1) {
        // the builder wrote these lists while emitting the edges, with the owned rows'
        // indices (cell - n_lo); the forward lists hold target ids
        ws.fwd.exc_rs = std::move(net.fwd_exc_rs);
        ws.fwd.exc_dst = std::move(net.fwd_exc_dst);
        ws.fwd.inh_rs = std::move(net.fwd_inh_rs);
        ws.fwd.inh_dst = std::move(net.fwd_inh_dst);
        net.has_fwd = false;
        if (net.own.n_lo) {
            if (net.exc.n_edges)
                add_offset_kernel<<<ceil_div(net.exc.n_edges, 256), 256, 0, st>>>(ws.fwd.exc_dst.get(),
                                                                                 net.exc.n_edges, net.own.n_lo);
            if (net.inh.n_edges)
                add_offset_kernel<<<ceil_div(net.inh.n_edges, 256), 256, 0, st>>>(ws.fwd.inh_dst.get(),
                                                                                 net.inh.n_edges, net.own.n_lo);
            AS_CUDA(cudaGetLastError());
        }
    } else {
        net.drop_forward();
        AS_TRY(invert_csr(net.exc, net.own.n_lo, rc.n_exc, ws.fwd.exc_rs, ws.fwd.exc_dst, nullptr, false, st));
        AS_TRY(invert_csr(net.inh, net.own.n_lo, net.sz.n_inh, ws.fwd.inh_rs, ws.fwd.inh_dst, nullptr, false, st));
    }
    AS_TRY(invert_csr(net.e2a, net.own.a_lo, rc.n_exc, ws.fwd.e2a_rs, ws.fwd.e2a_astro, &ws.fwd.e2a_pos, false, st));
    AS_TRY(invert_csr(net.sic, net.own.n_lo, rc.n_astro, ws.fwd.sic_rs, ws.fwd.sic_dst, nullptr, true, st));
    // Windows with more spikes than this use the pull gather instead of deposits.
    // ASTROSIM_PUSH_LIMIT overrides it (the tests force the pull path with 0).
    ws.push_limit = static_cast<u32>(std::max<u64>(1024, nN / 50));
    if (const char* env = std::getenv("ASTROSIM_PUSH_LIMIT")) ws.push_limit = static_cast<u32>(std::strtoul(env, nullptr, 10));
    const u32 cap = ws.push_limit + 1;
    AS_TRY(ws.nin_cnt.alloc_zero(2 * nN, st));
    AS_TRY(ws.ain_cnt.alloc_zero(2 * nA, st));
    AS_TRY(ws.nin_ent.alloc(2 * nN * kInboxSlots * db));
    AS_TRY(ws.ain_ent.alloc(2 * nA * kInboxSlots * db));
    AS_TRY(ws.spk_word.alloc_zero(2 * nN, st));
    AS_TRY(ws.spk_val.alloc_zero(2 * static_cast<u64>(ws.W) * nN * rb, st));
    AS_TRY(ws.spk_list.alloc(2 * static_cast<u64>(cap)));
    AS_TRY(ws.spk_count.alloc_zero(2, st));
    AS_TRY(ws.sic_win.alloc_zero(2 * nA * ws.W * rb, st));
    AS_TRY(ws.astro_active.alloc_zero(2 * ((nA + 31) / 32), st));
    AS_TRY(ws.sic_pos.alloc_zero(2 * nN, st));
    AS_TRY(ws.mode.alloc_zero(2, st));
    AS_TRY(ws.events.alloc(nN));
    AS_CUDA(cudaStreamSynchronize(st));
    return Status::Ok();
}

namespace {

// Variants the autotuner chooses from: (block size, minimum resident blocks per SM).
// Each block size comes with three occupancy targets (the same threads per SM as
// the 128-thread entries), trading registers (and a few spills) for occupancy.
struct Variant {
    int block, min_blocks;
};
constexpr Variant kVariantsF32[] = {{128, 6}, {128, 8}, {128, 4}, {64, 12}, {64, 16}, {64, 8},
                                    {256, 3}, {256, 4}, {256, 2}};
constexpr Variant kVariantsF64[] = {{128, 4}, {128, 5}, {128, 3}, {64, 8}, {64, 10}, {64, 6},
                                    {256, 2}, {256, 3}, {256, 1}};
constexpr int kNumVariants = 9;
constexpr int kVariantsPerBlock = 3;
constexpr int kTuneRounds = 2;
static_assert(sizeof(kVariantsF32) / sizeof(Variant) == kNumVariants, "variant table");
static_assert(sizeof(kVariantsF64) / sizeof(Variant) == kNumVariants, "variant table");

// The variants a run may use: every entry for block 0 (the autotuned choice), the
// three entries of a tuned block size, or the generic instantiation (index -1) for
// any other requested block size.
void variant_range(int block, int* first, int* count) {
    for (int b = 0; b < kNumVariants / kVariantsPerBlock; ++b)
        if (kVariantsF32[b * kVariantsPerBlock].block == block) {
            *first = b * kVariantsPerBlock;
            *count = kVariantsPerBlock;
            return;
        }
    if (block == 0) {
        *first = 0;
        *count = kNumVariants;
        return;
    }
    *first = -1;
    *count = 0;
}

std::mutex g_tune_mu;
std::map<std::tuple<int, int, int>, int> g_tuned;  // (precision, log2 size bucket, requested block) -> variant

template <typename R, int B, int M>
cudaError_t launch_one(cudaStream_t st, const RunConsts& rc, const StepPtrs<R>& p, const WinPtrs<R>& w, i64 start,
                       int s0, int s1, int buf, i64 mark, int block) {
    const CellTiles tiles = cell_tiles(rc.n_exc, 0, rc.n_neurons, 0, rc.n_astro, static_cast<u32>(block));
    window_kernel<R, B, M><<<total_tiles(tiles), block, sic_bytes<R>(w.W, block), st>>>(rc, p, w, start, s0, s1, buf,
                                                                                       mark, tiles);
    return cudaGetLastError();
}

template <typename R>
using LaunchFn = cudaError_t (*)(cudaStream_t, const RunConsts&, const StepPtrs<R>&, const WinPtrs<R>&, i64, int, int,
                                 int, i64, int);
template <typename R, int V>
constexpr LaunchFn<R> variant_launch() {
    constexpr Variant v = std::is_same<R, float>::value ? kVariantsF32[V] : kVariantsF64[V];
    return &launch_one<R, v.block, v.min_blocks>;
}
template <typename R, int... V>
constexpr std::array<LaunchFn<R>, sizeof...(V)> variant_launches(std::integer_sequence<int, V...>) {
    return {variant_launch<R, V>()...};
}

// Blocks of the table stay within the 48 KB of shared memory that every kernel may use.  The
// generic kernel's limit is set to its largest block's longest window, the same for every
// network, so that networks stepped by different threads don't lower each other's; and when
// a network first steps, not at each launch (48 networks built by 12 threads with such a call
// at each launch: 200 ms instead of 130).
template <typename R>
cudaError_t allow_generic_blocks() {
    return cudaFuncSetAttribute(window_kernel<R, 1024, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(sic_bytes<R>(kMaxWindow, 1024)));
}

// Launches variant `variant` (an index into the table; -1 = the generic kernel at
// `block` threads).
template <typename R>
cudaError_t launch_window(int variant, int block, cudaStream_t st, const RunConsts& rc, const StepPtrs<R>& p,
                          const WinPtrs<R>& w, i64 start, int s0, int s1, int buf, i64 mark) {
    static constexpr auto table = variant_launches<R>(std::make_integer_sequence<int, kNumVariants>());
    if (variant < 0) return launch_one<R, 1024, 1>(st, rc, p, w, start, s0, s1, buf, mark, block);
    const Variant v = std::is_same<R, float>::value ? kVariantsF32[variant] : kVariantsF64[variant];
    return table[variant](st, rc, p, w, start, s0, s1, buf, mark, v.block);
}

template <typename R>
Status launch_impl(const RunConsts& rc, StateBuffers& sb, Network& net, WindowState& ws, i64 raster_steps, i64 mark,
                   i64 first, i64 count, cudaStream_t st, int block) {
    constexpr bool f32 = std::is_same<R, float>::value;
    StepPtrs<R> p = make_ptrs<R>(sb, net, rc, raster_steps);
    WinPtrs<R> w = win_ptrs<R>(ws, rc);
    const int W = ws.W;
    const u32 push_warps = std::max<u32>(8, std::min<u32>(sm_count() * 64, ws.push_limit));
    int v_first = 0, v_count = 0;
    variant_range(block, &v_first, &v_count);
    if (v_first < 0 && ws.variant != -2) {  // a block size outside the table: the generic kernel, nothing to tune
        AS_CUDA(allow_generic_blocks<R>());
        ws.variant = -2;
    }
    int bucket = 0;
    while ((1ull << bucket) < rc.n_neurons) ++bucket;
    const std::tuple<int, int, int> key{f32 ? 1 : 0, bucket, block};
    if (ws.variant == -1) {
        if (const char* env = std::getenv("ASTROSIM_WINDOW_VARIANT")) {
            ws.variant = v_first + std::min(v_count - 1, std::max(0, std::atoi(env)));
        } else {
            std::lock_guard<std::mutex> lock(g_tune_mu);
            auto it = g_tuned.find(key);
            if (it != g_tuned.end()) ws.variant = it->second;
        }
    }
    const NetScalars ns = net_scalars(rc);
    auto push_and_draw = [&](int buf, u32 warps, bool draw, i64 next) -> Status {
        AS_CUDA(launch_push<R>(w, ns, buf, warps, draw, next * W, st));
        if (draw) ws.events_window = next;
        return Status::Ok();
    };
    i64 t = first;
    const i64 end = first + count;
    if (ws.events_window != first / W) AS_TRY(push_and_draw(0, 0, true, first / W));
    while (t < end) {
        const i64 k = t / W;
        const int s0 = static_cast<int>(t - k * W);
        const int s1 = static_cast<int>(std::min<i64>(W, end - k * W));
        const int buf = static_cast<int>(k & 1);
        const bool tuning = ws.variant == -1 && s0 == 0 && s1 == W;
        int v = ws.variant >= 0 ? ws.variant : (tuning ? v_first + ws.tune_step % v_count : v_first);
        if (ws.variant == -2) v = -1;
        if (tuning && !ws.tune_ev[0]) {  // made on the first tuned window only
            AS_CUDA(cudaEventCreate(&ws.tune_ev[0]));
            AS_CUDA(cudaEventCreate(&ws.tune_ev[1]));
        }
        if (tuning) AS_CUDA(cudaEventRecord(ws.tune_ev[0], st));
        AS_CUDA(launch_window<R>(v, block, st, rc, p, w, k * W, s0, s1, buf, mark));
        if (tuning) {
            AS_CUDA(cudaEventRecord(ws.tune_ev[1], st));
            AS_CUDA(cudaEventSynchronize(ws.tune_ev[1]));
            float ms = 0.f;
            AS_CUDA(cudaEventElapsedTime(&ms, ws.tune_ev[0], ws.tune_ev[1]));
            float& slot = ws.tune_ms[v];
            slot = std::min(slot, ms);  // min over rounds: the first launch also loads the kernel
            if (++ws.tune_step == v_count * kTuneRounds) {
                int best = v_first;
                for (int i = v_first + 1; i < v_first + v_count; ++i)
                    if (ws.tune_ms[i] < ws.tune_ms[best]) best = i;
                ws.variant = best;
                std::lock_guard<std::mutex> lock(g_tune_mu);
                g_tuned[key] = best;
            }
        }
        if (s1 == W) AS_TRY(push_and_draw(buf, push_warps, (k + 1) * W < end, k + 1));
        t = k * W + s1;
    }
    return Status::Ok();
}
}  // namespace

Status window_launch(const RunConsts& rc, StateBuffers& sb, Network& net, bool fp32, WindowState& ws,
                     i64 raster_steps, i64 mark_step, i64 first, i64 count, cudaStream_t st, int block) {
    if (fp32) return launch_impl<float>(rc, sb, net, ws, raster_steps, mark_step, first, count, st, block);
    return launch_impl<double>(rc, sb, net, ws, raster_steps, mark_step, first, count, st, block);
}

}  // namespace astrosim
