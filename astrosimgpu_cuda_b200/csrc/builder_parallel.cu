// builder_parallel.cu -- the chunked parallel connectivity builder.
//
// The reference builds connectivity from ONE sequential random stream
// (src/astrosim_fused.cu:631-723): after the pools, every presynaptic neuron
// ("pre") walks its postsynaptic block with geometric skips, and each landing may
// consume one or two more draws (the P_THIRD test and the pool pick).  The number
// of draws a pre consumes depends on the draws themselves, so the tape position
// where pre r starts is a prefix sum nobody knows in advance.  This file finds
// every pre's start exactly, in parallel, and then emits all edges in the
// reference's emission order:
//
//  1. Pools: each post's pool is 5 draws unless a duplicate forces a redraw;
//     offsets are found by a fixed-point iteration (each round fixes at least the
//     first misplaced post).
//  2. Draw cache: for every tape position the walks can reach, its skip
//     floor(log1p(-u) / log1p(-p)), its third-factor test and its pool pick in one
//     word, computed once (walk_chunked.cuh); ambiguous skips (quotient within a few
//     ulps of an integer) are settled with the host C library that the reference uses.
//  3. For each walk section (E block, I block, inhibitory pres): the length of the pre
//     that would start at each tape position (walk_chunked.cuh), in parallel.  The
//     section's tape is cut into chunks; from EVERY candidate entry position in
//     [T, T + delta) of a chunk -- its first pre start must be one of them -- a thread
//     follows the lengths to the chunk's end: an exact table entry -> (exit, pres
//     started).  Tables are composed (groups in parallel, then one thread over the
//     groups), which yields every chunk's true entry, and one thread per chunk then
//     writes every pre's start ("orbit").
//  4. The lengths ignore one index-dependent rule: in the E block a pre
//     that lands on its own index skips its P_THIRD draws (no autapses).  Such
//     landings are rare (about 80 per network) but shift the stream, so: every
//     pre whose walk lands within +-K of its own index is a hazard; one block then
//     replays the hazards in order with the running index shift: from each one that
//     is an autapse it follows the lengths, checking batches of pres for further
//     autapses, until it rejoins the table orbit, and splices the true orbit.
//  5. Count and emit: one thread per pre walks its row again (exact rules,
//     including autapses), first counting, then writing edges at scanned offsets.
//     The lists are in emission order (the two excitatory blocks interleaved by pre,
//     which makes the excitatory list source-major); the stable radix sort of
//     builder.cu turns them into the target-keyed CSRs, and the exc and inh lists
//     are kept as the windowed engine's forward lists.
// Every step is exact; the outcome is bit-identical to the sequential walk.

#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <vector>

#include "builder_internal.cuh"
#include "pool_offsets.h"
#include "walk.cuh"
#include "walk_chunked.cuh"

namespace astrosim {

namespace {

constexpr u32 kMaxDelta = kMaxPre;  // candidate entries per chunk
// A section with fewer than target_chunks() (8 per SM) chunks of kChunkLen positions
// runs with shorter chunks, down to kMinChunkLen (4 x kMaxDelta): the table and orbit
// passes follow one chunk per thread, pre after pre, so on small networks
// the chunk length, not the network, sets their time.  The chunking never changes
// the result, only how the walk is split.
inline u32 target_chunks() { return sm_count() * 8; }
constexpr u32 kMinChunkLen = 2048, kChunkLen = 16384;

// ---------------------------------------------------------------- pools
__global__ void pool_pass_kernel(u64 seed, u32 n_neurons, u32 n_astro, u32 take, u64 base, const u64* prefix,
                                 u32* pool, u64* extra) {
    const u32 q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n_neurons) return;
    u64 c = base + static_cast<u64>(take) * q + prefix[q];
    const u64 c0 = c;
    pool_one(seed, n_astro, c, pool + static_cast<u64>(q) * kPoolSize);
    extra[q] = c - c0 - take;
}

// Tape positions where a pool started there needs redraws (a duplicate pick), with
// the number of extra draws: every t in [t0, t0 + n).
struct PoolRedraw {
    u64 t;
    u32 extra, pad_;
};

__global__ void pool_redraw_kernel(u64 seed, u32 n_astro, u32 take, u64 t0, u64 n, PoolRedraw* out, unsigned* count,
                                   unsigned cap) {
    const u64 stride = static_cast<u64>(gridDim.x) * blockDim.x;
    u32 pl[kPoolSize];
    for (u64 i = static_cast<u64>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        u64 c = t0 + i;
        pool_one(seed, n_astro, c, pl);
        const u64 extra = c - (t0 + i) - take;
        if (extra) {
            const unsigned k = atomicAdd(count, 1u);
            if (k < cap) out[k] = PoolRedraw{t0 + i, static_cast<u32>(extra), 0u};
        }
    }
}

__global__ void scatter_extra_kernel(const u32* q, const u32* e, u32 n, u64* extra) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) extra[q[i]] = e[i];
}

__global__ void diff_kernel(const u64* a, const u64* b, u64 n, int* flag) {
    const u64 i = static_cast<u64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n && a[i] != b[i]) *flag = 1;
}

// ---------------------------------------------------------------- draw cache
__global__ void draw_cache_kernel(u64 seed, double L, u64 base, u64 n, u32 take, u32* cache, AmbiguityLog amb) {
    const u64 stride = static_cast<u64>(gridDim.x) * blockDim.x;
    const SkipTable none{};
    for (u64 i = static_cast<u64>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
        cache[i] = draw_word(rng_bits(seed, kSetupStream, base + i) >> 11, skip_value(seed, L, base + i, none, amb),
                             take);
}

// ---------------------------------------------------------------- pre lengths and chunk tables
// lens[i]: the length of the pre that starts at tape position start + i (0: it leaves the
// cache, kLongPre: it is too long).  One tile of positions per block, its words and jumps
// in shared memory: 56 KB for 4096 positions and the words a pre may reach past them.
// Bound by the shared-memory reads of the jumps.
constexpr u32 kLenTile = 4096, kLenBlock = 512;
constexpr u32 kLenWords = kLenTile + kWordsAhead + 64, kLenJumps = kLenTile + kJumpsAhead;
constexpr size_t kLenShared = (kLenWords + 2 * kLenJumps + 64) * sizeof(u32);

__global__ void __launch_bounds__(kLenBlock) pre_length_kernel(Sec s, u64 start, u64 n, u16* lens) {
    extern __shared__ u32 words[];
    u32* jumps4 = words + kLenWords;
    u32* jumps16 = jumps4 + kLenJumps + 48;
    const u64 tile = static_cast<u64>(blockIdx.x) * kLenTile;
    for (u32 i = threadIdx.x; i < kLenWords; i += kLenBlock) words[i] = peek(s, start + tile + i);
    __syncthreads();
    for (u32 i = threadIdx.x; i < kLenJumps + 36; i += kLenBlock) jumps4[i] = jump4(s, words, i);
    __syncthreads();
    for (u32 i = threadIdx.x; i < kLenJumps; i += kLenBlock) jumps16[i] = jump16(jumps4, i);
    __syncthreads();
    const u64 end = s.cache_base + s.cache_len;
    for (u32 i = threadIdx.x; i < kLenTile && tile + i < n; i += kLenBlock) {
        const u32 len = pre_length(s, words, jumps4, jumps16, i);
        lens[tile + i] = static_cast<u16>(start + tile + i + len > end ? 0u : len);
    }
}

// A chunk's lengths into shared memory (chunk_len is a multiple of 8, chunks are 16-byte aligned).
__device__ __forceinline__ void stage_lengths(const u16* lens, u32 chunk, u32 chunk_len, u16* shared) {
    const uint4* from = reinterpret_cast<const uint4*>(lens + static_cast<u64>(chunk) * chunk_len);
    uint4* to = reinterpret_cast<uint4*>(shared);
    for (u32 i = threadIdx.x; i < chunk_len / 8; i += blockDim.x) to[i] = from[i];
    __syncthreads();
}

// One block per chunk, one thread per candidate entry: t_exit/t_cnt[chunk * delta + d] for
// the walk from tape position sec_start + chunk * chunk_len + d.
__global__ void table_kernel(Sec s, const u16* lens, u64 sec_start, u32 chunk_len, u32 delta, u64* t_exit, u32* t_cnt) {
    extern __shared__ __align__(16) u16 len[];
    stage_lengths(lens, blockIdx.x, chunk_len, len);
    const u32 w = threadIdx.x;
    if (w >= delta) return;
    u32 c = w, cnt = 0;
    while (c < chunk_len) {
        const u32 l = len[c];
        if (l == 0 || l == kLongPre) {
            atomicOr(s.err, l ? kErrDelta : kErrCache);
            break;
        }
        c += l;
        ++cnt;
    }
    t_exit[static_cast<u64>(blockIdx.x) * delta + w] = sec_start + static_cast<u64>(blockIdx.x) * chunk_len + c;
    t_cnt[static_cast<u64>(blockIdx.x) * delta + w] = cnt;
}

// Composes the tables of `group` consecutive chunks: thread d follows candidate d.
__global__ void group_compose_kernel(Sec s, u64 sec_start, u32 chunk_len, u32 delta, u32 n_chunks, u32 group,
                                     const u64* t_exit, const u32* t_cnt, u64* g_exit, u64* g_cnt) {
    const u32 g = blockIdx.x, d = threadIdx.x;
    if (d >= delta) return;
    const u32 c0 = g * group;
    const u32 c1 = min(c0 + group, n_chunks);
    u64 x = d, cnt = 0, e = 0;
    for (u32 i = c0; i < c1; ++i) {
        if (x >= delta) {
            atomicOr(s.err, kErrDelta);
            break;
        }
        e = t_exit[static_cast<u64>(i) * delta + x];
        cnt += t_cnt[static_cast<u64>(i) * delta + x];
        x = e - (sec_start + static_cast<u64>(i + 1) * chunk_len);
    }
    g_exit[static_cast<u64>(g) * delta + d] = e;
    g_cnt[static_cast<u64>(g) * delta + d] = cnt;
}

// One thread over the groups: the true entry and pre index of every group, up to
// the group where `target` pres are reached (*end_group, n_groups if they are not).
__global__ void top_compose_kernel(Sec s, u64 sec_start, u32 chunk_len, u32 delta, u32 n_groups, u32 group,
                                   const u64* g_exit, const u64* g_cnt, u64 target, u64* g_entry, u64* g_g0,
                                   u32* end_group) {
    u64 e = sec_start, cnt = 0;
    u32 g = 0;
    for (; g < n_groups; ++g) {
        g_entry[g] = e;
        g_g0[g] = cnt;
        const u64 d = e - (sec_start + static_cast<u64>(g) * group * chunk_len);
        if (d >= delta) {
            atomicOr(s.err, kErrDelta);
            break;
        }
        cnt += g_cnt[static_cast<u64>(g) * delta + d];
        e = g_exit[static_cast<u64>(g) * delta + d];
        if (cnt >= target) break;
    }
    *end_group = g;
}

// Per group: the entry and first pre index of each of its chunks (a first index of all
// ones for the chunks after the end group, which start no pre that is needed).
__global__ void chunk_entry_kernel(Sec s, u64 sec_start, u32 chunk_len, u32 delta, u32 n_chunks, u32 n_groups, u32 group,
                                   const u64* t_exit, const u32* t_cnt, const u64* g_entry, const u64* g_g0,
                                   const u32* end_group, u64* c_entry, u64* c_g0) {
    const u32 g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n_groups) return;
    const u32 c0 = g * group, c1 = min(c0 + group, n_chunks);
    bool known = g <= *end_group;
    u64 e = known ? g_entry[g] : 0, cnt = known ? g_g0[g] : ~u64(0);
    for (u32 i = c0; i < c1; ++i) {
        const u64 d = e - (sec_start + static_cast<u64>(i) * chunk_len);
        if (known && d >= delta) {
            atomicOr(s.err, kErrDelta);
            known = false;
        }
        c_entry[i] = e;
        c_g0[i] = known ? cnt : ~u64(0);
        if (!known) continue;
        cnt += t_cnt[static_cast<u64>(i) * delta + d];
        e = t_exit[static_cast<u64>(i) * delta + d];
    }
}

// One block per chunk; its first thread writes the start of every pre that begins in the
// chunk, up to pre `limit`, and the end of pre `last`.
__global__ void materialize_kernel(Sec s, const u16* lens, u64 sec_start, u32 chunk_len, u32 n_chunks,
                                   const u64* c_entry, const u64* c_g0, u64 limit, u64 last, u64* orbit, u64* end) {
    extern __shared__ __align__(16) u16 len[];
    const u32 i = blockIdx.x;
    u64 idx = c_g0[i];
    if (idx >= limit) return;
    stage_lengths(lens, i, chunk_len, len);
    if (threadIdx.x) return;
    const u64 T0 = sec_start + static_cast<u64>(i) * chunk_len;
    u32 c = static_cast<u32>(c_entry[i] - T0);
    while (c < chunk_len && idx < limit) {
        const u32 l = len[c];
        if (l == 0 || l == kLongPre) return;  // the table pass flagged it
        orbit[idx] = T0 + c;
        c += l;
        if (idx == last) *end = T0 + c;
        ++idx;
    }
    if (idx < limit && i + 1 < n_chunks && c_g0[i + 1] != ~u64(0) && T0 + c != c_entry[i + 1])
        atomicOr(s.err, kErrOrbit);
}

// ---------------------------------------------------------------- autapse hazards (E block)
struct Hazard {
    u32 r;    // index in the table orbit
    int d;    // landing post - r
};

struct HazardVisit {
    u32 r;
    int K;
    Hazard* out;
    unsigned* n;
    unsigned cap;
    __device__ __forceinline__ void operator()(u32 post, bool, u32) const {
        const long long d = static_cast<long long>(post) - static_cast<long long>(r);
        if (d >= -K && d <= K) {
            const unsigned k = atomicAdd(n, 1u);
            if (k < cap) out[k] = Hazard{r, static_cast<int>(d)};
        }
    }
};

__global__ void hazard_kernel(Sec s, const u64* orbit, u64 n, int K, Hazard* out, unsigned* count, unsigned cap,
                              const u32* end_group, u32 n_groups) {
    const u64 r = static_cast<u64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (r >= n || *s.err || *end_group >= n_groups) return;  // no complete table orbit
    HazardVisit v{static_cast<u32>(r), K, out, count, cap};
    walk_pre(s, orbit[r], kNoSelf, v);
}

// Index of c in the sorted orbit, or -1.  `from` is a lower bound of where c can be; the
// search gallops from there, so a walk that keeps pace with the orbit costs one or two
// loads per query instead of a full binary search.
__device__ __forceinline__ long long find_in_orbit(const u64* orbit, u64 n, u64 c, u64 from) {
    u64 lo = from, hi = n;
    if (lo < n && orbit[lo] < c) {
        u64 step = 1;
        hi = lo + 1;
        while (hi < n && orbit[hi] < c) {
            lo = hi;
            step *= 2;
            hi = lo + step < n ? lo + step : n;
        }
        ++lo;  // orbit[lo - 1] < c
    } else {
        hi = lo;
    }
    while (lo < hi) {  // the first index in [lo, hi) with orbit[index] >= c
        const u64 mid = (lo + hi) >> 1;
        if (orbit[mid] < c) lo = mid + 1; else hi = mid;
    }
    return (lo < n && orbit[lo] == c) ? static_cast<long long>(lo) : -1;
}

// The spliced orbit: piece p covers true indices [t_start[p], t_start[p] + len) and
// is read from src[p]; pieces are in index order and tile [0, n).
struct OrbitPiece {
    const u64* src;
    u64 t_start, len;
};

struct Replay {
    u64 end;         // tape position after the section
    u32 n_pieces;
    u32 retry;       // the shift left the hazards' range, or the table orbit was too short for it
    u32 full;        // more pieces than their table holds
    u32 pad_;
};

constexpr u32 kReplayOrbit = 64;  // table starts that the replay keeps around its walk

// The first of the kReplayOrbit ascending entries that is not below c (the last is not).
__device__ __forceinline__ u32 lower_bound_near(const u64* entries, u64 c) {
    u32 lo = 0, hi = kReplayOrbit - 1;
    while (lo < hi) {
        const u32 mid = (lo + hi) >> 1;
        if (entries[mid] < c) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// The replay of the E block's autapses in order (one block).  On the table orbit with
// running shift d (true index - table index) the next autapse is the next hazard that
// lands d from its table index.  From there the walk leaves the table orbit: its pres are
// taken in batches of up to 32, whose starts follow from the lengths; a lane walks each pre
// in full for a landing on its true index and looks its start up in the table orbit.  The
// first of the two ends the batch: an autapse sends the walk on from that pre's exact end,
// a start on the table orbit ends it.  (The first batch, of 4, ends after its first pre,
// the autapse that the walk starts at; walks rejoin after a median of 2 pres from there,
// some after hundreds.)  What bounds it is
// latency: the load of the window and a lane's walk of about a hundred words.  512 threads
// load, look through the hazards in shared memory and through the table starts around the
// walk, and a landing waits once for its two words: 1.3 ms at N = 1e3, 2.6 ms at N = 3e5 (1.5
// and 3.0 with a wait for each); 128 threads that read hazards and table
// starts from global memory took 2.8 and 6.3 ms.
constexpr u32 kReplayBlock = 512, kReplayBatch = 32, kReplayWindow = 8192;
constexpr u32 kReplayWords = kReplayWindow + kWordsAhead;
constexpr u32 kReplayHazards = 6144;  // hazards kept in shared memory (5200 expected), all or none
constexpr size_t kReplayShared = kReplayWords * sizeof(u32) + kReplayWindow * sizeof(u16) + kReplayHazards * sizeof(Hazard);

__global__ void __launch_bounds__(kReplayBlock) replay_kernel(Sec s, const u16* lens, u64 sec_start, u64 n_lens,
                                                              const Hazard* hz, const unsigned* n_hz_ptr,
                                                              unsigned hz_cap, const u64* orbit, u64 n_orbit,
                                                              u64 n_pres, int K, const u32* end_group, u32 n_groups,
                                                              u64* starts, OrbitPiece* pieces, u32 piece_cap,
                                                              Replay* out) {
    extern __shared__ __align__(16) u32 words[];
    u16* len = reinterpret_cast<u16*>(words + kReplayWords);
    Hazard* near_hz = reinterpret_cast<Hazard*>(len + kReplayWindow);
    __shared__ u64 batch[kReplayBatch + 1];  // the batch's starts, and where it ends
    __shared__ u64 near_orbit[kReplayOrbit];
    __shared__ u32 n_batch;
    __shared__ unsigned best;
    __shared__ u64 merge_k, auto_end;
    __shared__ u32 merge_at, auto_at, past_lens;
    Replay res{0, 0, 0, 0, 0};
    // an unfinished or failed table pass: the host looks at its flags first
    const unsigned n_hz = *n_hz_ptr;
    if (*s.err || *end_group >= n_groups || n_hz > hz_cap) {
        if (threadIdx.x == 0) *out = res;
        return;
    }
    const bool staged_hz = n_hz <= kReplayHazards;
    if (staged_hz) {
#pragma unroll 4
        for (u32 i = threadIdx.x; i < n_hz; i += kReplayBlock) near_hz[i] = hz[i];
        __syncthreads();
    }
    auto add_piece = [&](const u64* src, u64 t, u64 n) {
        if (n == 0) return;
        if (res.n_pieces == piece_cap) {
            res.full = 1;
            return;
        }
        if (threadIdx.x == 0) pieces[res.n_pieces] = OrbitPiece{src, t, n};
        ++res.n_pieces;
    };
    long long d = 0;
    u64 cur_f = 0, cur_t = 0, n_starts = 0;
    bool ended = false;
    while (!ended && !res.full && !res.retry) {
        // the next hazard on the orbit at this shift
        if (threadIdx.x == 0) best = 0xFFFFFFFFu;
        __syncthreads();
        unsigned mine = 0xFFFFFFFFu;
        for (u32 i = threadIdx.x; i < n_hz; i += kReplayBlock) {
            const Hazard h = staged_hz ? near_hz[i] : hz[i];
            if (h.d == d && h.r >= cur_f) mine = min(mine, h.r);
        }
        if (mine != 0xFFFFFFFFu) atomicMin(&best, mine);
        __syncthreads();
        const unsigned at = best;
        if (at == 0xFFFFFFFFu || static_cast<long long>(at) + d >= static_cast<long long>(n_pres)) break;
        add_piece(orbit + cur_f, cur_t, at - cur_f);
        u64 c = orbit[at], r = static_cast<u64>(static_cast<long long>(at) + d);
        const u64 t_autapse = r, first_start = n_starts;
        u64 from = at;
        bool on_orbit_start = true;  // batch 0's first pre is the hazard itself, on the table orbit
        bool rejoined = false;
        u32 batch_max = 4;
        while (!rejoined && !ended) {
            const u64 i0 = c - sec_start;  // the window: lengths and words from c on
            const u32 window = batch_max == 4 ? 4 * kMaxPre : kReplayWindow;
#pragma unroll 8
            for (u32 i = threadIdx.x; i < window; i += kReplayBlock) len[i] = i0 + i < n_lens ? lens[i0 + i] : u16(0);
#pragma unroll 8
            for (u32 i = threadIdx.x; i < window + kWordsAhead; i += kReplayBlock) words[i] = peek(s, c + i);
            if (threadIdx.x < kReplayOrbit)
                near_orbit[threadIdx.x] = from + threadIdx.x < n_orbit ? orbit[from + threadIdx.x] : ~u64(0);
            if (threadIdx.x == 0) {
                merge_at = auto_at = 0xFFFFFFFFu;
                past_lens = 0;
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                u32 x = 0, n = 0;
                while (n < batch_max && r + n < n_pres && x + kMaxPre <= window) {
                    const u32 l = len[x];
                    if (l == 0 || l == kLongPre) {
                        if (i0 + x >= n_lens) past_lens = 1;
                        else atomicOr(s.err, l ? kErrDelta : kErrCache);
                        break;
                    }
                    batch[n++] = c + x;
                    x += l;
                }
                batch[n] = c + x;
                n_batch = n;
            }
            __syncthreads();
            const u32 n = n_batch;
            if (n == 0) {  // the walk left the lengths, or (flagged) the cache, or met a pre that is too long
                res.retry = past_lens;
                if (threadIdx.x == 0) *out = res;
                return;
            }
            if (threadIdx.x < n) {
                const u32 q = threadIdx.x;
                const u64 start = batch[q];
                // an autapse: the walk lands on its true index (src/astrosim_fused.cu:696)
                const unsigned lanes = n == 32 ? 0xFFFFFFFFu : (1u << n) - 1u;
                const u32 self = static_cast<u32>(r + q) - s.post_off;
                u32 x = static_cast<u32>(start - c), left = s.post_count;
                bool hit_self = false;
                u32 skip = words[x++], test = words[x];  // the test's word with the skip's: one wait per landing
                for (;;) {
                    const u32 g = skip & kSkipMax;
                    if (g >= left) break;
                    if (x + 4 > window + kWordsAhead) {
                        atomicOr(s.err, kErrDelta);
                        break;
                    }
                    const bool own = s.post_count - left + g == self;
                    hit_self = hit_self || own;
                    left -= g + 1;
                    if (s.third && !own) x += (test & kHitBit) ? 2 : 1;
                    if (left == 0) break;
                    skip = words[x++];
                    test = words[x];
                }
                long long k = -1;
                if (q || !on_orbit_start) {
                    if (start <= near_orbit[kReplayOrbit - 1]) {
                        const u32 at_near = lower_bound_near(near_orbit, start);
                        if (near_orbit[at_near] == start) k = static_cast<long long>(from + at_near);
                    } else {
                        k = find_in_orbit(orbit, n_orbit, start, from + kReplayOrbit - 1);
                    }
                }
                if (k >= 0) atomicMin(&merge_at, q);
                if (hit_self) atomicMin(&auto_at, q);
                __syncwarp(lanes);
                if (k >= 0 && merge_at == q) merge_k = static_cast<u64>(k);
                if (hit_self && auto_at == q) auto_end = c + x;
            }
            __syncthreads();
            const u32 m = merge_at, a = auto_at;
            const u32 taken = m <= a && m != 0xFFFFFFFFu ? m : (a != 0xFFFFFFFFu ? a + 1 : n);
            if (threadIdx.x < taken) starts[n_starts + threadIdx.x] = batch[threadIdx.x];
            n_starts += taken;
            r += taken;
            if (m <= a && m != 0xFFFFFFFFu) {
                cur_f = merge_k;
                cur_t = r;
                d = static_cast<long long>(r) - static_cast<long long>(cur_f);
                rejoined = true;
            } else {
                c = a != 0xFFFFFFFFu ? auto_end : batch[n];
                if (r >= n_pres) {
                    ended = true;
                    res.end = c;
                    cur_t = r;
                }
            }
            on_orbit_start = false;
            batch_max = kReplayBatch;
            // the table starts from the walk's place on; one that outran them catches up by a search
            if (c <= near_orbit[kReplayOrbit - 1]) {
                from += lower_bound_near(near_orbit, c);
            } else {
                u64 lo = from + kReplayOrbit - 1, hi = n_orbit;
                while (lo < hi) {
                    const u64 mid = (lo + hi) >> 1;
                    if (orbit[mid] < c) lo = mid + 1; else hi = mid;
                }
                from = lo;
            }
            __syncthreads();  // the batch and the window are read before the next ones are written
        }
        add_piece(starts + first_start, t_autapse, n_starts - first_start);
        if (rejoined && (d < -K || d > K)) res.retry = 1;
    }
    if (!ended && !res.full && !res.retry) {
        const u64 n = n_pres - cur_t;
        if (cur_f + n > n_orbit) {
            res.retry = 1;  // the table orbit ends before the section does
        } else {
            add_piece(orbit + cur_f, cur_t, n);
            // the last pre is no autapse (it would have been a hazard), so its length holds
            if (n) res.end = orbit[cur_f + n - 1] + lens[orbit[cur_f + n - 1] - sec_start];
        }
    }
    if (threadIdx.x == 0) *out = res;
}

__global__ void splice_orbit_kernel(const OrbitPiece* pieces, const Replay* replay, u64 n, u64* dst) {
    const u64 i = static_cast<u64>(blockIdx.x) * blockDim.x + threadIdx.x;
    const u32 n_pieces = replay->n_pieces;
    if (i >= n || n_pieces == 0) return;
    u32 lo = 0, hi = n_pieces;  // the last piece with t_start <= i
    while (hi - lo > 1) {
        const u32 mid = (lo + hi) >> 1;
        if (pieces[mid].t_start <= i) lo = mid; else hi = mid;
    }
    const OrbitPiece p = pieces[lo];
    if (i - p.t_start < p.len) dst[i] = p.src[i - p.t_start];
}

// ---------------------------------------------------------------- count and emit
// Owned targets of the build (CellRange): an exc/inh edge and an a2n (sic) edge are
// kept when their neuron target is owned, an e2a edge when its astrocyte is.
struct Owned {
    u32 n_lo, n_hi, a_lo, a_hi;
    __device__ __forceinline__ bool neuron(u32 post) const { return post >= n_lo && post < n_hi; }
    __device__ __forceinline__ bool astro(u32 a) const { return a >= a_lo && a < a_hi; }
};

// Per pre: kept primary edges, kept e2a edges, kept sic edges; and every edge for
// the whole network's totals.
struct CountVisit {
    Owned own;
    u64 ne = 0, na = 0, ns = 0;
    u32 te = 0, tt = 0;
    __device__ __forceinline__ void operator()(u32 post, bool hit, u32 astro) {
        const bool pn = own.neuron(post);
        ++te;
        ne += pn ? 1u : 0u;
        if (hit) {
            ++tt;
            na += own.astro(astro) ? 1u : 0u;
            ns += pn ? 1u : 0u;
        }
    }
};

__device__ __forceinline__ u32 self_post_of(int mode, u32 r, u32 self_off) {
    return mode == 0 ? kNoSelf : r + self_off;  // mode 1: autapse at post == r + self_off
}

// totals[0] += every primary edge, totals[1] += every third-factor edge (one atomic per warp).
__global__ void count_kernel(Sec s, const u64* orbit, u64 n, int self_mode, u32 self_off, Owned own, u64* ce,
                             u64* ca, u64* cs, unsigned long long* totals) {
    const u64 r = static_cast<u64>(blockIdx.x) * blockDim.x + threadIdx.x;
    CountVisit v{own};
    if (r < n) {
        walk_pre(s, orbit[r], self_post_of(self_mode, static_cast<u32>(r), self_off), v);
        ce[r] = v.ne;
        ca[r] = v.na;
        cs[r] = v.ns;
    }
    unsigned long long te = v.te, tt = v.tt;
    for (int off = 16; off > 0; off >>= 1) {
        te += __shfl_down_sync(0xffffffffu, te, off);
        tt += __shfl_down_sync(0xffffffffu, tt, off);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&totals[0], te);
        atomicAdd(&totals[1], tt);
    }
}

// One output stream of one emitting thread: values go to p[o], p[o + 1], ...  Whole
// 32-byte sectors leave as two 16-byte stores from an 8-value buffer in shared
// memory; only the partial sectors at the two ends of a pre's run get single
// stores.  With a single 4-byte store per value, L2 held partly written sectors
// and filled each from DRAM before writing it back: at N = 3e6 the E block's
// emission moved 32 GB of DRAM traffic for about 1.7 GB of edges.  The buffer is
// stream-major in shared memory (value k of thread t at buf[k * kEmitBlock]), so
// lanes at the same fill level hit different banks.
constexpr u32 kEmitBlock = 128;

struct SectorWriter {
    u32* p;
    u64 o;
    u32* buf;
    u32 k;
    __device__ __forceinline__ void put(u32 v) {
        if (k == 0 && (reinterpret_cast<unsigned long long>(p + o) & 31u)) {  // up to the next sector boundary
            p[o++] = v;
            return;
        }
        buf[k * kEmitBlock] = v;
        if (++k == 8) {
            const uint4 a = make_uint4(buf[0], buf[kEmitBlock], buf[2 * kEmitBlock], buf[3 * kEmitBlock]);
            const uint4 b = make_uint4(buf[4 * kEmitBlock], buf[5 * kEmitBlock], buf[6 * kEmitBlock],
                                       buf[7 * kEmitBlock]);
            *reinterpret_cast<uint4*>(p + o) = a;
            *reinterpret_cast<uint4*>(p + o + 4) = b;
            o += 8;
            k = 0;
        }
    }
    __device__ __forceinline__ void flush() {
        for (u32 i = 0; i < k; ++i) p[o + i] = buf[i * kEmitBlock];
        o += k;
        k = 0;
    }
};

// The edges of one pre.  The sources of the exc, inh and e2a lists are the pre
// itself and are filled in afterwards (fill_rows_kernel); the sic list's sources
// are astrocytes and are written here.
struct EmitVisit {
    Owned own;
    SectorWriter e_dst, t_dst, s_src, s_dst;
    __device__ __forceinline__ void operator()(u32 post, bool hit, u32 astro) {
        const bool pn = own.neuron(post);
        if (pn) e_dst.put(post - own.n_lo);
        if (hit) {
            if (own.astro(astro)) t_dst.put(astro - own.a_lo);
            if (pn) {
                s_src.put(astro);
                s_dst.put(post - own.n_lo);
            }
        }
    }
};

__global__ void __launch_bounds__(kEmitBlock) emit_kernel(Sec s, const u64* orbit, u64 n, int self_mode,
                                                          u32 self_off, Owned own, const u64* oe, const u64* oa,
                                                          const u64* os, u64 base_e, u64 base_a, u64 base_s,
                                                          u32* e_dst, u32* t_dst, u32* s_src, u32* s_dst) {
    __shared__ u32 sbuf[4 * 8 * kEmitBlock];
    const u64 r = static_cast<u64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (r >= n) return;
    u32* b = sbuf + threadIdx.x;
    EmitVisit v{own,
                SectorWriter{e_dst, base_e + oe[r], b, 0u},
                SectorWriter{t_dst, base_a + oa[r], b + 8 * kEmitBlock, 0u},
                SectorWriter{s_src, base_s + os[r], b + 16 * kEmitBlock, 0u},
                SectorWriter{s_dst, base_s + os[r], b + 24 * kEmitBlock, 0u}};
    walk_pre(s, orbit[r], self_post_of(self_mode, static_cast<u32>(r), self_off), v);
    v.e_dst.flush();
    v.t_dst.flush();
    v.s_src.flush();
    v.s_dst.flush();
}

// out[i] = r for every i of row r, rows [base + o[r], base + o[r + 1]) (the last one
// ends at base + total): the source lists whose source is the row's pre.  One warp
// per row, so the writes are coalesced.
__global__ void fill_rows_kernel(const u64* o, u64 n, u64 base, u64 total, u32* out) {
    const u64 t = static_cast<u64>(blockIdx.x) * blockDim.x + threadIdx.x;
    const u64 r = t >> 5;
    if (r >= n) return;
    const u64 b = base + o[r], e = base + (r + 1 < n ? o[r + 1] : total);
    for (u64 i = b + (threadIdx.x & 31u); i < e; i += 32) out[i] = static_cast<u32>(r);
}

// Excitatory edge layout, source-major: pre r's E-block edges (exc targets) then its
// I-block edges (inh targets) at fwd_rs[r] = oe_e[r] + oe_i[r] (the two blocks'
// exclusive scans over the same pres); o_e / o_i (the scans, in place) become each
// block's emission offsets.  fwd_rs[n] = total.
__global__ void exc_layout_kernel(u64 n, u64* o_e, u64* o_i, const u64* c_e, u64 total, u32* fwd_rs) {
    const u64 r = static_cast<u64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (r < n) {
        const u64 base = o_e[r] + o_i[r];
        fwd_rs[r] = static_cast<u32>(base);
        o_e[r] = base;
        o_i[r] = base + c_e[r];
    }
    if (r == 0) fwd_rs[n] = static_cast<u32>(total);
}

// Row starts of a source-major list from its exclusive scan: rs[r] = o[r], rs[n] = total.
__global__ void rows_from_scan_kernel(u64 n, const u64* o, u64 total, u32* rs) {
    const u64 r = static_cast<u64>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (r < n) rs[r] = static_cast<u32>(o[r]);
    if (r == 0) rs[n] = static_cast<u32>(total);
}

__global__ void max_row_kernel(const u32* rs, u32 n, unsigned* mx) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) atomicMax(mx, rs[i + 1] - rs[i]);
}

// ---------------------------------------------------------------- host helpers
Status exclusive_scan_u64(const u64* in, u64* out, u64 n, cudaStream_t st) {
    size_t bytes = 0;
    AS_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, bytes, in, out, n, st));
    DevBuf<unsigned char> tmp;
    AS_TRY(tmp.alloc(bytes));
    AS_CUDA(cub::DeviceScan::ExclusiveSum(tmp.get(), bytes, in, out, n, st));
    return Status::Ok();
}

template <typename T>
Status to_host(T* dst, const T* src, size_t n, cudaStream_t st) {
    AS_CUDA(cudaMemcpyAsync(dst, src, n * sizeof(T), cudaMemcpyDeviceToHost, st));
    AS_CUDA(cudaStreamSynchronize(st));
    return Status::Ok();
}

Status read_err(const DevBuf<int>& err, int* out, cudaStream_t st) { return to_host(out, err.get(), 1, st); }

// A first guess of the pools' start offsets: prefix[q] = the extra draws of the
// pools before post q.  Pool q starts at c0 + take * q + prefix[q], and only the
// positions where a pool would need redraws matter -- about 250 of the 5 nN at any
// size (a duplicate among 5 picks from nA = N / 5 astrocytes).  They are found in
// one pass; walking them in order on the host with the running shift gives the
// offsets.  The fixed-point loop that follows checks the guess (one round when it
// is right, as it always is unless the list overflowed).
Status guess_pool_prefix(u64 seed, u32 nN, u32 nA, u32 take, u64 c0, u64* prefix, cudaStream_t st) {
    if (nN == 0 || take < kPoolSize || static_cast<u64>(take) * 4 >= nA) return Status::Ok();  // no redraws
    // the positions past the last pool's nominal start: about 4x the expected extra
    // draws (a pool redraws with probability about 10 / nA)
    const u64 margin = 4096 + static_cast<u64>(static_cast<double>(nN) * 40.0 / nA);
    const u64 n = static_cast<u64>(take) * nN + margin;
    const unsigned cap = 1u << 16;
    DevBuf<PoolRedraw> list;
    DevBuf<unsigned> count;
    AS_TRY(list.alloc(cap));
    AS_TRY(count.alloc_zero(1, st));
    pool_redraw_kernel<<<sm_count() * 8, 256, 0, st>>>(seed, nA, take, c0, n, list.get(), count.get(), cap);
    AS_CUDA(cudaGetLastError());
    unsigned m = 0;
    AS_TRY(to_host(&m, count.get(), 1, st));
    if (m > cap) return Status::Ok();  // leave the zero guess to the loop
    std::vector<PoolRedraw> h(m);
    if (m) AS_TRY(to_host(h.data(), list.get(), m, st));
    std::vector<PoolRedrawAt> sorted(m);
    for (unsigned i = 0; i < m; ++i) sorted[i] = PoolRedrawAt{h[i].t, h[i].extra};
    std::sort(sorted.begin(), sorted.end(), [](const PoolRedrawAt& a, const PoolRedrawAt& b) { return a.t < b.t; });
    std::vector<u32> bq, be;
    pools_with_redraws(sorted, c0, take, nN, bq, be);
    if (bq.empty()) return Status::Ok();
    DevBuf<u64> extra;
    DevBuf<u32> dq, de;
    AS_TRY(extra.alloc_zero(nN, st));
    AS_TRY(dq.alloc(bq.size()));
    AS_TRY(de.alloc(be.size()));
    AS_CUDA(cudaMemcpyAsync(dq.get(), bq.data(), bq.size() * sizeof(u32), cudaMemcpyHostToDevice, st));
    AS_CUDA(cudaMemcpyAsync(de.get(), be.data(), be.size() * sizeof(u32), cudaMemcpyHostToDevice, st));
    scatter_extra_kernel<<<ceil_div(bq.size(), 256), 256, 0, st>>>(dq.get(), de.get(), static_cast<u32>(bq.size()),
                                                                   extra.get());
    AS_CUDA(cudaGetLastError());
    AS_TRY(exclusive_scan_u64(extra.get(), prefix, nN, st));
    AS_CUDA(cudaStreamSynchronize(st));  // bq / be are host vectors
    return Status::Ok();
}

// Lets the kernels below use more than 48 KB of shared memory, once per device.
Status allow_large_shared() {
    static std::atomic<bool> done[64];
    int dev = 0;
    AS_CUDA(cudaGetDevice(&dev));
    if (dev < 64 && done[dev].load()) return Status::Ok();
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    AS_CUDA(cudaFuncSetAttribute(pre_length_kernel, attr, static_cast<int>(kLenShared)));
    AS_CUDA(cudaFuncSetAttribute(replay_kernel, attr, static_cast<int>(kReplayShared)));
    if (dev < 64) done[dev].store(true);
    return Status::Ok();
}

// Several arrays in one allocation: a build makes hundreds of small ones otherwise, and
// concurrent builds queue for the allocator.
class Arena {
public:
    template <typename T>
    void want(T** p, u64 n) {
        slots_.push_back(Slot{reinterpret_cast<void**>(p), bytes_});
        bytes_ += (n * sizeof(T) + 255) / 256 * 256;
    }
    Status alloc() {
        AS_TRY(buf_.alloc(bytes_));
        for (const Slot& s : slots_) *s.p = buf_.get() + s.at;
        return Status::Ok();
    }

private:
    struct Slot {
        void** p;
        size_t at;
    };
    std::vector<Slot> slots_;
    size_t bytes_ = 0;
    DevBuf<unsigned char> buf_;
};

struct SectionPlan {
    const char* name;
    u32 post_count, post_off;
    int third;
    u64 n_pres;
    double draws_per_pre;
    u32 delta;
    int self_mode;  // 0: no autapse possible; 1: autapse at post == r + self_off
    u32 self_off;
    bool autapse_shifts_stream;
};

// What the host reads back after a section's passes.
struct SectionResult {
    int err;
    u32 end_group;
    u64 end;
    unsigned n_hazards;
    u32 pad_;
    Replay replay;
};

// Finds the start of every pre of one section (steps 3 and 4 of the file comment).
// On success `orbit` holds n_pres starts and *end the tape position after the section.
// All passes are enqueued before the one read-back.
Status section_orbit(const SectionPlan& P, Sec s, u64 start, DevBuf<u64>& orbit, u64* end, cudaStream_t st) {
    u32 chunk_len = kChunkLen, delta = P.delta;
    {
        const double draws = static_cast<double>(P.n_pres) * P.draws_per_pre;
        while (chunk_len > kMinChunkLen && draws / chunk_len < target_chunks()) chunk_len /= 2;
    }
    double slack = 1.04;
    int K = 32;
    constexpr u32 kPieces = 65536;
    AS_TRY(allow_large_shared());
    PhaseClock pc(st);
    for (int attempt = 0; attempt < 8; ++attempt) {
        const u64 margin = P.autapse_shifts_stream ? static_cast<u64>(K) + 16 : 0;
        const u64 target = P.n_pres + margin;
        const double est = static_cast<double>(target) * P.draws_per_pre * slack + 8.0 * chunk_len;
        const u32 n_chunks = std::max<u32>(1, static_cast<u32>(est / chunk_len) + 1);
        // groups of about the square root: the compositions follow a group's chunks, then the groups
        u32 group = 8;
        while (group < 64 && group * group < n_chunks) group *= 2;
        const u32 n_groups = ceil_div(n_chunks, group);
        const u64 n_lens = static_cast<u64>(n_chunks) * chunk_len;
        const unsigned hz_cap =
            P.autapse_shifts_stream ? static_cast<unsigned>(std::min<double>(4e6, 200.0 * (2 * K + 1) + 4096)) : 0;
        Arena mem;
        u16* lens = nullptr;
        u64 *t_exit = nullptr, *g_exit = nullptr, *g_cnt = nullptr, *g_entry = nullptr, *g_g0 = nullptr,
            *c_entry = nullptr, *c_g0 = nullptr, *forbit = nullptr, *starts = nullptr;
        u32* t_cnt = nullptr;
        Hazard* hz = nullptr;
        OrbitPiece* pieces = nullptr;
        SectionResult* res = nullptr;
        mem.want(&lens, n_lens);
        mem.want(&t_exit, static_cast<u64>(n_chunks) * delta);
        mem.want(&t_cnt, static_cast<u64>(n_chunks) * delta);
        mem.want(&g_exit, static_cast<u64>(n_groups) * delta);
        mem.want(&g_cnt, static_cast<u64>(n_groups) * delta);
        mem.want(&g_entry, n_groups);
        mem.want(&g_g0, n_groups);
        mem.want(&c_entry, n_chunks);
        mem.want(&c_g0, n_chunks);
        mem.want(&res, 1);
        if (P.autapse_shifts_stream) {
            mem.want(&forbit, target);
            mem.want(&hz, hz_cap);
            mem.want(&starts, P.n_pres + kReplayBatch);
            mem.want(&pieces, kPieces);
        }
        AS_TRY(mem.alloc());
        AS_TRY(orbit.alloc(P.n_pres));
        AS_CUDA(cudaMemsetAsync(res, 0, sizeof(SectionResult), st));
        s.err = &res->err;
        u64* const table_orbit = P.autapse_shifts_stream ? forbit : orbit.get();
        pre_length_kernel<<<ceil_div(n_lens, kLenTile), kLenBlock, kLenShared, st>>>(s, start, n_lens, lens);
        AS_CUDA(cudaGetLastError());
        table_kernel<<<n_chunks, delta, chunk_len * sizeof(u16), st>>>(s, lens, start, chunk_len, delta, t_exit, t_cnt);
        AS_CUDA(cudaGetLastError());
        group_compose_kernel<<<n_groups, delta, 0, st>>>(s, start, chunk_len, delta, n_chunks, group, t_exit, t_cnt,
                                                         g_exit, g_cnt);
        AS_CUDA(cudaGetLastError());
        top_compose_kernel<<<1, 1, 0, st>>>(s, start, chunk_len, delta, n_groups, group, g_exit, g_cnt, target, g_entry,
                                            g_g0, &res->end_group);
        AS_CUDA(cudaGetLastError());
        chunk_entry_kernel<<<ceil_div(n_groups, 32), 32, 0, st>>>(s, start, chunk_len, delta, n_chunks, n_groups, group,
                                                                  t_exit, t_cnt, g_entry, g_g0, &res->end_group,
                                                                  c_entry, c_g0);
        AS_CUDA(cudaGetLastError());
        materialize_kernel<<<n_chunks, 128, chunk_len * sizeof(u16), st>>>(s, lens, start, chunk_len, n_chunks, c_entry,
                                                                           c_g0, target, P.n_pres - 1, table_orbit,
                                                                           &res->end);
        AS_CUDA(cudaGetLastError());
        if (P.autapse_shifts_stream) {
            hazard_kernel<<<ceil_div(target, 128), 128, 0, st>>>(s, table_orbit, target, K, hz, &res->n_hazards, hz_cap,
                                                                 &res->end_group, n_groups);
            AS_CUDA(cudaGetLastError());
            replay_kernel<<<1, kReplayBlock, kReplayShared, st>>>(s, lens, start, n_lens, hz, &res->n_hazards, hz_cap,
                                                                  table_orbit, target, P.n_pres, K, &res->end_group,
                                                                  n_groups, starts, pieces, kPieces, &res->replay);
            AS_CUDA(cudaGetLastError());
            splice_orbit_kernel<<<ceil_div(P.n_pres, 256), 256, 0, st>>>(pieces, &res->replay, P.n_pres, orbit.get());
            AS_CUDA(cudaGetLastError());
        }
        SectionResult h{};
        AS_TRY(to_host(&h, res, 1, st));
        pc.mark("  lengths, tables, orbit");
        if (h.err & kErrDelta) {
            if (delta >= kMaxDelta) return make_error(ASTROSIM_ERR_UNSUPPORTED, "%s: a pre longer than %u draws", P.name, kMaxDelta);
            delta = std::min<u32>(kMaxDelta, delta * 2);
            continue;
        }
        if (h.err & kErrCache) return make_error(ASTROSIM_ERR_UNSUPPORTED, "%s walk left the draw cache", P.name);
        if (h.end_group >= n_groups) { slack *= 1.25; continue; }
        if (h.err) return make_error(ASTROSIM_ERR_CUDA, "%s orbit materialisation failed (flags %d)", P.name, h.err);
        if (!P.autapse_shifts_stream) {
            *end = h.end;
            return Status::Ok();
        }
        if (h.n_hazards > hz_cap)
            return make_error(ASTROSIM_ERR_UNSUPPORTED, "%s: %u autapse hazards exceed the buffer", P.name, h.n_hazards);
        if (h.replay.full) return make_error(ASTROSIM_ERR_UNSUPPORTED, "%s: more than %u orbit pieces", P.name, kPieces);
        if (h.replay.retry) { K *= 4; slack *= 1.05; continue; }
        *end = h.replay.end;
        return Status::Ok();
    }
    return make_error(ASTROSIM_ERR_CUDA, "%s: chunked walk did not settle", P.name);
}

}  // namespace

Status build_parallel(const Sizes& sz, u64 seed, u64 c0, Network& net, cudaStream_t st) {
    if (sz.p >= 1.0 || sz.n_astro <= 20)
        return build_sequential(sz, seed, c0, net, st);  // all-to-all networks are tiny
    const u32 nN = sz.n_neurons, nA = sz.n_astro;
    const u32 take = nA < kPoolSize ? nA : kPoolSize;
    PhaseClock pc(st);
    DevBuf<int> err;
    AS_TRY(err.alloc_zero(1, st));

    // ---- 1. pools
    DevBuf<u32> pool;
    DevBuf<u64> extra, prefix, prefix_new;
    DevBuf<int> flag;
    AS_TRY(pool.alloc(static_cast<u64>(nN) * kPoolSize));
    AS_TRY(extra.alloc(nN));
    AS_TRY(prefix.alloc_zero(nN, st));
    AS_TRY(guess_pool_prefix(seed, nN, nA, take, c0, prefix.get(), st));
    AS_TRY(prefix_new.alloc(nN));
    AS_TRY(flag.alloc(1));
    u64 pools_end = 0;
    for (int it = 0;; ++it) {
        if (it > 100000) return make_error(ASTROSIM_ERR_CUDA, "pool offsets did not converge");
        pool_pass_kernel<<<ceil_div(nN, 256), 256, 0, st>>>(seed, nN, nA, take, c0, prefix.get(), pool.get(),
                                                            extra.get());
        AS_CUDA(cudaGetLastError());
        AS_TRY(exclusive_scan_u64(extra.get(), prefix_new.get(), nN, st));
        AS_CUDA(cudaMemsetAsync(flag.get(), 0, sizeof(int), st));
        diff_kernel<<<ceil_div(nN, 256), 256, 0, st>>>(prefix.get(), prefix_new.get(), nN, flag.get());
        AS_CUDA(cudaGetLastError());
        int changed = 0;
        AS_TRY(to_host(&changed, flag.get(), 1, st));
        if (!changed) {
            u64 last_prefix = 0, last_extra = 0;
            AS_TRY(to_host(&last_prefix, prefix.get() + (nN - 1), 1, st));
            AS_TRY(to_host(&last_extra, extra.get() + (nN - 1), 1, st));
            pools_end = c0 + static_cast<u64>(take) * nN + last_prefix + last_extra;
            break;
        }
        std::swap(prefix, prefix_new);
    }
    extra.release();
    prefix.release();
    prefix_new.release();
    pc.mark("pools");

    // ---- 2. draw cache over every tape position the three sections can reach
    if (nN >= kSkipMax) return make_error(ASTROSIM_ERR_OUT_OF_MEMORY, "%u neurons need a draw cache of over 100 GB", nN);
    const double ne = sz.n_exc, ni = sz.n_inh, nn = nN, p = sz.p;
    SectionPlan plans[3] = {
        {"E block", sz.n_exc, 0, 1, sz.n_exc, 1.0 + p * ne * (2.0 + kPThird), 384, 1, 0, true},
        {"I block", sz.n_inh, sz.n_exc, 1, sz.n_exc, 1.0 + p * ni * (2.0 + kPThird), 192, 0, 0, false},
        {"inhibitory", nN, 0, 0, sz.n_inh, 1.0 + p * nn, 192, 1, sz.n_exc, false},
    };
    double est_total = 0.0;
    for (const auto& P : plans) est_total += static_cast<double>(P.n_pres) * P.draws_per_pre;
    const u64 cache_len = static_cast<u64>(est_total * 1.12) + 64ull * 65536 + 1000000;
    DevBuf<u32> cache;
    AS_TRY(cache.alloc(cache_len));
    const double L = std::log1p(-p);  // host value, as the reference computes it (src/astrosim_fused.cu:622)
    {
        DevBuf<u64> amb_pos;
        DevBuf<double> amb_val;
        DevBuf<unsigned> amb_n;
        const unsigned amb_cap = 1u << 16;
        AS_TRY(amb_pos.alloc(amb_cap));
        AS_TRY(amb_val.alloc(amb_cap));
        AS_TRY(amb_n.alloc_zero(1, st));
        AmbiguityLog amb{amb_pos.get(), amb_val.get(), amb_n.get(), amb_cap};
        draw_cache_kernel<<<sm_count() * 16, 256, 0, st>>>(seed, L, pools_end, cache_len, take, cache.get(), amb);
        AS_CUDA(cudaGetLastError());
        unsigned n_amb = 0;
        AS_TRY(to_host(&n_amb, amb_n.get(), 1, st));
        if (n_amb > amb_cap) return make_error(ASTROSIM_ERR_UNSUPPORTED, "too many ambiguous skip draws");
        std::vector<u64> pos(n_amb);
        if (n_amb) AS_TRY(to_host(pos.data(), amb_pos.get(), n_amb, st));
        for (u64 t : pos) {  // settle with the host formula
            const u32 v = draw_word(rng_bits(seed, kSetupStream, t) >> 11, skip_value_host(seed, L, t), take);
            AS_CUDA(cudaMemcpyAsync(cache.get() + (t - pools_end), &v, sizeof(u32), cudaMemcpyHostToDevice, st));
            AS_CUDA(cudaStreamSynchronize(st));
        }
    }

    pc.mark("draw cache");
    // ---- 3-4. every pre's start, section by section
    Sec s{};
    s.seed = seed;
    s.cache = cache.get();
    s.cache_base = pools_end;
    s.cache_len = cache_len;
    s.err = err.get();
    s.take = take;
    s.pool = pool.get();
    DevBuf<u64> orbits[3];
    u64 start = pools_end;
    for (int k = 0; k < 3; ++k) {
        s.post_count = plans[k].post_count;
        s.post_off = plans[k].post_off;
        s.third = plans[k].third;
        u64 end = 0;
        AS_TRY(section_orbit(plans[k], s, start, orbits[k], &end, st));
        start = end;
        pc.mark(plans[k].name);
    }

    // ---- 5. count, scan, emit (only the edges whose target this network owns)
    const Owned own{net.own.n_lo, net.own.n_hi, net.own.a_lo, net.own.a_hi};
    DevBuf<u64> oe[3], oa[3], os[3];
    DevBuf<unsigned long long> totals;
    AS_TRY(totals.alloc_zero(6, st));
    u64 tot_e[3] = {0, 0, 0}, tot_a[3] = {0, 0, 0}, tot_s[3] = {0, 0, 0};
    DevBuf<u64> ce_block0;  // the E block's per-pre primary counts (the exc layout needs them)
    for (int k = 0; k < 3; ++k) {
        const SectionPlan& P = plans[k];
        s.post_count = P.post_count;
        s.post_off = P.post_off;
        s.third = P.third;
        DevBuf<u64> ce, ca, cs;
        AS_TRY(ce.alloc(P.n_pres));
        AS_TRY(ca.alloc(P.n_pres));
        AS_TRY(cs.alloc(P.n_pres));
        AS_TRY(oe[k].alloc(P.n_pres));
        AS_TRY(oa[k].alloc(P.n_pres));
        AS_TRY(os[k].alloc(P.n_pres));
        count_kernel<<<ceil_div(P.n_pres, 128), 128, 0, st>>>(s, orbits[k].get(), P.n_pres, P.self_mode, P.self_off,
                                                             own, ce.get(), ca.get(), cs.get(),
                                                             totals.get() + 2 * k);
        AS_CUDA(cudaGetLastError());
        AS_TRY(exclusive_scan_u64(ce.get(), oe[k].get(), P.n_pres, st));
        AS_TRY(exclusive_scan_u64(ca.get(), oa[k].get(), P.n_pres, st));
        AS_TRY(exclusive_scan_u64(cs.get(), os[k].get(), P.n_pres, st));
        u64 h[6] = {0, 0, 0, 0, 0, 0};
        AS_TRY(to_host(&h[0], oe[k].get() + (P.n_pres - 1), 1, st));
        AS_TRY(to_host(&h[1], ce.get() + (P.n_pres - 1), 1, st));
        AS_TRY(to_host(&h[2], oa[k].get() + (P.n_pres - 1), 1, st));
        AS_TRY(to_host(&h[3], ca.get() + (P.n_pres - 1), 1, st));
        AS_TRY(to_host(&h[4], os[k].get() + (P.n_pres - 1), 1, st));
        AS_TRY(to_host(&h[5], cs.get() + (P.n_pres - 1), 1, st));
        tot_e[k] = h[0] + h[1];
        tot_a[k] = h[2] + h[3];
        tot_s[k] = h[4] + h[5];
        if (k == 0) ce_block0 = std::move(ce);
    }
    // Both excitatory blocks walk the same pres (the exc neurons), so their edges can
    // be laid out source-major: the list is then the forward exc list itself, and the
    // target CSR (a stable sort by target) is unchanged, since each target row's
    // sources all come from one block, in ascending pre order either way.  The
    // inhibitory section's emission order is already source-major.
    if (plans[0].n_pres != plans[1].n_pres)
        return make_error(ASTROSIM_ERR_CUDA, "excitatory blocks over different pres (%llu, %llu)",
                          static_cast<unsigned long long>(plans[0].n_pres),
                          static_cast<unsigned long long>(plans[1].n_pres));
    if (tot_e[0] + tot_e[1] >= (1ull << 32) || tot_e[2] >= (1ull << 32))
        return make_error(ASTROSIM_ERR_UNSUPPORTED, "more than 2^32 - 1 primary edges in one CSR");
    DevBuf<u32> fwd_exc_rs, fwd_inh_rs;
    AS_TRY(fwd_exc_rs.alloc(plans[0].n_pres + 1));
    AS_TRY(fwd_inh_rs.alloc(plans[2].n_pres + 1));
    exc_layout_kernel<<<ceil_div(std::max<u64>(1, plans[0].n_pres), 256), 256, 0, st>>>(
        plans[0].n_pres, oe[0].get(), oe[1].get(), ce_block0.get(), tot_e[0] + tot_e[1], fwd_exc_rs.get());
    AS_CUDA(cudaGetLastError());
    rows_from_scan_kernel<<<ceil_div(std::max<u64>(1, plans[2].n_pres), 256), 256, 0, st>>>(
        plans[2].n_pres, oe[2].get(), tot_e[2], fwd_inh_rs.get());
    AS_CUDA(cudaGetLastError());
    ce_block0.release();
    {
        unsigned long long t[6];
        AS_TRY(to_host(t, totals.get(), 6, st));
        net.total_edges[0] = t[0] + t[2];  // excitatory primary edges: sections 0 and 1
        net.total_edges[1] = t[4];         // inhibitory: section 2
        net.total_edges[2] = t[1] + t[3];  // third-factor pairs: one e2a and one sic edge each
        net.total_edges[3] = t[1] + t[3];
    }
    EdgeStorage es;
    es.cap_exc = tot_e[0] + tot_e[1];
    es.cap_inh = tot_e[2];
    const u64 cap_e2a = tot_a[0] + tot_a[1], cap_sic = tot_s[0] + tot_s[1];
    AS_TRY(es.exc_src.alloc(es.cap_exc));
    AS_TRY(es.exc_dst.alloc(es.cap_exc));
    AS_TRY(es.inh_src.alloc(es.cap_inh));
    AS_TRY(es.inh_dst.alloc(es.cap_inh));
    AS_TRY(es.e2a_src.alloc(cap_e2a));
    AS_TRY(es.e2a_dst.alloc(cap_e2a));
    AS_TRY(es.sic_src.alloc(cap_sic));
    AS_TRY(es.sic_dst.alloc(cap_sic));
    AS_TRY(es.counts.alloc_zero(4, st));
    for (int k = 0; k < 3; ++k) {
        const SectionPlan& P = plans[k];
        s.post_count = P.post_count;
        s.post_off = P.post_off;
        s.third = P.third;
        const u64 base_e = 0, base_a = k == 1 ? tot_a[0] : 0, base_s = k == 1 ? tot_s[0] : 0;
        u32* e_dst = k == 2 ? es.inh_dst.get() : es.exc_dst.get();
        emit_kernel<<<ceil_div(P.n_pres, kEmitBlock), kEmitBlock, 0, st>>>(
            s, orbits[k].get(), P.n_pres, P.self_mode, P.self_off, own, oe[k].get(), oa[k].get(), os[k].get(),
            base_e, base_a, base_s, e_dst, es.e2a_dst.get(), es.sic_src.get(), es.sic_dst.get());
        AS_CUDA(cudaGetLastError());
    }
    // the pre-index sources: exc (both blocks, source-major), inh, and e2a (E block, then I block)
    const auto fill = [&](const DevBuf<u64>& o, u64 n, u64 base, u64 total, u32* out) -> Status {
        if (n == 0 || total == 0) return Status::Ok();
        fill_rows_kernel<<<ceil_div(n * 32, 256), 256, 0, st>>>(o.get(), n, base, total, out);
        AS_CUDA(cudaGetLastError());
        return Status::Ok();
    };
    AS_TRY(fill(oe[0], plans[0].n_pres, 0, tot_e[0] + tot_e[1], es.exc_src.get()));
    AS_TRY(fill(oe[2], plans[2].n_pres, 0, tot_e[2], es.inh_src.get()));
    AS_TRY(fill(oa[0], plans[0].n_pres, 0, tot_a[0], es.e2a_src.get()));
    AS_TRY(fill(oa[1], plans[1].n_pres, tot_a[0], tot_a[1], es.e2a_src.get()));
    int herr = 0;
    AS_TRY(read_err(err, &herr, st));
    if (herr) return make_error(ASTROSIM_ERR_CUDA, "edge emission failed (flags %d)", herr);
    for (int k = 0; k < 3; ++k) {
        orbits[k].release();
        oe[k].release();
        oa[k].release();
        os[k].release();
    }
    cache.release();
    pool.release();
    pc.mark("count + emit");
    const u64 counts[4] = {es.cap_exc, es.cap_inh, cap_e2a, cap_sic};
    AS_TRY(edge_lists_to_network(es.view(), counts, net, st));
    net.fwd_exc_rs = std::move(fwd_exc_rs);
    net.fwd_exc_dst = std::move(es.exc_dst);
    net.fwd_inh_rs = std::move(fwd_inh_rs);
    net.fwd_inh_dst = std::move(es.inh_dst);
    net.has_fwd = true;
    pc.mark("CSR sort");

    // The astrocyte out-degree cap (src/astrosim_fused.cu:702) drops a third-factor
    // edge only once an astrocyte already has 10000; with at most 10000 candidates
    // per astrocyte it never fires and the lists above are exact.
    DevBuf<unsigned> mx;
    AS_TRY(mx.alloc_zero(1, st));
    const u32 own_astro = net.own.a_hi - net.own.a_lo;  // each rank checks its own astrocytes
    if (own_astro)
        max_row_kernel<<<ceil_div(own_astro, 256), 256, 0, st>>>(net.e2a.row_start.get(), own_astro, mx.get());
    AS_CUDA(cudaGetLastError());
    unsigned hmx = 0;
    AS_TRY(to_host(&hmx, mx.get(), 1, st));
    if (hmx > kMaxAstroOutDegree)
        return make_error(ASTROSIM_ERR_UNSUPPORTED,
                          "an astrocyte has %u third-factor candidates; the out-degree cap of %u would bind", hmx,
                          kMaxAstroOutDegree);
    return Status::Ok();
}

}  // namespace astrosim
