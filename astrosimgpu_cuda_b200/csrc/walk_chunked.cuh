// walk_chunked.cuh -- one pre's walk over its postsynaptic block for the chunked
// parallel builder (builder_parallel.cu), on the precomputed draw cache.
//
// Every draw of the walks is a function of its tape position alone: the skip it would
// give, whether it passes the third-factor test and which pool entry it would pick.  The
// cache holds all three in one word per position, so a walk is a chain of cached words
// and needs no hashing: a landing costs one load latency instead of a load after a dependent
// hash (one thread walking one pre after the other: 260 ns per landing with hashes).
//
// Device code, also compiled on the host by CPU tests (tests/walk_equivalence.cpp,
// tests/walk_words.cpp) that supply __ldg and atomicOr.
#pragma once

#include "model.cuh"

namespace astrosim {

constexpr u32 kNoSelf = 0xFFFFFFFFu;  // no autapse rule for this walk

enum ErrBits : int {
    kErrCache = 1,     // a walk left the skip cache
    kErrHash = 2,      // claim table full
    kErrDelta = 4,     // an entry fell outside the candidate window
    kErrOrbit = 8      // materialised chunk did not meet its successor (internal)
};

struct Sec {
    u64 seed;
    const u32* cache;
    u64 cache_base, cache_len;
    int* err;
    u32 post_count, post_off;
    int third;
    u32 take;
    const u32* pool;
};

// A cached draw: its skip (kSkipMax and longer ones alike, past every block's end), the
// pool entry it would pick and its third-factor test.
constexpr u32 kSkipMax = (1u << 28) - 1;
constexpr u32 kPickShift = 28, kPickMask = 7;  // kPoolSize picks
constexpr u32 kHitBit = 1u << 31;

// The third-factor test u < P_THIRD (src/astrosim_fused.cu:699) on the 53-bit integer m
// of u = m * 2^-53: u < P_THIRD exactly when m < kThirdLim = ceil(P_THIRD * 2^53)
// (the product is exact, a power-of-two scaling).
constexpr double kThirdScaled = kPThird * 9007199254740992.0;
constexpr u64 kThirdLim = static_cast<u64>(kThirdScaled) +
                          (static_cast<double>(static_cast<u64>(kThirdScaled)) < kThirdScaled ? 1u : 0u);

// The word of the draw with 53-bit integer m, given its skip.
__host__ __device__ __forceinline__ u32 draw_word(u64 m, double skip, u32 take) {
    const u32 g = skip >= static_cast<double>(kSkipMax) ? kSkipMax : static_cast<u32>(skip);
    const double u = static_cast<double>(m) * (1.0 / 9007199254740992.0);
    const u32 pick = take ? static_cast<u32>(static_cast<u64>(u * static_cast<double>(take)) % take) : 0;
    return g | pick << kPickShift | (m < kThirdLim ? kHitBit : 0u);
}

// The word at tape position t, loaded ahead of knowing whether the walk draws it
// (no error flag: the walk checks the positions it draws).
__device__ __forceinline__ u32 peek(const Sec& s, u64 t) {
    const u64 i = t - s.cache_base;
    return i < s.cache_len ? __ldg(s.cache + i) : 0xFFFFFFFFu;
}

struct NoVisit {
    __device__ __forceinline__ void operator()(u32, bool, u32) const {}
};

// One pre's walk from tape position c (src/astrosim_fused.cu:688-707, 712-723).
// A landing on `self_post` is an autapse: no edge and no third-factor draws.
// Returns the tape position after the walk; a walk that draws past the cache flags
// kErrCache and stops.  The draws and their order are the reference's.  The words that
// the next landing may need are loaded before this landing's test is looked at (a miss
// moves the next test two positions on, a hit three), so the loads overlap the chain.
template <class V>
__device__ __forceinline__ u64 walk_pre(const Sec& s, u64 c, u32 self_post, V& visit) {
    u32 pos = 0;
    const u32 n = s.post_count;
    if (n == 0) return c;
    const u64 end = s.cache_base + s.cache_len;
    u32 skip = peek(s, c);
    u32 w0 = peek(s, c + 1), w1 = peek(s, c + 2), w2 = peek(s, c + 3);
    ++c;  // the position after the skip: w0's
    for (;;) {
        if (c > end) {
            atomicOr(s.err, kErrCache);
            break;
        }
        const u32 g = skip & kSkipMax;
        if (g >= n - pos) break;  // the skip reaches the end of the block
        pos += g;
        const u32 post = s.post_off + pos;
        ++pos;
        const bool more = pos < n;  // another skip is drawn after this post
        const u32 w3 = peek(s, c + 3);
        if (!s.third || post == self_post) {  // the next draw is a skip
            if (post != self_post) visit(post, false, 0u);
            if (!more) break;
            skip = w0;
            w0 = w1;
            w1 = w2;
            w2 = w3;
            ++c;
        } else {
            const u32 w4 = peek(s, c + 4), w5 = peek(s, c + 5);
            const bool hit = (w0 & kHitBit) != 0;
            u32 astro = 0;
            if (hit) astro = s.pool[static_cast<u64>(post) * kPoolSize + ((w1 >> kPickShift) & kPickMask)];
            c += hit ? 2 : 1;  // the test, and the pool pick after a hit
            if (c > end) {
                atomicOr(s.err, kErrCache);
                break;
            }
            visit(post, hit, astro);
            if (!more) break;
            skip = hit ? w2 : w1;
            w0 = hit ? w3 : w2;
            w1 = hit ? w4 : w3;
            w2 = hit ? w5 : w4;
            ++c;
        }
    }
    return c;
}

// walk_pre for a walk that only needs the tape position it ends at.
__device__ __forceinline__ u64 walk_pre_end(const Sec& s, u64 c, u32 self_post) {
    NoVisit nv;
    return walk_pre(s, c, self_post, nv);
}

// A stretch of consecutive pres as a machine that makes one landing per step, pre ends
// included: the lanes of a warp then stay together whatever their pres' lengths.  It holds
// the words around its place, so that a step is a short chain of selections; the words
// that it may need next are read behind it.  `at` is the cache index after the current
// skip's, less `origin`.  It draws exactly what walk_pre draws, pre after pre.
struct Stretch {
    u64 origin;
    u32 at, rem;           // rem: posts left in the current pre's block
    u32 skip, test, a1, a2, a3;  // the words at - 1, at, at + 1, at + 2, at + 3
    // From tape position c, with cache index `first` of its segment as the origin.
    __device__ __forceinline__ Stretch(const Sec& s, u64 c, u64 first)
        : origin(first), at(static_cast<u32>(c - s.cache_base - first) + 1), rem(s.post_count), skip(0), test(0), a1(0),
          a2(0), a3(0) {}
    template <class Word>
    __device__ __forceinline__ void begin(Word word) {
        skip = word(at - 1);
        test = word(at);
        a1 = word(at + 1);
        a2 = word(at + 2);
        a3 = word(at + 3);
    }
    // When a pre has just ended: the next one's start (its skip is already taken).
    __device__ __forceinline__ u64 start(const Sec& s) const { return s.cache_base + origin + at - 1; }
    // Past the cache: the current skip (a walk that goes on), or a draw before start().
    __device__ __forceinline__ bool out(const Sec& s) const { return origin + at > s.cache_len; }
    __device__ __forceinline__ bool overran(const Sec& s) const { return origin + at - 1 > s.cache_len; }
    // `self_post`: the current pre's autapse.  Returns true when the pre ended.
    template <class Word>
    __device__ __forceinline__ bool step(const Sec& s, u32 self_post, Word word) {
        const u32 g = skip & kSkipMax, n = s.post_count;
        const bool past = g >= rem;
        const bool self = s.post_off + (n - rem) + g == self_post;
        const bool tested = s.third && !past && !self;
        const bool hit = tested && (test & kHitBit);
        const u32 left = rem - g - 1;
        const bool ended = past || left == 0;
        rem = ended ? n : left;
        at += hit ? 3u : (tested ? 2u : 1u);
        skip = hit ? a2 : (tested ? a1 : test);
        test = hit ? a3 : (tested ? a2 : a1);
        a1 = word(at + 1);
        a2 = word(at + 2);
        a3 = word(at + 3);
        return ended;
    }
};

#ifdef __CUDACC__
// The tape ahead of a warp's stretches: a ring of four segments of 32 words per walking
// lane in shared memory, filled by asynchronous copies.  One thread walks one stretch of
// the tape after another; reading the cache directly, some lane of the warp crossed into
// a new 32-byte sector at every landing and the warp waited for it: 650 ns per landing
// from DRAM (N = 3e5), 230 ns from L2 (N = 1e3).  Every kRefill landings all lanes top
// up together (the copies of a warp are counted together, so a lane that waited for its
// own would wait for the others' newest) and copies have two more refills to arrive.
// The cache is padded past its end to whole segments (cache_words).
constexpr u32 kSegment = 32, kRingSegments = 4, kRefill = 8;
constexpr u32 kRingWords = kRingSegments * kSegment + 4;  // an odd number of 16-byte units: lanes spread over the banks
static_assert(3 * kRefill + 4 <= kSegment, "a refill of one segment keeps up with the walk");
inline __host__ __device__ u64 cache_words(u64 len) { return (len / kSegment + 2 * kRingSegments) * kSegment; }

struct TapeRing {
    u32* ring;   // this lane's kRingWords
    u64 first;   // the segment that the stretch starts in
    u32 filled;  // segments from `first` on that are in the ring or on their way
    __device__ __forceinline__ void fetch(const Sec& s) {
        const u64 g = first + filled;
        const u32 slot = filled++ & (kRingSegments - 1);
        if (g >= cache_words(s.cache_len) / kSegment) return;  // a walk that left the cache
        const u32* from = s.cache + g * kSegment;
        const u32 to = static_cast<u32>(__cvta_generic_to_shared(ring + slot * kSegment));
#pragma unroll
        for (u32 k = 0; k < kSegment / 4; ++k)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 16 * k), "l"(from + 4 * k) : "memory");
    }
    __device__ __forceinline__ TapeRing(const Sec& s, u32* shared, bool live, u64 c)
        : ring(shared), first((c - s.cache_base) / kSegment), filled(0) {
        if (live)
            for (u32 k = 0; k < kRingSegments; ++k) fetch(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    // Every lane of the warp, every kRefill landings.
    __device__ __forceinline__ void refill(const Sec& s, bool live, u32 at) {
        if (live && filled < (at - 1) / kSegment + kRingSegments) fetch(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 2;" ::: "memory");
    }
    __device__ __forceinline__ u32 word(u32 i) const { return ring[i & (kRingSegments * kSegment - 1)]; }
};

// The lane's stretch from tape position c (when live), on its ring in `shared`: on_pre(start)
// is called at every pre end with the next pre's start and says whether to go on; self()
// names the current pre's autapse.  Every lane of the warp takes part.
template <class OnPre, class Self>
__device__ __forceinline__ void walk_stretch(const Sec& s, u64 c, bool live, u32* shared, OnPre on_pre, Self self) {
    live = live && s.post_count != 0;
    if (live && c - s.cache_base >= s.cache_len) {
        atomicOr(s.err, kErrCache);
        live = false;
    }
    if (!live) c = s.cache_base;
    TapeRing ring(s, shared, live, c);
    Stretch w(s, c, ring.first * kSegment);
    auto word = [&](u32 i) { return ring.word(i); };
    if (live) w.begin(word);
    while (__any_sync(0xffffffffu, live)) {
        if (live) {
#pragma unroll
            for (u32 k = 0; k < kRefill; ++k) {
                if (w.step(s, self(), word)) {
                    if (w.overran(s)) {
                        atomicOr(s.err, kErrCache);
                        live = false;
                    } else {
                        live = on_pre(w.start(s));
                    }
                    if (!live) break;
                }
            }
            if (live && w.out(s)) {
                atomicOr(s.err, kErrCache);
                live = false;
            }
        }
        __syncwarp();
        ring.refill(s, live, w.at);
    }
}

// Walks per warp for `walks` stretches: all 32 lanes when there are warps enough for every
// scheduler, fewer otherwise, because a warp waits whenever one of its lanes ends a pre.
inline u32 walking_lanes(u64 walks, u32 schedulers) {
    u32 lanes = 32;
    while (lanes > 1 && walks * 2 / lanes <= 2ull * schedulers) lanes /= 2;
    return lanes;
}
#endif

}  // namespace astrosim
