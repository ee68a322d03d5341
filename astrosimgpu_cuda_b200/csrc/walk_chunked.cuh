// walk_chunked.cuh -- one pre's walk over its postsynaptic block for the chunked
// parallel builder (builder_parallel.cu), on the precomputed draw cache.
//
// Every draw of the walks is a function of its tape position alone: the skip it would
// give, whether it passes the third-factor test and which pool entry it would pick.  The
// cache holds all three in one word per position, so a walk is a chain of cached words
// and needs no hashing: a landing costs one load latency instead of a load after a dependent
// hash.  And because where a pre that starts at a position ends is then a function of that
// position alone (but for its autapse), the lengths of the pres at all positions are
// computed in parallel, and walking pre after pre is one table read per pre.
//
// Device code, also compiled on the host by CPU tests (tests/walk_equivalence.cpp,
// tests/walk_words.cpp) that supply __ldg and atomicOr.
#pragma once

#include "model.cuh"

namespace astrosim {

constexpr u32 kNoSelf = 0xFFFFFFFFu;  // no autapse rule for this walk

enum ErrBits : int {
    kErrCache = 1,     // a walk left the draw cache
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

// ------------------------------------------------------------------ pre lengths
// How many draws a pre takes that starts at a tape position, for every position.  A walk
// of a pre moves on by landings, and where a landing at a position leads does not depend
// on how the walk got there; so the landings are first joined into jumps of 4 and of 16
// (their posts passed and draws taken added up), and a pre is then a few jumps that stay
// inside its block and the last landings one by one: about 8 steps instead of 68.
constexpr u32 kMaxPre = 512;         // the longest pre, in draws (E block: 178 on average)
constexpr u32 kLongPre = 0xFFFF;     // a longer one
constexpr u32 kJumpFull = (1u << 26) - 1;  // posts of a jump that passes more than fit

// posts << 6 | draws
__host__ __device__ __forceinline__ u32 landing_jump(const Sec& s, u32 skip_word, u32 test_word) {
    const u32 g = skip_word & kSkipMax;
    const u32 posts = g >= kJumpFull ? kJumpFull : g + 1;
    return posts << 6 | (s.third ? ((test_word & kHitBit) ? 3u : 2u) : 1u);
}
__host__ __device__ __forceinline__ u32 join_jumps(u32 a, u32 b) {
    const u32 posts = (a >> 6) + (b >> 6);
    return (posts < kJumpFull ? posts : kJumpFull) << 6 | ((a & 63u) + (b & 63u));
}
// Four landings from index i of `words`.
__host__ __device__ __forceinline__ u32 jump4(const Sec& s, const u32* words, u32 i) {
    u32 j = 0;
    for (int k = 0; k < 4; ++k) j = join_jumps(j, landing_jump(s, words[i + (j & 63u)], words[i + (j & 63u) + 1]));
    return j;
}
// Sixteen, from the jumps of four.
__host__ __device__ __forceinline__ u32 jump16(const u32* jumps4, u32 i) {
    u32 j = 0;
    for (int k = 0; k < 4; ++k) j = join_jumps(j, jumps4[i + (j & 63u)]);
    return j;
}
// The draws of the pre that starts at index i (kLongPre: more than kMaxPre).
__host__ __device__ __forceinline__ u32 pre_length(const Sec& s, const u32* words, const u32* jumps4,
                                                   const u32* jumps16, u32 i) {
    u32 at = i, left = s.post_count;
    for (u32 j = jumps16[at]; (j >> 6) < left && (j >> 6) != kJumpFull; j = jumps16[at]) {
        left -= j >> 6;
        at += j & 63u;
        if (at - i > kMaxPre) return kLongPre;
    }
    for (u32 j = jumps4[at]; (j >> 6) < left && (j >> 6) != kJumpFull; j = jumps4[at]) {
        left -= j >> 6;
        at += j & 63u;
        if (at - i > kMaxPre) return kLongPre;
    }
    while (at - i <= kMaxPre) {
        const u32 g = words[at] & kSkipMax;
        if (g >= left) {  // the skip reaches the end of the block
            ++at;
            break;
        }
        left -= g + 1;
        at += landing_jump(s, words[at], words[at + 1]) & 63u;
        if (left == 0) break;
    }
    return at - i > kMaxPre ? kLongPre : at - i;
}
// Words that pre_length may read past index i, and those its jumps start at.
constexpr u32 kWordsAhead = kMaxPre + 64, kJumpsAhead = kMaxPre + 48;

}  // namespace astrosim
