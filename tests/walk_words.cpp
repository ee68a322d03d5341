// Host check of the builder's cached walk (astrosimgpu_cuda_b200/csrc/walk_chunked.cuh),
// compiled with g++ by test_walk_words.py: over random streams, sections and autapse
// positions, walk_pre on the cached words visits the posts, third-factor results and
// pool picks, and ends at the position, of a walk that makes every draw from the counter
// stream itself in the reference's order (src/astrosim_fused.cu:617-624, 688-723).
// The pre lengths joined from jumps are those of the same walk, at every position.
// Test infrastructure.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <random>
#include <tuple>
#include <vector>

template <class T>
inline T __ldg(const T* p) { return *p; }
inline int atomicOr(int* p, int v) {
    const int o = *p;
    *p |= v;
    return o;
}

#include "../astrosimgpu_cuda_b200/csrc/walk_chunked.cuh"

using namespace astrosim;
using Visit = std::tuple<u32, bool, u32>;

struct Record {
    std::vector<Visit>& out;
    void operator()(u32 post, bool hit, u32 astro) { out.emplace_back(post, hit, hit ? astro : 0u); }
};

static u64 plain_walk(const Sec& s, double L, u64 c, u32 self, std::vector<Visit>& out) {
    auto uniform = [&] { return rng_uniform(s.seed, kSetupStream, c++); };
    u32 pos = 0;
    while (pos < s.post_count) {
        const u32 left = s.post_count - pos;
        const double g = std::floor(std::log1p(-uniform()) / L);
        pos += g >= static_cast<double>(left) ? left : static_cast<u32>(g);
        if (pos >= s.post_count) break;
        const u32 post = s.post_off + pos;
        ++pos;
        if (post == self) continue;
        bool hit = false;
        u32 astro = 0;
        if (s.third && uniform() < kPThird) {
            hit = true;
            astro = s.pool[static_cast<u64>(post) * kPoolSize + static_cast<u64>(uniform() * s.take) % s.take];
        }
        out.emplace_back(post, hit, astro);
    }
    return c;
}

int main(int argc, char** argv) {
    const int trials = argc > 1 ? std::atoi(argv[1]) : 500;
    std::mt19937_64 rng(11);
    long walks = 0, bad = 0, overruns = 0, hits = 0, lengths = 0, longs = 0;
    for (int trial = 0; trial < trials; ++trial) {
        const u64 len = 500 + rng() % 6000;
        const double p = trial % 5 == 0 ? 1e-9 : 0.01 + static_cast<double>(rng() % 1000) / 1000.0 * 0.8;
        const double L = std::log1p(-p);
        Sec s{};
        s.seed = rng();
        s.cache_base = rng() % 100000;
        s.cache_len = len;
        s.post_count = static_cast<u32>(rng() % (trial % 3 ? 400 : 1500));
        s.post_off = static_cast<u32>(rng() % 5000);
        s.third = static_cast<int>(rng() % 4 != 0);
        s.take = 1 + static_cast<u32>(rng() % 5);
        std::vector<u32> cache(len), pool((static_cast<size_t>(s.post_off) + s.post_count + 1) * kPoolSize);
        for (auto& a : pool) a = static_cast<u32>(rng() % 100000);
        for (u64 i = 0; i < len; ++i) {
            const u64 m = rng_bits(s.seed, kSetupStream, s.cache_base + i) >> 11;
            cache[i] = draw_word(m, std::floor(std::log1p(-static_cast<double>(m) * 0x1p-53) / L), s.take);
        }
        s.cache = cache.data();
        s.pool = pool.data();
        // the lengths of the pres at every position against the plain walk's
        std::vector<u32> words(len + kWordsAhead + 64, 0xFFFFFFFFu), jumps4(len + kJumpsAhead + 48), jumps16(len + kJumpsAhead);
        std::copy(cache.begin(), cache.end(), words.begin());
        for (u64 i = 0; i < len + kJumpsAhead + 36; ++i) jumps4[i] = jump4(s, words.data(), static_cast<u32>(i));
        for (u64 i = 0; i < len + kJumpsAhead; ++i) jumps16[i] = jump16(jumps4.data(), static_cast<u32>(i));
        for (u64 i = 0; s.post_count && i < len; i += 1 + rng() % 7) {
            std::vector<Visit> none;
            const u64 draws = plain_walk(s, L, s.cache_base + i, kNoSelf, none) - s.cache_base - i;
            if (i + draws > len) continue;  // past the cache, where the lengths are not used
            ++lengths;
            if (pre_length(s, words.data(), jumps4.data(), jumps16.data(), static_cast<u32>(i)) !=
                (draws > kMaxPre ? kLongPre : draws))
                ++bad;
            longs += draws > kMaxPre;
        }
        for (int w = 0; w < 40; ++w) {
            const u64 c0 = s.cache_base + rng() % len;
            const u32 self = rng() % 2 ? kNoSelf : s.post_off + static_cast<u32>(rng() % (s.post_count + 1));
            std::vector<Visit> a, b;
            int err = 0;
            s.err = &err;
            Record v{a};
            const u64 e1 = walk_pre(s, c0, self, v), e2 = plain_walk(s, L, c0, self, b);
            ++walks;
            for (const auto& x : b) hits += std::get<1>(x);
            if (e2 > s.cache_base + len) {  // drew past the cache: flagged, and a prefix of the visits
                ++overruns;
                if (!(err & kErrCache) || a.size() > b.size()) ++bad;
            } else if (err || e1 != e2 || a != b) {
                ++bad;
            }
        }
    }
    std::printf("walks %ld mismatches %ld cache_overruns %ld hits %ld lengths %ld long %ld\n", walks, bad, overruns, hits,
                lengths, longs);
    return bad != 0;
}
