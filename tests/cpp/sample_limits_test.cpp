// Host-only check of the admission rule of the sampling kernels' candidate lists (retrograd_b200/csrc/sample_limits.hpp): the
// kernel's selection restated, on values in random order.
#include "../../retrograd_b200/csrc/sample_limits.hpp"

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

using namespace rb200;

#define CHECK(cond)                                                                  \
    do {                                                                             \
        if (!(cond)) {                                                               \
            std::fprintf(stderr, "CHECK failed at line %d: %s\n", __LINE__, #cond);  \
            std::exit(1);                                                            \
        }                                                                            \
    } while (0)

// Candidates of a row, and the most of any chunk.
static int candidates(int vocab, int need, std::mt19937 & rng, int & most) {
    int total = 0;
    most = 0;
    for (int base = 0; base < vocab; base += kSampleChunk) {
        const int n = std::min(kSampleChunk, vocab - base);
        std::vector<uint32_t> v(n), top(kSampleChunkThreads, 0);
        for (int i = 0; i < n; ++i) {
            v[i] = rng() | 1u;
            top[i % kSampleChunkThreads] = std::max(top[i % kSampleChunkThreads], v[i]);
        }
        std::nth_element(top.begin(), top.begin() + need - 1, top.end(), std::greater<uint32_t>());
        const int count = (int)std::count_if(v.begin(), v.end(), [&](uint32_t x) { return x >= top[need - 1]; });
        total += count;
        most = std::max(most, count);
    }
    return total;
}

int main() {
    std::mt19937 rng(7);
    for (int vocab : {260, 4097, 32000, 98304, 128256, 151936, 201088, 262144}) {
        int limit = 0;
        for (int need = 1; need <= kSampleMaxNeed; ++need) {
            if (!sample_candidates_fit(vocab, need)) break;
            limit = need;
        }
        for (int need = limit + 1; need <= 2 * kSampleMaxNeed; ++need) CHECK(!sample_candidates_fit(vocab, need));
        int most, worst = 0;
        for (int trial = 0; trial < 60; ++trial) {
            worst = std::max(worst, candidates(vocab, limit, rng, most));
            CHECK(most <= kSampleChunkCands);
        }
        std::printf("%d logits: up to %d, at most %d candidates\n", vocab, limit, worst);
        CHECK(worst <= kSampleRowCands);
        if (limit < kSampleMaxNeed) CHECK(candidates(vocab, limit + 8, rng, most) > kSampleRowCands);      // the rule gives little away
    }
    // rows that never ask for candidates are served whatever their size, up to one chunk per thread of the finishing block
    CHECK(sample_chunked(4 << 20, true, 0, 0.f, 1.f, 0) && !sample_chunked((4 << 20) + 1, true, 0, 0.f, 1.f, 0));
    CHECK(sample_chunked(128256, true, 40, 0.05f, 0.95f, 500) && !sample_chunked(128256, true, 0, 0.05f, 1.f, 0));
    CHECK(!sample_chunked(128256, true, 0, 0.f, 0.95f, 0) && !sample_chunked(128256, false, 40, 0.f, 0.95f, 0));
    CHECK(sample_chunked(128256, false, 40, 0.5f, 1.f, 20) && !sample_chunked(128256, false, 0, 0.f, 1.f, 120));
    return 0;
}
