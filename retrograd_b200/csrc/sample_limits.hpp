// Which sampling rows the per-chunk candidate lists of sample.cu can serve. Host and device, no CUDA types.
#pragma once

#include <cmath>
#include <cstdint>

namespace rb200 {

constexpr int kSampleChunk = 4096, kSampleChunkThreads = 256;
constexpr int kSampleRowThreads = 1024;         // of the finishing block, one per chunk
constexpr int kSampleMaxNeed = 128;             // largest top_k (or, without top_k, n_top) of a row, in a vocabulary of few chunks
constexpr int kSampleChunkCands = 256;          // candidates a chunk may hand on: 177 +- 9 of 4096 values in random order for 128 wanted
constexpr int kSampleRowCands = 4096;           // candidates of a row the finishing block stages in shared memory

// Whether a row's candidates fit the finishing block when `need` values are wanted. A chunk hands on the values at or above the
// need-th largest of its threads' maxima: with the values in random order, as many as it takes to meet `need` different threads,
// 256 ln(1 / (1 - x)) of them with x = need / 256, variance 256 (x / (1 - x) + ln(1 - x)). Admitted up to six standard deviations:
// 96 at 128 256 logits, 84 at 151 936, 67 at 201 088, 54 at 262 144. Rows that overflow pay for the chunks and the general
// passes (a step of 160 rows of 201 088 logits, top_k 80: 7296 us, against 6931 by the general passes alone; 1203 at top_k 64
// from lists that fit).
inline bool sample_candidates_fit(int n_vocab, int need) {
    if (need <= 0) return true;
    if (need > kSampleMaxNeed) return false;
    const int chunks = (n_vocab + kSampleChunk - 1) / kSampleChunk;
    const double x = need / (double)kSampleChunkThreads, l = -std::log1p(-x);
    const double mean = kSampleChunkThreads * l, variance = kSampleChunkThreads * (x / (1.0 - x) - l);
    return chunks * mean + 6.0 * std::sqrt(chunks * variance) <= kSampleRowCands;
}

// Whether a row with these options is served from per-chunk results (the caller then sets kSampleFlagChunked, provided the row
// has no grammar mask and no forced token).
inline bool sample_chunked(int n_vocab, bool v2, int top_k, float min_p, float top_p, uint32_t n_top) {
    if ((n_vocab + kSampleChunk - 1) / kSampleChunk > kSampleRowThreads) return false;
    if (v2 && top_k > 0 && top_k < n_vocab) return sample_candidates_fit(n_vocab, top_k);
    return top_p >= 1.0f && !(v2 && min_p > 0.0f) && sample_candidates_fit(n_vocab, (int)(n_top < (uint32_t)n_vocab ? n_top : (uint32_t)n_vocab));
}

} // namespace rb200
