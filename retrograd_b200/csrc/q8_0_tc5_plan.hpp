// How the Q8_0 tcgen05 GEMM cuts a product into tiles and splits of the reduction. Host only, no CUDA types.
#pragma once

#include <cstdint>

namespace rb200 {

constexpr int kQ8Tc5MaxSplits = 8, kQ8Tc5MinSplitStages = 8;

struct Q8Tc5Plan {
    bool wide;      // token tiles of 256 instead of 128
    int splits;     // ranges of the reduction, each ceil(stages / splits) stages of 64 columns (the last one may be shorter)
};

// The form and the number of splits with the shortest estimated time, in cycles, for whole waves of one CTA per SM.
// 256-token tiles halve the decode work per product (measured per 64-column stage: about 1800 cycles at N = 256, where the
// twelve MMAs take 1536, and 1300 at N = 128, where the producers set the pace; narrower MMAs do not help the producers).
// Every wave pays for its CTAs' beginning and end. A split costs the finish kernel, its CTAs' stores of partial results (nothing
// of the CTA runs beside them) and the reads of the finish kernel. The constants were fitted to ten shapes at 24 to 1024 tokens,
// each unsplit and with every number of splits: the chosen form is within 1.2 % of the fastest measured everywhere, and nowhere
// slower than unsplit. us unsplit -> split:
//   4096 x 4096     50 -> 24 at 17 tokens, 53 -> 38 at 200 (four splits); 54 at 300 and 56 at 512, where two would take 56 and 64
//   4096 x 14 336  153 -> 52 at 17 tokens, 156 -> 76 at 200 (four), 161 -> 142 at 512 (two)
//   4096 x 2880     41 -> 34 at 200 (four); 42 at 320, where two would take 49
// `tail`: the finish kernel would also do the row-wise step that follows. Unsplit, that step is a kernel of its own and the residual
// is read at the end of each tile: in steps of 257 to 640 tokens that took 14 to 22 us per layer (eight layers, 4096 x 4096
// with the RMS norm behind it, 320 tokens: 4424 us unsplit, 4253 in two; 2880 x 4096, 640 tokens: 2727 and 2585).
inline Q8Tc5Plan q8_0_tc5_plan(uint32_t n_out, uint32_t n_in, int n_tokens, int n_sm, bool tail, int forced_tile = 0) {
    const int n_it = (int)n_in / 64, row_tiles = (int)((n_out + 127) / 128);
    Q8Tc5Plan best{false, 1};
    long long best_cycles = -1;
    for (int wide = 0; wide < 2; ++wide) {
        if (wide && (n_tokens <= 128 || forced_tile == 128)) continue;
        if (!wide && n_tokens > 128 && forced_tile == 256) continue;
        const long long tiles = (long long)row_tiles * ((n_tokens + (wide ? 255 : 127)) / (wide ? 256 : 128));
        for (int splits = 1; splits <= kQ8Tc5MaxSplits && (splits == 1 || n_it / splits >= kQ8Tc5MinSplitStages); ++splits) {
            const int per_split = (n_it + splits - 1) / splits;
            if ((n_it + per_split - 1) / per_split != splits) continue;      // an empty last range
            if (splits > 1 && tiles * splits > n_sm) break;                  // a split that does not fit one wave gains too little for its traffic
            const long long waves = (tiles * splits + n_sm - 1) / n_sm;
            long long cycles = waves * ((long long)per_split * (wide ? 1800 : 1300) + (wide ? 10000 : 6000));
            if (splits > 1) cycles += 6000 + (long long)n_tokens * n_out * (60 + 9 * splits) / 5000;
            else if (tail) cycles += 26000;
            if (best_cycles < 0 || cycles < best_cycles) {
                best_cycles = cycles;
                best = Q8Tc5Plan{wide != 0, splits};
            }
        }
    }
    return best;
}

} // namespace rb200
