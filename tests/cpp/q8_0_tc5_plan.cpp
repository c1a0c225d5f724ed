// Prints "wide splits stages-of-the-last-range stages-per-range" of the Q8_0 tcgen05 GEMM on 148 SMs for every four arguments
// (rows, columns, tokens, whether a row-wise step follows that the finish kernel can do).
#include "../../retrograd_b200/csrc/q8_0_tc5_plan.hpp"

#include <cstdio>
#include <cstdlib>

int main(int argc, char ** argv) {
    for (int i = 1; i + 3 < argc; i += 4) {
        const int n_out = std::atoi(argv[i]), n_in = std::atoi(argv[i + 1]), n_tokens = std::atoi(argv[i + 2]), n_it = n_in / 64;
        const rb200::Q8Tc5Plan plan = rb200::q8_0_tc5_plan(n_out, n_in, n_tokens, 148, std::atoi(argv[i + 3]) != 0);
        const int per_split = (n_it + plan.splits - 1) / plan.splits;
        std::printf("%d %d %d %d\n", plan.wide ? 256 : 128, plan.splits, n_it - (plan.splits - 1) * per_split, per_split);
    }
    return 0;
}
