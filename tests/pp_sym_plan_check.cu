// Host check of the pair-once sum's plan (pp_sym.cu), run by test_pp_sym_plan.py: no
// heap memory (the entry point without allocation makes one on each call), and for
// every number of blocks ranges that cover all tiles once and change block at most
// once.
#include <cstdio>

#include "pp_sym.cu"

extern int allocations;  // counted by the operators in test_pp_sym_plan.py

using namespace nbody;

int main() {
    for (int sms : {148, 152, 132, 20}) {
        for (int64_t blocks = 1; blocks <= kSymMaxBlocks + 1; ++blocks) {
            allocations = 0;
            const SymPlan p = pp_sym_plan(blocks * kSymB - 7, sms);
            if (allocations) return std::printf("FAILED: %d heap allocations\n", allocations), 1;
            if (p.blocks == 0) continue;
            if (p.blocks != blocks || p.ctas > kSymMaxCtas || p.begin[0] != 0 ||
                p.begin[p.ctas] != sym_first(p, p.blocks))
                return std::printf("FAILED: range, %d blocks on %d SMs\n", p.blocks, sms), 1;
            for (int c = 0; c < p.ctas; ++c) {
                const int first = p.begin[c], past = p.begin[c + 1];
                if (past < first) return std::printf("FAILED: order, %d blocks on %d SMs\n", p.blocks, sms), 1;
                if (past > first && sym_block(p, past - 1) - sym_block(p, first) > 1)
                    return std::printf("FAILED: two changes of block, %d blocks on %d SMs\n", p.blocks, sms), 1;
            }
        }
        if (pp_sym_plan((kSymMaxBlocks + 1) * int64_t{kSymB}, sms).blocks != 0) return std::printf("FAILED: limit\n"), 1;
    }
    return 0;
}
