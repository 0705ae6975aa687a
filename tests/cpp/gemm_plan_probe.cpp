// The plan of a launch of linear layers and the pair kernel's tile rules as C functions, for tests/test_gemm_plan.py.
#include "../../brodiffusion_b200/csrc/gemm_plan.h"

using namespace bdattn;

extern "C" {

// shapes: n rows of M, N, K; out: pair, width, split, pair_cols
void probe_plan(const int* shapes, int n, int geglu, int heads, int sms, int* out) {
    GemmShape s[3];
    for (int i = 0; i < n; ++i)
        s[i] = {shapes[3 * i], shapes[3 * i + 1], shapes[3 * i + 2], geglu != 0, heads != 0,
                shapes[3 * i + 1] % gemm_pair_cols(geglu != 0) == 0};
    const GemmPlan p = plan_gemm(s, n, sms);
    out[0] = p.pair;
    out[1] = p.width;
    out[2] = p.split;
    out[3] = p.pair_cols;
}

// the fewest K blocks that any CTA of a tile has
int probe_fewest_blocks(int K, int split) {
    const int all = gemm_k_blocks(K);
    int least = all;
    for (int i = 0; i < split; ++i) {
        const int n = gemm_part_begin(all, split, i + 1) - gemm_part_begin(all, split, i);
        least = n < least ? n : least;
    }
    return least;
}

int probe_acc_reused(int tile, int pairs, int total_tiles) { return pair_acc_reused(tile, pairs, total_tiles); }

}
