// Which kernel, tile width and number of CTAs per tile a launch of linear layers gets.
// Plain C++ without CUDA headers, so that the rule can be checked on any host.
#pragma once

#ifdef __CUDACC__
#define BDATTN_HD __host__ __device__
#else
#define BDATTN_HD
#endif

namespace bdattn {

// One problem  C[M, N] = A[M, K] . W[N, K]^T  of a launch.
struct GemmShape {
    int M, N, K;
    bool geglu;
    bool heads;      // whole heads with norm + RoPE
    bool whole;      // whole 256-column tiles (128 for GEGLU)
};

struct GemmPlan {
    bool pair;
    int width, split;
};

BDATTN_HD constexpr int gemm_k_blocks(int K) { return (K + 63) / 64; }
// The K blocks of a tile that CTA `part` of `split` takes begin here (and end where the next one's
// begin).  Every CTA has at least one as long as split <= k_blocks.
BDATTN_HD constexpr int gemm_part_begin(int k_blocks, int split, int part) { return part * k_blocks / split; }

BDATTN_HD constexpr int gemm_row_tiles(int M) { return (M + 127) / 128; }
// Output tiles of the pair kernel: 256 rows x 256 columns (GEGLU: 128 and their gates)
BDATTN_HD constexpr int gemm_pair_row_tiles(int row_tiles) { return (row_tiles + 1) / 2; }
BDATTN_HD constexpr int gemm_pair_cols(bool geglu) { return geglu ? 128 : 256; }

// A pair of CTAs takes the tiles  first, first + pairs, ...  and its two accumulators in turn: whether the
// accumulator of `tile` is used again, so that its release is waited for.
BDATTN_HD constexpr bool pair_acc_reused(int tile, int pairs, int total_tiles) {
    return tile + 2 * pairs < total_tiles;
}

// The least of the modelled times, fitted to FP16 calls of 64 x 1280 x 1280 to 9216 x 320 x 1280
// (M x N x K) on one B200.  A K block of 64 costs a CTA 0.30 us with 64 or 128 columns and a
// pair 0.28 us; the rest of a call is 3 us (64 columns, one CTA per SM), 4.3 (64, several), 4.2
// (128) or 7.5 (pairs), and the exchange of a split tile 1.5, as much again for a second wave.
// Several CTAs of 64 columns share an SM and hide part of each other.  Examples, measured:
//   64 x 1280 x 5120   64 columns 27.2 us, split over four 10.6, pairs 28.9
//   256 x 1280 x 1280  64 columns  8.8 us, split over two 8.1, over four 9.6
//   4096 x 320 x 320   64 columns  6.4 us, 128 columns 5.5
//   1024 x 3072 x 3072 64 columns 36.8 us, 128 columns 37.9, pairs 21.8
// GEGLU: 64 x 1280 -> 5120 64 columns 16.0 us, pairs 14; 256 x 320 -> 1280 8.5 and 9.
// None is split: the two accumulators of a tile double the exchange.
// (BF16 is within a few per cent of FP16: 64 x 1280 x 5120 9.6 us against 9.8, 4096 x 3072 x 3072 54.5 against 57.0.)
// The problems of a launch may differ in K (the queries and the keys of a cross-attention): the
// longest sets the time, the shortest how far its tiles can be split, a CTA without a K
// block would have nothing to add and nothing to wait for.
inline GemmPlan plan_gemm(const GemmShape* p, int n, int sms) {
    bool whole = true, geglu = false, heads = false;
    int kb = 0, kb_min = 0;
    for (int i = 0; i < n; ++i) {
        whole = whole && p[i].whole;
        geglu = geglu || p[i].geglu;
        heads = heads || p[i].heads;
        const int b = gemm_k_blocks(p[i].K);
        kb = b > kb ? b : kb;
        kb_min = i == 0 || b < kb_min ? b : kb_min;
    }
    // whole heads with norm + RoPE are faster on pairs at any size (16 rows of 3072: 31 against 24 us; three
    // tiles on three pairs, 1024 rows to 2 heads of 128 with K = 1024, 17.7 us, half of it on the narrow kernel 27.7)
    if (heads) return {whole, 64, 1};
    auto tiles = [&](int w) {
        long long t = 0;
        for (int i = 0; i < n; ++i) t += static_cast<long long>(gemm_row_tiles(p[i].M)) * ((p[i].N + w - 1) / w);
        return t;
    };
    auto waves = [&](int w, int s) { return static_cast<double>((tiles(w) * s + sms - 1) / sms); };
    GemmPlan best = {false, 64, 1};
    double best_us;
    {
        const double x = waves(64, 1), b = kb * (geglu ? 0.45 : 0.30) * (geglu ? x : 1.0);
        best_us = x <= 1.0 ? b + 3.0 : (geglu ? b : 0.62 * x * b) + 4.3;
        if (geglu) best_us += 3.0 * x;
    }
    auto offer = [&](const GemmPlan& o, double us) {
        if (us < best_us) { best = o; best_us = us; }
    };
    if (!geglu) {
        offer({false, 128, 1}, waves(128, 1) * kb * 0.31 + 4.2);
        // (beyond one and a half CTAs per SM a split only adds waves: 256 x 3072 x 3072 over four 21.4 us,
        // over two 16.2)
        for (int s = 2; s <= 8 && kb >= 3 * s && kb_min >= s && tiles(64) * s * 2 <= 3LL * sms; s *= 2) {
            const double x = waves(64, s), b = 0.30 * kb / s;
            offer({false, 64, s}, (x <= 1.0 ? b : 0.725 * x * b) + 4.5 + 1.5 * (x - 1.0));
        }
    }
    if (whole) {
        int pair_tiles = 0;
        for (int i = 0; i < n; ++i)
            pair_tiles += gemm_pair_row_tiles(gemm_row_tiles(p[i].M)) * (p[i].N / gemm_pair_cols(p[i].geglu));
        const double x = (pair_tiles + sms / 2 - 1) / (sms / 2);
        offer({true, 64, 1}, x * (kb * 0.28 + (geglu ? 2.5 : 0.0)) + (geglu ? 5.3 : 7.5));
    }
    return best;
}

}  // namespace bdattn
