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
    bool whole;      // whole 256-column tiles (128 for GEGLU) of the pair kernel
};

struct GemmPlan {
    bool pair;
    int width, split;
    int pair_cols = 256;     // accumulator columns of a pair's tile
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

// The least of the modelled times, fitted to calls of 64 x 1280 x 1280 to 9216 x 320 x 1280 (M x N x K) in
// FP16 with cold weights on one B200; x stands for waves of CTAs (pairs), k for K blocks of 64.  Measured, in us:
//                          64 columns  80     96     128 columns  pairs x 128  pairs x 256
//   4096 x  320 x  320          6.6      4.2    4.2       4.5          -            -
//   4096 x  320 x 1280          9.3      6.9    7.4       7.9          -            -
//   9216 x  320 x 1280         16.8     10.9   16.8      17.4          -            -
//   1024 x  640 x 2560          8.9      9.4   10.5      11.0        10.7           -
//    576 x 1280 x 1280          6.1      6.5    6.7       7.2         7.4         11.1
//    512 x 3072 x 3072         17.5     17.4   12.6      13.7        13.2         20.0
//   2304 x  640 x 2560         15.3     10.0   11.1      11.9        11.5           -
//   1024 x 3072 x 3072         30.5       -      -       31.4        21.8         21.0
//   4096 x 3072 x 3072         92         -      -       88          64.5         57
//   GEGLU  256 x  640 -> 2560   8.3       -      -         -          6.3          8.8
//   GEGLU 1024 x  640 -> 2560  18.1       -      -         -         12.0         12.5
//   GEGLU 4096 x  320 -> 1280  22.2       -      -         -         17.0         14.9
//   Q, K, V with norm + RoPE, K = 3072: 256 rows 18.2 with 128 columns, 26.5 with 256; 512 rows 29.2 and
//   27.7; 1024 rows 50.3 and 46.7
// A tile split over CTAs pays where few tiles have a long K: 64 x 1280 x 5120 14.3 us, 10.1 over two CTAs, 7.8 over
// four, 9.2 over eight; 256 x 1280 x 5120 14.2, 11.4, 13.7.  The splits are entered at about 0.8 us less than they
// take when all CTAs run at once, and three when not: with the times themselves launches of a few tiles would be
// split less than tests/test_gemm_plan.py has it (256 x 1280 x 1280 6.4 us over two, 5.7 whole).
// GEGLU is not split: the two accumulators of a tile double the exchange.
// The problems of a launch may differ in K (the queries and the keys of a cross-attention): the
// longest sets the time, the shortest how far its tiles can be split, a CTA without a K
// block would have nothing to add and nothing to wait for.
inline GemmPlan plan_gemm(const GemmShape* p, int n, int sms) {
    bool geglu = false, heads = false;
    int kb = 0, kb_min = 0;
    for (int i = 0; i < n; ++i) {
        geglu = geglu || p[i].geglu;
        heads = heads || p[i].heads;
        const int b = gemm_k_blocks(p[i].K);
        kb = b > kb ? b : kb;
        kb_min = i == 0 || b < kb_min ? b : kb_min;
    }
    auto tiles = [&](int w) {
        long long t = 0;
        for (int i = 0; i < n; ++i) t += static_cast<long long>(gemm_row_tiles(p[i].M)) * ((p[i].N + w - 1) / w);
        return t;
    };
    auto waves = [&](int w, int s) { return static_cast<double>((tiles(w) * s + sms - 1) / sms); };
    GemmPlan best = {false, 64, 1};
    // whole heads with norm + RoPE are faster on pairs at any size (the narrow kernel: 256 rows 37 us, 1024 rows 128)
    double best_us = 1e30;
    auto offer = [&](const GemmPlan& o, double us) {
        if (us < best_us) { best = o; best_us = us; }
    };
    if (!heads) {
        const double x = waves(64, 1);
        if (geglu) offer(best, kb * 0.45 * x + 4.3 + 3.0 * x);
        else offer(best, x <= 1.0 ? 2.2 + 0.165 * kb : 2.5 + x * (0.8 + 0.155 * kb));
    }
    if (!geglu && !heads) {
        // Between 64 and 128 columns for widths that these divide badly (320, 640) and for what 64 columns make two
        // waves of; with several CTAs to an SM only 80 columns, whose rings still fit twice (a short K has
        // rings of two stages there and gains nothing: 9216 x 320 x 320 8.0 us, 7.7 with 64 or 128).
        for (int w = 80; w < 128; w += 16) {
            if (waves(w, 1) <= 1.0) offer({false, w, 1}, 1.6 + 0.6 * w / 64 + (0.12 + 0.045 * w / 64) * kb);
            else if (w == 80 && kb > 8) offer({false, w, 1}, 2.5 + waves(w, 1) * (1.15 + 0.14 * kb));
        }
        const double x = waves(128, 1);
        offer({false, 128, 1}, x <= 1.0 ? 2.8 + 0.21 * kb : 2.0 + x * (1.0 + 0.30 * kb));
        for (int s = 2; s <= 8 && kb >= 3 * s && kb_min >= s && tiles(64) * s * 2 <= 3LL * sms; s *= 2) {
            // (with more CTAs than SMs a longer part of K costs more than the split saves)
            if (waves(64, s) <= 1.0) offer({false, 64, s}, 3.15 + 0.15 * kb / s);
            else if (kb <= 12 * s) offer({false, 64, s}, 3.22 + 0.27 * kb / s * tiles(64) * s / sms);
        }
    }
    for (int cols = 256; cols >= 128; cols /= 2) {
        bool whole = true;
        long long t = 0;
        for (int i = 0; i < n; ++i) {
            const int out = gemm_pair_cols(p[i].geglu) * cols / 256;
            whole = whole && (cols == 256 ? p[i].whole : p[i].N % out == 0);
            t += static_cast<long long>(gemm_pair_row_tiles(gemm_row_tiles(p[i].M))) * (p[i].N / out);
        }
        if (!whole) continue;
        const double x = static_cast<double>((t + sms / 2 - 1) / (sms / 2));
        if (cols == 256) offer({true, 64, 1, 256}, heads ? 8.0 + x * (1.0 + 0.37 * kb) : geglu ? 2.5 + 0.17 * kb + x * (2.6 + 0.24 * kb) : 4.5 + x * (0.8 + 0.32 * kb));
        else offer({true, 64, 1, 128}, heads ? 6.5 + x * (1.0 + 0.215 * kb) : geglu ? 2.0 + x * (2.4 + 0.15 * kb) : 3.2 + x * (0.5 + 0.20 * kb));
    }
    return best;
}

}  // namespace bdattn
