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

// The least of the modelled times, fitted to calls of 16 x 64 x 64 to 9300 x 5200 x 3800 (M x N x K) in BF16
// with cold weights on one B200; x stands for waves of CTAs (pairs), k for K blocks of 64.  The choice takes 2 %
// longer than the best of the kernels over 960 plain layers (5 % with terms fitted to long K alone), 0.1 % over 340
// GEGLU layers and 0.5 % over 290 with norm + RoPE.  Measured, in us:
//                          64 columns  80     96     128 columns  pairs x 128  pairs x 256
//   4096 x  320 x  320          5.4      4.0    4.0       4.3          -            -
//   4096 x 1280 x  320         11.5      8.7    9.7       8.7        10.1         10.5
//   4096 x 2560 x  112         12.1     12.0   11.0      11.2        14.2         12.8
//   4096 x  320 x 1280          9.3      6.9    7.4       7.9          -            -
//   9216 x  320 x 1280         16.8     10.9   16.8      17.4          -            -
//   9216 x 1280 x  640         29.4     26.5   36.7      29.6        19.7         17.7
//    576 x 5120 x  448          8.6      9.3    8.6       8.8         7.7          8.1
//   1024 x  640 x 2560          8.9      9.4   10.5      11.0        10.7           -
//    576 x 1280 x 1280          6.1      6.5    6.7       7.2         7.4         11.1
//    512 x 3072 x 3072         17.5     17.4   12.6      13.7        13.2         20.0
//   2304 x  640 x 2560         15.3     10.0   11.1      11.9        11.5           -
//   2240 x 2304 x 2240         34.2     27.1   34.5      34.3        24.1         26.7
//   1024 x 3072 x 3072         30.5       -      -       31.4        21.8         21.0
//   4096 x 3072 x 3072         92         -      -       88          64.5         57
//    576 x 4096 x  936         19.1     15.2   16.5      16.6        13.1         11.5
//   GEGLU   64 x 1280 -> 5120  12.8       -      -         -         12.4         13.0
//   GEGLU 1024 x  640 -> 2560  18.1       -      -         -         12.2         12.6
//   GEGLU 4096 x  320 -> 1280  22.2       -      -         -         17.0         14.9
//   GEGLU 4096 x 2808 -> 1280 112         -      -         -         70.2         59.2
//   Q, K, V with norm + RoPE, K = 3072: 256 rows 18.9 with 128 columns, 26.9 with 256; 512 rows 28.4 and
//   27.8; 1024 rows 49.1 and 45.3; 3580 rows to 16 heads of 64, K = 1288, 38.7 and 35.0
// A tile of a pair costs its epilogue, 2 to 5 us, however short its K is, so that narrow tiles, twice as many, pay
// where wide ones leave pairs idle and not by their lower time per K block alone.  Where the rows are no multiple of 32 bytes (K of 936 or
// 2808) a box row touches five sectors instead of four, and a K block takes 1.6 times as long with a CTA for every tile and
// several rounds of them (2.4 with 80 columns), 1.35 on pairs with 128 columns, 1.15 with 256.
// A tile split over CTAs pays where few tiles have a long K: 64 x 1280 x 5120 14.3 us, 10.1 over two CTAs, 7.8 over
// four, 8.8 over eight; 256 x 1280 x 5120 14.2, 11.4, 13.7.  The splits are entered at about 0.8 us less than they
// take when all CTAs run at once, and three when not: with the times themselves launches of a few tiles would be
// split less than tests/test_gemm_plan.py has it (256 x 1280 x 1280 6.1 us over two, 5.7 whole).
// GEGLU is not split: the two accumulators of a tile double the exchange.
// The problems of a launch may differ in K (the queries and the keys of a cross-attention): the
// longest sets the time, the shortest how far its tiles can be split, a CTA without a K
// block would have nothing to add and nothing to wait for.
inline GemmPlan plan_gemm(const GemmShape* p, int n, int sms) {
    bool geglu = false, heads = false, odd = false;
    int kb = 0, kb_min = 0, m_max = 0;
    for (int i = 0; i < n; ++i) {
        geglu = geglu || p[i].geglu;
        heads = heads || p[i].heads;
        odd = odd || p[i].K % 16 != 0;
        m_max = p[i].M > m_max ? p[i].M : m_max;
        const int b = gemm_k_blocks(p[i].K);
        kb = b > kb ? b : kb;
        kb_min = i == 0 || b < kb_min ? b : kb_min;
    }
    auto tiles = [&](int w) {
        long long t = 0;
        for (int i = 0; i < n; ++i) t += static_cast<long long>(gemm_row_tiles(p[i].M)) * ((p[i].N + w - 1) / w);
        return t;
    };
    auto rounds = [&](long long t, long long at_once) { return static_cast<double>((t + at_once - 1) / at_once); };
    auto waves = [&](int w, int s) { return rounds(tiles(w) * s, sms); };
    GemmPlan best = {false, 64, 1};
    // whole heads with norm + RoPE are faster on pairs at any size (the narrow kernel: 256 rows 37 us, 1024 rows 128)
    double best_us = 1e30;
    auto offer = [&](const GemmPlan& o, double us) {
        if (us < best_us) { best = o; best_us = us; }
    };
    if (geglu && !heads) {
        const double k = odd ? 1.65 * kb : kb;
        offer(best, 2.3 + 0.15 * k + waves(64, 1) * (2.5 + 0.245 * k));
    } else if (!heads) {
        // A ring of two (K of at most 512) lets three CTAs of 128 columns, or four of 64, share an SM, and the time
        // jumps where there are more (4096 x 1280 x 320: 320 tiles of 128 columns, 2.2 to an SM, 8.7 us; 640 of 64, 4.3,
        // 11.5; 10.1 on pairs).  With a longer K an SM has two CTAs of 64 or 80 columns (1024 x 2560 x 1280, 256 tiles
        // of 80, 10.1, 1024 x 3072 x 1280, 312, 16.5) and one of 128.
        const bool short_k = kb <= 8;
        const double k64 = odd ? (short_k ? 1.7 : 1.85) * kb : kb, k80 = odd ? 2.4 * kb : kb;
        auto per_sm = [&](int w) { return static_cast<double>(tiles(w)) / sms; };
        auto late = [](double a) { return a > 0.0 ? a : 0.0; };
        const double x = waves(64, 1), t64 = per_sm(64), y = waves(128, 1), t128 = per_sm(128);
        // Short K off 32 bytes and more tiles than SMs: the L2 sets the pace, in proportion to the tiles, so that wide ones
        // are better but for the CTAs that they leave over: two CTAs of 64 columns to an SM, or four, that run at once
        // instead of 128 columns in a second round (64, 96 and 128 columns: 3573 x 704 x 152 7.2, 7.3, 8.1 us,
        // 7290 x 392 x 216 8.4, 8.0, 10.3, 1911 x 2112 x 200 9.1, 8.0, 9.4, 3829 x 5016 x 392 44.7, 39.7, 35.1; with the terms
        // for even rows up to 30 % longer than the best of 64 and 128, over 183 shapes now 3 % on average).
        const bool odd_short = odd && short_k && y > 1.0;
        if (odd_short) {
            offer({false, t64 <= 2.0 ? 64 : t64 <= 4.0 ? 96 : 128, 1}, 3.0 + 0.11 * kb + t128 * (1.46 + 0.37 * kb));
        } else if (short_k && y > 1.0 && t128 <= 3.0) {
            // All of these CTAs run at once, three to an SM with 96 columns and more: the width that leaves no SM with one more
            // than the others.  Measured behind another kernel, where nothing of the launch before is left to run
            // beside (64, 96, 112, 128 columns and pairs with 128): 4096 x 960 x 320 7.8, 7.0, 6.8, 7.2 us, 1564 x 2752 x 256 7.8,
            // 7.1, 7.6, 6.4, 4096 x 1280 x 320 10.6, 9.9, 8.2, 8.7, 10.9, 3628 x 896 x 320 7.2, 6.3, 6.7, 6.8, 8.4, 1672 x 1792 x 512
            // 8.6, 7.5, 8.0, 8.1, 9.3.  (Behind itself a launch starts in the SMs that its predecessor leaves, and
            // pairs look up to 1 us better than they are.)
            const double t96 = per_sm(96), t112 = per_sm(112);
            if (t64 <= 2.0) offer({false, 64, 1}, 3.5 + 0.25 * kb + t64 * (0.3 + 0.07 * kb));
            else if (t128 > 1.78 && t128 <= 2.0) offer({false, 128, 1}, 3.5 + 0.25 * kb + t128 * (0.5 + 0.09 * kb));
            else if (t96 <= 3.0) offer({false, 96, 1}, 3.5 + 0.25 * kb + t96 * (0.5 + 0.08 * kb));
            else if (t112 <= 3.0) offer({false, 112, 1}, 3.9 + 0.25 * kb + t112 * (0.6 + 0.1 * kb));
            else offer({false, 128, 1}, 3.9 + 0.25 * kb + t128 * (0.7 + 0.11 * kb));
        } else {
            offer(best, x <= 1.0  ? 2.2 + 0.165 * kb
                        : short_k ? 4.4 + 0.61 * k64 - late(2.0 - t64) * (1.7 + 0.1 * k64) + late(t64 - 4.0) * 0.9 +
                                        (rounds(tiles(64), 4LL * sms) - 1.0) * (1.0 + 0.48 * k64)
                                  : 1.15 + x * (0.6 + 0.05 * k64) + rounds(tiles(64), 2LL * sms) * (1.45 + 0.176 * k64));
        }
        // Between 64 and 128 columns for widths that these divide badly (320, 640) and for what 64 columns make two
        // waves of; with several CTAs to an SM only 80 columns, whose rings still fit twice (a short K has
        // rings of two stages there and gains nothing: 9216 x 320 x 320 8.0 us, 7.7 with 64 or 128).
        for (int w = 80; w < 128; w += 16) {
            if (waves(w, 1) <= 1.0) offer({false, w, 1}, 1.6 + 0.6 * w / 64 + (0.12 + 0.045 * w / 64) * kb);
            else if (w == 80 && !short_k) offer({false, w, 1}, 1.0 + waves(w, 1) * (1.4 + 0.065 * k80) + rounds(tiles(w), 2LL * sms) * (0.5 + 0.166 * k80));
        }
        if (!odd_short && !(short_k && y > 1.0 && t128 <= 3.0))
            offer({false, 128, 1}, y <= 1.0  ? 2.8 + 0.21 * kb
                                   : short_k ? 5.6 + 0.68 * kb - late(3.0 - t128) * (0.4 + 0.05 * kb) + late(t128 - 3.0) * 0.9 +
                                                   (rounds(tiles(128), 3LL * sms) - 1.0) * (2.5 + 0.45 * kb)
                                             : odd ? y * (2.9 + 0.38 * kb) : y * (3.0 + 0.265 * kb));
        for (int s = 2; s <= 8 && kb >= 3 * s && kb_min >= s && tiles(64) * s * 2 <= 3LL * sms; s *= 2) {
            // (with more CTAs than SMs a longer part of K costs more than the split saves, and of tiles with more than 64 rows
            // any: 135 x 640 x 5120 over eight 11.5 us, over four 8.0, and the same for 100 shapes drawn at random)
            if (waves(64, s) <= 1.0) offer({false, 64, s}, 3.15 + 0.15 * kb / s);
            else if (kb <= 12 * s && m_max <= 64) offer({false, 64, s}, 3.22 + 0.27 * kb / s * tiles(64) * s / sms);
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
        const double x = rounds(t, sms / 2);
        if (cols == 256) {
            const double f = odd ? 1.15 * kb : kb;
            offer({true, 64, 1, 256}, heads ? 9.3 + x * (3.0 + 0.3 * f) : geglu ? 4.4 + 0.03 * f + x * (2.6 + 0.24 * f)
                                                                           : 3.75 + 0.06 * f + x * (2.5 + 0.228 * f));
        } else {
            const double f = odd ? 1.35 * kb : kb;
            offer({true, 64, 1, 128}, heads ? 3.7 + 0.06 * f + x * (4.0 + 0.165 * f) : geglu ? 1.9 + 0.02 * f + x * (2.1 + 0.147 * f)
                                                                                     : 1.45 + 0.06 * f + x * (2.04 + 0.143 * f));
        }
    }
    return best;
}

}  // namespace bdattn
