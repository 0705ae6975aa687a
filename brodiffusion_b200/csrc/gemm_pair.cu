// Persistent two-SM linear layer for the large projections (Q/K/V of a DiT block:
// src/dit/flux.cpp:471-484; out-projection: src/dit/flux.cpp:519-525):
//   C[M,N] = A[M,K] . W[N,K]^T (+ bias) [-> per-head RMSNorm -> RoPE]
// Same operand layout and epilogue arithmetic as gemm_tc05_kernel; what differs is the
// schedule, for the larger problems, for GEGLU and, whatever their size, for whole heads
// with norm + RoPE (gemm_plan.h):
//   * a cluster of two CTAs owns a tile of 256 rows x kN = 256 or 128 columns and computes it with
//     tcgen05.mma.cta_group::2: every CTA stages its 128 rows of A and half of the tile's
//     weight rows, so a K block of 64 costs an SM 32 KB of L2 reads per 512 tensor-pipe cycles, with
//     128 columns 24 KB per 256.  An SM is fed at about 70 bytes a cycle, so the wide tile is the better
//     one wherever it fills the SMs and the narrow one where it does not: QKV of 256 rows of 3072 is 36
//     tiles of 256 columns for 74 pairs, 26.5 us, or 72 of 128, 18.2; of 512 rows 72 wide tiles 27.7,
//     144 narrow ones 29.2;
//   * a stage is 128 columns of K: the wait and the commit around a stage stand against sixteen MMAs' worth of the
//     tensor pipe and not eight (with stages of 64 a K block took 610 cycles where the pipe needs 512);
//   * the pairs walk a list of tiles (up to three problems in one launch; tiles of one
//     column block adjacent, in groups of sixteen row blocks, so that what runs together
//     reads few weight and few activation tiles);
//   * the accumulator is double-buffered in tensor memory (2 x kN columns), so the epilogue
//     of tile i (bias, RMSNorm, RoPE, stores) runs while the MMAs of tile i+1 are issued;
//   * the cos / sin rows and the outputs go through 2 KB of shared memory per epilogue warp, so
//     that global accesses are whole row pieces (a load or store with a row per lane touches 32
//     cache lines), and everything the epilogue reads from global memory is on its way before it is
//     needed: the bias in shared memory and the first table rows in registers before the
//     accumulator is ready, the next rows while a piece is worked on.  With bias values and table rows
//     loaded where they are used the epilogue of norm + RoPE took 19300 cycles a tile, 10 of the 31 us of
//     a 256-row prompt's projections, where the last one has nothing to hide behind.
// GEGLU (src/fused_transformer.cu:89-92,275-282) runs here too: a tile is then kN / 2 value
// columns + as many gate columns (the first CTA stages the value rows of the weight, the
// second the gate rows), one MMA computes both and the epilogue stores
// value * gelu_exact(gate).
// Roles in each CTA: warp 0 = TMA producer, warp 1 = TMEM owner and, in the first CTA of
// the pair, tcgen05.mma issuer for both, warps 2-9 = epilogue of the CTA's 128 rows (warp w
// owns TMEM lanes 32 * (w % 4)..; warps 2-5 take the first half of a tile's output columns,
// warps 6-9 the second half).
#include "gemm_plan.h"
#include "sdpa_internal.h"
#include "tc05.cuh"

namespace bdattn {
namespace {

constexpr int kPThreads = 320;
constexpr int kPRows = 256;                   // rows of a pair's tile
constexpr int kPChunk = 128 * 64 * 2;         // 128 rows x 64 columns: one TMA box of A
constexpr int kPStgBytes = 2048 + 512;        // one epilogue warp: staging, and 128 bias values as FP32
constexpr int kPPrefetch = 384;               // columns of K whose weights are asked for ahead
constexpr int kPGroup = 16;                   // row blocks of a group

// kN: accumulator columns of a tile, 256 or 128.  A stage of a CTA is two chunks (128 columns of K) of its
// 128 rows of A and two of its kN / 2 weight rows.
template <int kN>
struct PairCfg {
    static constexpr int kStages = kN == 256 ? 3 : 4;
    static constexpr int kBChunk = kN / 2 * 64 * 2;
    static constexpr int kStageBytes = 2 * kPChunk + 2 * kBChunk;
    static constexpr int kSmemBytes = kStages * kStageBytes + 8 * kPStgBytes + 256 + 3 * 128 * 4 + 1024;
    static constexpr int kHalf = kN / 2;      // output columns of an epilogue warp
    static_assert(kSmemBytes <= 227 * 1024, "shared memory of one CTA");
};

struct PairTile {
    int z, m0, n0;
};

// Output columns of one tile: kN, or half of them for GEGLU (the other accumulator
// columns hold the gate).
template <int kN>
__host__ __device__ __forceinline__ int pair_out_cols(const GemmProblem& p) { return p.geglu_offset > 0 ? kN / 2 : kN; }
__host__ __device__ __forceinline__ int pair_tiles_m(const GemmProblem& p) { return gemm_pair_row_tiles(p.tiles_m); }

template <int kN>
__device__ __forceinline__ PairTile pair_tile(const GemmArgs& g, int tile) {
    int z = 0;
    int local = tile;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int cnt = pair_tiles_m(g.p[i]) * (g.p[i].N / pair_out_cols<kN>(g.p[i]));
        if (z == i && local >= cnt) {
            local -= cnt;
            z = i + 1;
        }
    }
    const GemmProblem& p = z == 0 ? g.p[0] : (z == 1 ? g.p[1] : g.p[2]);
    const int cols = pair_out_cols<kN>(p), tm = pair_tiles_m(p), tn = p.N / cols;
    const int first = local / (kPGroup * tn) * kPGroup;      // first row block of the group
    const int rows = min(kPGroup, tm - first);
    local -= first * tn;
    PairTile t;
    t.z = z;
    t.n0 = (local / rows) * cols;
    t.m0 = (first + local % rows) * kPRows;
    return t;
}

template <bool kBf16>
__device__ __forceinline__ float load16(const void* base, long long i) {
    const uint16_t b = reinterpret_cast<const uint16_t*>(base)[i];
    return kBf16 ? __uint_as_float(static_cast<uint32_t>(b) << 16)
                 : __half2float(*reinterpret_cast<const __half*>(&b));
}

// The cos / sin values of 32 rows and 16 pairs, spread over a warp: lane -> (row lane / 4 of a group of eight,
// 16-byte piece lane % 4).
struct TablePiece {
    float4 c[4], s[4];
    __device__ __forceinline__ void load(const GemmProblem& p, int half_hd, int row0, int rows, int first_pair, int lane) {
        const long long at = static_cast<long long>(p.rope_row0 + row0 + (lane >> 2)) * half_hd + first_pair + (lane & 3) * 4;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i * 8 + (lane >> 2) < rows) {
                c[i] = __ldg(reinterpret_cast<const float4*>(p.cos + at + static_cast<long long>(i * 8) * half_hd));
                s[i] = __ldg(reinterpret_cast<const float4*>(p.sin + at + static_cast<long long>(i * 8) * half_hd));
            } else {
                c[i] = s[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        }
    }
    // This lane's own row, through 2 KB of shared memory: sixteen rows at a time.
    __device__ __forceinline__ void rows_of_lanes(uint8_t* stg, int lane, float (&cs)[16], float (&sn)[16]) const {
        const int tr = lane >> 2, tq = lane & 3;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                uint8_t* const row = stg + (i * 8 + tr) * 128;
                *reinterpret_cast<float4*>(row + ((tq ^ tr) << 4)) = c[2 * h + i];
                *reinterpret_cast<float4*>(row + (((tq + 4) ^ tr) << 4)) = s[2 * h + i];
            }
            __syncwarp();
            if ((lane >> 4) == h) {
                const uint8_t* const row = stg + (lane & 15) * 128;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 a = *reinterpret_cast<const float4*>(row + ((i ^ (lane & 7)) << 4));
                    const float4 b = *reinterpret_cast<const float4*>(row + (((i + 4) ^ (lane & 7)) << 4));
                    cs[4 * i] = a.x; cs[4 * i + 1] = a.y; cs[4 * i + 2] = a.z; cs[4 * i + 3] = a.w;
                    sn[4 * i] = b.x; sn[4 * i + 1] = b.y; sn[4 * i + 2] = b.z; sn[4 * i + 3] = b.w;
                }
            }
            __syncwarp();
        }
    }
};

// Epilogue of kW columns of a tile of whole heads of 128 or 64 columns; this thread owns one
// token's row of them: RMSNorm over the head and the rotary embedding are
// thread-local (src/dit/flux.cpp:462-469, src/dit/common.cpp:192-193).  Two
// passes over the accumulator (tensor memory reads are cheap): sum of squares
// per head first (the whole head, also where this warp finishes half of it), then 32 columns at a time.
// One loop for both head dims: two instantiations do not fit the registers.  gain_s: the gains of a head in
// shared memory as FP32, or null for no RMSNorm.  row0: the warp's first row.  tacc, bias_w and cbase: accumulator,
// bias and output of 128 columns, of which this warp takes c_first and on; tab: the table values of its
// first 32 columns, where there is RoPE.
template <bool kBf16, int kW>
__device__ __forceinline__ void epilogue_heads(const GemmProblem& p, uint32_t tacc, int row0, uint16_t* cbase,
                                               int c_first, const float* gain_s, const float* bias_w, uint8_t* stg,
                                               TablePiece& tab, int lane) {
    const int rows = min(32, p.M - row0);
    const int hd = p.n_tile;
    float inv0 = 1.0f, inv1 = 1.0f;
    if (gain_s != nullptr) {
        float ss0 = 0.0f, ss1 = 0.0f;
        // (kW = 64: the one head that the warp has columns of)
        const int c_norm = kW == 128 ? 0 : c_first & ~(hd - 1), n_norm = kW == 128 ? 128 : hd;
#pragma unroll 1
        for (int c = c_norm; c < c_norm + n_norm; c += 32) {
            uint32_t v[32];
            tmem_ld32(tacc + c, v);
            tmem_wait_ld();
            float f[32];
            add_bias(v, bias_w + c, f);
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
                ss0 = fmaf(f[i], f[i], ss0);
                ss1 = fmaf(f[i + 1], f[i + 1], ss1);
            }
            if (((c + 32) & (hd - 1)) == 0) {          // the head's last columns
                const float inv = rsqrtf((ss0 + ss1) / static_cast<float>(hd) + p.eps);
                if (kW == 64 || c < hd) inv0 = inv;
                else inv1 = inv;
                ss0 = ss1 = 0.0f;
            }
        }
    }
    const bool rope = p.cos != nullptr;
#pragma unroll 1
    for (int c = c_first; c < c_first + kW; c += 32) {
        const float inv = kW == 64 || c < hd ? inv0 : inv1;
        const float* const gain_c = gain_s + (c & (hd - 1));
        float cs[16], sn[16];
        if (rope) tab.rows_of_lanes(stg, lane, cs, sn);
        // sixteen columns at a time: with 32 the registers do not suffice
        uint32_t packed[16];
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            uint32_t v[16];
            tmem_ld16(tacc + c + hf * 16, v);
            tmem_wait_ld();
            float f[16];
            add_bias(v, bias_w + c + hf * 16, f);
            if (gain_s != nullptr) {
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    const float4 g = *reinterpret_cast<const float4*>(gain_c + hf * 16 + i);
                    f[i] *= inv * g.x;
                    f[i + 1] *= inv * g.y;
                    f[i + 2] *= inv * g.z;
                    f[i + 3] *= inv * g.w;
                }
            }
            if (rope) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float a0 = f[2 * i], b0 = f[2 * i + 1];
                    f[2 * i] = a0 * cs[hf * 8 + i] - b0 * sn[hf * 8 + i];
                    f[2 * i + 1] = a0 * sn[hf * 8 + i] + b0 * cs[hf * 8 + i];
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) packed[hf * 8 + i] = pack2<kBf16>(f[2 * i], f[2 * i + 1]);
        }
        if (rope && c + 32 < c_first + kW) tab.load(p, hd >> 1, row0, rows, ((c + 32) & (hd - 1)) >> 1, lane);
        store_words32(packed, stg, lane, cbase + c, p.ldc, rows, 32);
    }
}

// What the epilogue does with a tile: one instantiation each, so that each has the registers to itself and no
// code to fetch around (GEGLU 4096 x 320 -> 1280 16.2 -> 14.9 us, 1024 x 640 -> 2560 12.8 -> 12.0, QKV of 256 rows 18.6 -> 18.4).
enum PairEpilogue { kEpiPlain, kEpiGeglu, kEpiHeads };

template <bool kBf16, int kN, PairEpilogue kEpi>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmA1,
                 const __grid_constant__ CUtensorMap tmA2, const __grid_constant__ CUtensorMap tmB0,
                 const __grid_constant__ CUtensorMap tmB1, const __grid_constant__ CUtensorMap tmB2,
                 const GemmArgs g, const int total_tiles) {
    using C = PairCfg<kN>;
    constexpr int kPStages = C::kStages;
    constexpr int kPStageBytes = C::kStageBytes;
    extern __shared__ uint8_t gemm_pair_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gemm_pair_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
    uint8_t* stg_all = smem + kPStages * kPStageBytes;      // [8][kPStgBytes]
    uint64_t* bars = reinterpret_cast<uint64_t*>(stg_all + 8 * kPStgBytes);
    uint64_t* full = bars;                   // [kPStages]
    uint64_t* empty = bars + kPStages;       // [kPStages]
    uint64_t* acc_full = empty + kPStages;   // [2]
    uint64_t* acc_empty = acc_full + 2;      // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    float* gain_s = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + 256);   // [3][128]

    const int warp = warp_index();
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kPStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], 16);       // the epilogue warps of both CTAs
        }
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc_pair(tmem_slot, 2 * kN);
        tmem_relinquish_pair();
    }
    // The first tile of this pair: found before the wait for the kernel before this one, so that the first
    // look at the problems in the parameters is behind it too.
    const int rank = static_cast<int>(cluster_ctarank());
    const int pairs = static_cast<int>(gridDim.x) >> 1;
    const int first_tile = static_cast<int>(blockIdx.x) >> 1;
    const PairTile first = pair_tile<kN>(g, first_tile);
    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(first.z == 0 ? &tmA0 : (first.z == 1 ? &tmA1 : &tmA2));
        tma_prefetch_desc(first.z == 0 ? &tmB0 : (first.z == 1 ? &tmB1 : &tmB2));
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_relaxed();       // the peer signals these barriers too
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // only now: a dependent CTA that took tensor memory first could keep this one from getting its own
    dependents_may_launch();
    // While the kernel before this one ends, the first weights come into the L2 (the activations
    // may still be being written): once for the row blocks that share them.  No more than a few stages: all
    // of the first tile's weights took the first stages' bandwidth (QKV of 256 rows 26.6 -> 29.4 us).
    if (warp == 0 && first.m0 % (kPGroup * kPRows) == 0 && elect_one()) {
        const GemmProblem& p = first.z == 0 ? g.p[0] : (first.z == 1 ? g.p[1] : g.p[2]);
        const CUtensorMap* tmB = first.z == 0 ? &tmB0 : (first.z == 1 ? &tmB1 : &tmB2);
        const int row = first.n0 + rank * (p.geglu_offset > 0 ? p.geglu_offset : kN / 2);
        for (int x = 0; x < p.K && x < kPPrefetch; x += 64) tma_prefetch_l2_2d(tmB, x, row);
    }
    // barriers, tensor memory and descriptors are set up; from here on global memory is touched
    wait_for_prior_grid();

    if (warp == 0) {
        // ---------------------------------------------------- TMA producer
        // Both CTAs load their part of a stage; the copies of both complete on the first
        // CTA's barrier, where the MMA issuer waits.
        if (lane == 0) {
            int it = 0;          // stage uses so far, over all tiles of this pair
            int slot = 0;
            uint32_t phase = 1;  // parity that a fresh barrier passes
            bool ok = true;
            for (int tile = first_tile; ok && tile < total_tiles; tile += pairs) {
                const PairTile t = tile == first_tile ? first : pair_tile<kN>(g, tile);
                const CUtensorMap* tmA = t.z == 0 ? &tmA0 : (t.z == 1 ? &tmA1 : &tmA2);
                const CUtensorMap* tmB = t.z == 0 ? &tmB0 : (t.z == 1 ? &tmB1 : &tmB2);
                const int K = t.z == 0 ? g.p[0].K : (t.z == 1 ? g.p[1].K : g.p[2].K);
                const int geglu_off = t.z == 0 ? g.p[0].geglu_offset : (t.z == 1 ? g.p[1].geglu_offset : g.p[2].geglu_offset);
                const int chunks = (K + 63) / 64;
                const int a_row = t.m0 + rank * 128;
                const int b_row = t.n0 + rank * (geglu_off > 0 ? geglu_off : kN / 2);
                for (int c = 0; c < chunks; c += 2, ++it) {
                    ok = mbar_wait(&empty[slot], phase);
                    if (!ok) break;
                    uint8_t* st = smem + slot * kPStageBytes;
                    const int n = min(2, chunks - c);          // an odd last chunk stands alone
                    if (rank == 0) mbar_arrive_expect_tx(&full[slot], n * 2 * (kPChunk + C::kBChunk));
                    const uint32_t bar = mapa(smem_u32(&full[slot]), 0);
                    for (int i = 0; i < n; ++i) {
                        tma_load_2d_pair(st + i * kPChunk, tmA, bar, (c + i) * 64, a_row);
                        tma_load_2d_pair(st + 2 * kPChunk + i * C::kBChunk, tmB, bar, (c + i) * 64, b_row);
                    }
                    if (++slot == kPStages) { slot = 0; phase ^= 1; }
                }
            }
            if (ok) {
                // the last commits arrive here too: both CTAs see them before they end
                for (int i = max(0, it - kPStages); i < it; ++i)
                    mbar_wait(&empty[i % kPStages], static_cast<uint32_t>((i / kPStages) & 1));
            } else if (rank == 0) {
                // a wait ran out: let the copies in flight land before the CTAs end
                for (int i = max(0, it - kPStages); i < it; ++i)
                    mbar_wait(&full[i % kPStages], static_cast<uint32_t>((i / kPStages) & 1));
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------------------------------- MMA issuer (first CTA of the pair)
        constexpr uint32_t idesc = make_idesc_f16(kBf16 ? 1 : 0, kPRows, kN, 0, 0);
        const uint64_t a0 = make_smem_desc_sw128(smem_u32(smem), 16, 1024);
        const uint64_t b0 = make_smem_desc_sw128(smem_u32(smem) + 2 * kPChunk, 16, 1024);
        int slot = 0;
        uint32_t phase = 0;
        int ti = 0;              // tiles done by this pair
        bool ok = rank == 0;
        for (int tile = first_tile; ok && tile < total_tiles; tile += pairs, ++ti) {
            const PairTile t = tile == first_tile ? first : pair_tile<kN>(g, tile);
            const int K = t.z == 0 ? g.p[0].K : (t.z == 1 ? g.p[1].K : g.p[2].K);
            const int chunks = (K + 63) / 64;
            const int as = ti & 1;
            if (ti >= 2) {       // both epilogues must have drained this accumulator (tile ti - 2)
                ok = mbar_wait_warp(&acc_empty[as], static_cast<uint32_t>(((ti >> 1) - 1) & 1));
                if (!ok) break;
                tc_fence_after();
            }
            const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(as * kN);
            for (int c = 0; c < chunks; c += 2) {
                ok = mbar_wait_warp(&full[slot], phase);
                if (!ok) break;
                tc_fence_after();
                // (the lane is elected for each stage: with one thread running the loop GEGLU over
                // 9216 x 320 -> 1280 takes 28.4 us, this way 26.2)
                if (elect_one()) {
                    const uint64_t ad = a0 + slot * (kPStageBytes >> 4), bd = b0 + slot * (kPStageBytes >> 4);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        umma_ss_pair(d_tmem, ad + 2 * kk, bd + 2 * kk, idesc, (c > 0 || kk > 0) ? 1u : 0u);
                    if (c + 1 < chunks) {
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            umma_ss_pair(d_tmem, ad + (kPChunk >> 4) + 2 * kk, bd + (C::kBChunk >> 4) + 2 * kk, idesc, 1u);
                    }
                    umma_commit_pair(&empty[slot]);
                    if (c + 2 >= chunks) umma_commit_pair(&acc_full[as]);
                }
                __syncwarp();
                if (++slot == kPStages) { slot = 0; phase ^= 1; }
            }
        }
    } else {
        // -------------------------------------------------------- epilogue
        const int q = warp & 3;             // TMEM lane quarter of this warp
        const int half = (warp - 2) >> 2;   // which half of the tile's output columns
        uint8_t* const stg = stg_all + (warp - 2) * kPStgBytes;
        float* const bias_w = reinterpret_cast<float*>(stg + 2048);    // behind the output staging
        // RMSNorm gains of the three problems as FP32 for the 256 threads of these warps
        for (int idx = threadIdx.x - 64; idx < 3 * 128; idx += kPThreads - 64) {
            const GemmProblem& gp = idx < 128 ? g.p[0] : (idx < 256 ? g.p[1] : g.p[2]);
            const int i = idx & 127;
            float gv = 1.0f;
            if (gp.norm_rope && gp.gain != nullptr && i < gp.n_tile)
                gv = gp.gain_is_f32 ? __ldg(reinterpret_cast<const float*>(gp.gain) + i) : load16<kBf16>(gp.gain, i);
            gain_s[idx] = gv;
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        int ti = 0;
        bool ok = true;
        for (int tile = first_tile; tile < total_tiles; tile += pairs, ++ti) {
            const PairTile t = tile == first_tile ? first : pair_tile<kN>(g, tile);
            const GemmProblem& p = t.z == 0 ? g.p[0] : (t.z == 1 ? g.p[1] : g.p[2]);
            const int as = ti & 1;
            const int row0 = t.m0 + rank * 128 + q * 32;
            const int rows = min(32, p.M - row0);
            // a projection without norm and RoPE (V) has nothing but its bias to add
            const bool heads = kEpi == kEpiHeads && p.norm_rope && (p.gain != nullptr || p.cos != nullptr);
            const bool geglu = kEpi == kEpiGeglu && p.geglu_offset > 0;
            // where the 128 columns whose bias this warp keeps begin in the tile, and its own among them
            constexpr bool kWide = kN == 256;
            const int c_base = kWide ? half * 128 : 0, c_own = kWide ? 0 : half * C::kHalf;
            {
                // 128 bias values (GEGLU: 64 and those of their gates), fetched while the tile is computed
                const int lc = lane * 4;
                const long long at = geglu
                                         ? t.n0 + (c_base >> 1) + (lc < 64 ? lc : static_cast<long long>(p.geglu_offset) + lc - 64)
                                         : t.n0 + c_base + lc;
                float4 b = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (p.bias != nullptr)
                    b = make_float4(load16<kBf16>(p.bias, at), load16<kBf16>(p.bias, at + 1), load16<kBf16>(p.bias, at + 2),
                                    load16<kBf16>(p.bias, at + 3));
                *reinterpret_cast<float4*>(bias_w + lc) = b;
                __syncwarp();
            }
            TablePiece tab;
            if constexpr (kEpi == kEpiHeads)
                if (heads && p.cos != nullptr && rows > 0) tab.load(p, p.n_tile >> 1, row0, rows, (c_own & (p.n_tile - 1)) >> 1, lane);
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[as], static_cast<uint32_t>((ti >> 1) & 1)));
            if (!ok) break;
            tc_fence_after();
            const uint32_t tacc = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(as * kN);
            uint16_t* cbase = reinterpret_cast<uint16_t*>(p.C) + static_cast<long long>(row0) * p.ldc + t.n0;
            if (rows <= 0) {
                // rows past the matrix: nothing to store
            } else if (heads) {
                if constexpr (kEpi == kEpiHeads) {
                    const float* gs = p.gain != nullptr ? gain_s + t.z * 128 : nullptr;
                    epilogue_heads<kBf16, C::kHalf>(p, tacc + c_base, row0, cbase + c_base, c_own, gs, bias_w, stg, tab, lane);
                }
            } else if (geglu) {
                if constexpr (kEpi == kEpiGeglu) {
                    // values in the first half of the accumulator's columns, gates in the second
#pragma unroll 1
                    for (int c = (c_base + c_own) / 2; c < (c_base + c_own + C::kHalf) / 2; c += 32) {
                        const float* bv = bias_w + (c - c_base / 2);
                        uint32_t packed[16];
#pragma unroll
                        for (int hf = 0; hf < 2; ++hf) {
                            uint32_t v[16], gt[16];
                            tmem_ld16(tacc + c + hf * 16, v);
                            tmem_ld16(tacc + kN / 2 + c + hf * 16, gt);
                            tmem_wait_ld();
                            float f[16], gate[16];
                            add_bias(v, bv + hf * 16, f);
                            add_bias(gt, bv + 64 + hf * 16, gate);
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                packed[hf * 8 + i] = pack2<kBf16>(f[2 * i] * gelu_exact(gate[2 * i]),
                                                                  f[2 * i + 1] * gelu_exact(gate[2 * i + 1]));
                        }
                        store_words32(packed, stg, lane, cbase + c, p.ldc, rows, 32);
                    }
                }
            } else {
#pragma unroll 1
                for (int c = c_base + c_own; c < c_base + c_own + C::kHalf; c += 32) {
                    uint32_t v[32];
                    tmem_ld32(tacc + c, v);
                    tmem_wait_ld();
                    float f[32];
                    add_bias(v, bias_w + (c - c_base), f);
                    store_tile32<kBf16>(f, stg, lane, cbase + c, p.ldc, rows, 32);
                }
            }
            // this accumulator may be overwritten by the MMAs of tile ti + 2; where there is none, nobody
            // would wait for the arrival, and the first CTA could have left before it comes
            tc_fence_before();
            __syncwarp();
            if (lane == 0 && pair_acc_reused(tile, pairs, total_tiles))
                mbar_arrive_cluster(mapa(smem_u32(&acc_empty[as]), 0));
        }
    }

    tc_fence_before();
    // Neither CTA leaves while the other may still signal or read it.  (Every arrival at a peer's barrier
    // has been waited for by then: the barrier itself orders none.)
    cluster_sync_relaxed();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 2 * kN);
    }
}

}  // namespace

template <int kN>
static cudaError_t launch_gemm_pair_n(const GemmLaunch& L, cudaStream_t stream) {
    int total = 0;
    for (int i = 0; i < L.n_problems; ++i)
        total += pair_tiles_m(L.args.p[i]) * (L.args.p[i].N / pair_out_cols<kN>(L.args.p[i]));
    const int pairs = sm_count() / 2;
    const dim3 grid(static_cast<unsigned>(2 * (total < pairs ? total : pairs)));
    auto go = [&](auto kern) {
        cudaError_t e = set_max_smem_once(kern, PairCfg<kN>::kSmemBytes);
        if (e != cudaSuccess) return e;
        return launch_dependent(kern, grid, dim3(kPThreads), PairCfg<kN>::kSmemBytes, stream, L.tmA[0], L.tmA[1], L.tmA[2],
                                L.tmB[0], L.tmB[1], L.tmB[2], L.args, total);
    };
    bool geglu = false, heads = false;
    for (int i = 0; i < L.n_problems; ++i) {
        geglu = geglu || L.args.p[i].geglu_offset > 0;
        heads = heads || L.args.p[i].norm_rope;
    }
    if (geglu && heads) return cudaErrorInvalidValue;        // no entry point asks for both
    if (geglu) return L.bf16 ? go(gemm_pair_kernel<true, kN, kEpiGeglu>) : go(gemm_pair_kernel<false, kN, kEpiGeglu>);
    if (heads) return L.bf16 ? go(gemm_pair_kernel<true, kN, kEpiHeads>) : go(gemm_pair_kernel<false, kN, kEpiHeads>);
    return L.bf16 ? go(gemm_pair_kernel<true, kN, kEpiPlain>) : go(gemm_pair_kernel<false, kN, kEpiPlain>);
}

cudaError_t launch_gemm_pair(const GemmLaunch& L, int tile_cols, cudaStream_t stream) {
    return tile_cols == 128 ? launch_gemm_pair_n<128>(L, stream) : launch_gemm_pair_n<256>(L, stream);
}

}  // namespace bdattn
