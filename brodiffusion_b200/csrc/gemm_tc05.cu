// Linear layers on the sm_100a tensor cores:  C[M,N] = A[M,K] . B[N,K]^T (+ bias)
// with 16-bit operands, FP32 accumulation in tensor memory and a fused
// epilogue.  Weights are stored (out_features, in_features) as in the
// reference (src/unet_blocks.cpp:264-271), so both operands are K-major and
// are staged by TMA with the 128-byte swizzle.
//
// Up to three independent problems share one launch (blockIdx.z): the Q, K
// and V projections of one attention call.  A CTA computes one 128-row x
// n_tile-column tile:
//   warp 0     TMA producer (A tile 128 x 64, B tile n_tile x 64 per K block)
//   warp 1     tcgen05.mma issuer, owns the TMEM allocation
//   warps 2-5  epilogue: tcgen05.ld -> bias / GEGLU -> 16-byte stores
// Where the tiles leave SMs idle (the 64- and 256-token levels of a U-Net, short
// prompts), a cluster of up to eight CTAs shares one tile: each takes a part of the K
// blocks, the partial sums meet in distributed shared memory, and every CTA finishes
// 128 / split rows of the tile (kSplit).
//
// GEGLU mode (src/fused_transformer.cu:89-92,275-282): a second B tile from
// weight row n0 + D_out feeds a second accumulator and the epilogue stores
// value * gelu_exact(gate), so the (B, 2*D_out) intermediate never exists.
#include <cooperative_groups.h>
#include <type_traits>

#include "gemm_plan.h"
#include "sdpa_internal.h"
#include "tc05.cuh"

namespace bdattn {
namespace {

constexpr int kGemmThreads = 192;
constexpr int kGemmPrefetch = 20;            // K blocks whose weights are asked for ahead
constexpr int kGemmMaxStages = 8;
constexpr int kGemmABytes = 128 * 64 * 2;   // A stage
// A B (or gate) tile is n_tile rows x 128 B; a stage holds A, B and, for GEGLU,
// the gate tile, rounded up to the 1024-byte swizzle period.  Sizing the stage by
// the tile shape keeps a 64-column GEMM at 96 KB so that two CTAs share an SM.
__host__ __device__ inline int gemm_b_bytes(int n_tile) { return (n_tile * 128 + 1023) / 1024 * 1024; }
__host__ __device__ inline int gemm_stage_bytes(int n_tile, bool geglu) {
    return kGemmABytes + (geglu ? 2 : 1) * gemm_b_bytes(n_tile);
}

// Partial sums of a split tile in shared memory: row-major, four floats of padding per
// row so that both a thread per row and several threads per row read and write
// float4 without bank conflicts.
__host__ __device__ inline int gemm_red_ld(int n_tile) { return n_tile + 4; }

template <bool kBf16>
__device__ __forceinline__ float gemm_ld16(const void* base, long long i) {
    const uint16_t b = reinterpret_cast<const uint16_t*>(base)[i];
    return kBf16 ? __uint_as_float(static_cast<uint32_t>(b) << 16)
                 : __half2float(*reinterpret_cast<const __half*>(&b));
}

// Epilogue of a split tile.  Every CTA of the cluster holds a partial 128 x n_tile sum
// at the same shared-memory address; this one finishes its share of the rows, eight columns to a thread, so that
// eight threads read and write a whole row piece, and asks for
// all partial sums of a piece before it adds the first (a thread walking the columns of a row, one remote read
// behind the other, took 2 to 4 us; with the bias ahead 64 x 1280 x 1280 over four 5.3 -> 4.7 us, 1024 x 640 x 2560
// over two 13.4 -> 11.5).  Up to 64 rows are dealt out one by one, so that every CTA has some; more are
// taken as blocks (128 x 640 x 5120 over eight 7.8 us dealt out, 7.4; 64 x 1280 x 1280 4.7, 5.2 in blocks).  Of a narrow
// tile no thread gets columns that do not exist: 5251 x 8 x 1064 8.0 -> 6.9 us, 113 x 8 x 680 5.4 -> 4.2.
template <bool kBf16>
__device__ __forceinline__ void epilogue_split(const GemmProblem& p, cooperative_groups::cluster_group& cluster,
                                               float* red, const float* bias_s, int split, int part, int tid, int m0, int n0) {
    const int ld = gemm_red_ld(p.n_tile);
    const int n_valid = min(p.n_tile, p.N - n0);           // a multiple of eight
    const int sh = n_valid > 64 ? 4 : n_valid > 32 ? 3 : n_valid > 16 ? 2 : n_valid > 8 ? 1 : 0;
    const int rows = min(128, p.M - m0);
    const bool dealt = rows <= 64;
    const float* src[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) src[k] = cluster.map_shared_rank(red, min(k, split - 1));
#pragma unroll 2
    for (int i = tid; i < (128 / split) << sh; i += 128) {
        const int j = i >> sh, c = (i & ((1 << sh) - 1)) * 8;
        const int r = dealt ? part + split * j : part * (128 / split) + j;
        if (r >= rows || c >= n_valid) continue;
        float4 u[8], v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (k < split) {
                const float4* at = reinterpret_cast<const float4*>(src[k] + r * ld + c);
                u[k] = at[0];
                v[k] = at[1];
            }
        }
        float f[8] = {};
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (k < split) {
                f[0] += u[k].x; f[1] += u[k].y; f[2] += u[k].z; f[3] += u[k].w;
                f[4] += v[k].x; f[5] += v[k].y; f[6] += v[k].z; f[7] += v[k].w;
            }
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] += bias_s[c + e];
        uint4 w;
        w.x = pack2<kBf16>(f[0], f[1]); w.y = pack2<kBf16>(f[2], f[3]);
        w.z = pack2<kBf16>(f[4], f[5]); w.w = pack2<kBf16>(f[6], f[7]);
        *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.C) + static_cast<long long>(m0 + r) * p.ldc + n0 + c) = w;
    }
}

// One instantiation per epilogue (plain, GEGLU, norm + RoPE, plain split tiles): the
// GEGLU and the norm + RoPE code are long, and an epilogue that only branches around them
// spent more time fetching instructions than storing (5.6 us for one 128 x 128 tile
// against 2.3 us).
template <bool kBf16, bool kGeglu, bool kNormRope, bool kSplit>
__global__ void __launch_bounds__(kGemmThreads)
gemm_tc05_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmA1,
                 const __grid_constant__ CUtensorMap tmA2, const __grid_constant__ CUtensorMap tmB0,
                 const __grid_constant__ CUtensorMap tmB1, const __grid_constant__ CUtensorMap tmB2,
                 const GemmArgs g) {
    const int split = kSplit ? g.split : 1;
    const int z = kSplit ? static_cast<int>(blockIdx.z) / split : static_cast<int>(blockIdx.z);
    const int part = kSplit ? static_cast<int>(blockIdx.z) % split : 0;    // the cluster spans `split` CTAs of z
    const GemmProblem& p = z == 0 ? g.p[0] : (z == 1 ? g.p[1] : g.p[2]);
    const CUtensorMap* tmA = z == 0 ? &tmA0 : (z == 1 ? &tmA1 : &tmA2);
    const CUtensorMap* tmB = z == 0 ? &tmB0 : (z == 1 ? &tmB1 : &tmB2);
    const int tile_n = blockIdx.x;
    const int tile_m = blockIdx.y;
    if (tile_n >= p.tiles_n || tile_m >= p.tiles_m) return;

    extern __shared__ uint8_t gemm_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gemm_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
    const int kGemmStages = g.stages;
    const int kGemmBBytes = gemm_b_bytes(g.n_tile_max);
    const int kGemmStageBytes = gemm_stage_bytes(g.n_tile_max, g.any_geglu != 0);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kGemmStages * kGemmStageBytes);
    uint64_t* full = bars;
    uint64_t* empty = bars + kGemmMaxStages;
    uint64_t* acc_done = empty + kGemmMaxStages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_done + 1);
    float* bias_s = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + 256);    // [128] and [128] of the gate

    const int warp = warp_index();
    const int lane = threadIdx.x & 31;
    const int k_all = gemm_k_blocks(p.K);
    const int k_begin = kSplit ? gemm_part_begin(k_all, split, part) : 0;
    const int k_blocks = (kSplit ? gemm_part_begin(k_all, split, part + 1) : k_all) - k_begin;
    const int n0 = tile_n * p.n_tile;
    const int m0 = tile_m * 128;
    const bool geglu = kGeglu && p.geglu_offset > 0;
    constexpr uint32_t kTmemCols = kGeglu ? 256 : 128;     // the gate accumulator sits 128 columns up

    if (threadIdx.x == 0) {
        for (int s = 0; s < kGemmStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(acc_done, 1);
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // only now: a dependent CTA that took tensor memory first could keep this one from getting its own
    if (!kNormRope || g.one_wave) dependents_may_launch();
    // While the kernel before this one ends, this tile's weights come into the L2 (its activations may still
    // be being written): once for the row tiles that share them (the eleven calls of a 64-token block of 1280
    // channels, weights cold, 62.2 -> 59.4 us).
    if (warp == 0 && tile_m == 0 && elect_one()) {
        for (int kb = 0; kb < k_blocks && kb < kGemmPrefetch; ++kb) {
            tma_prefetch_l2_2d(tmB, (k_begin + kb) * 64, n0);
            if (geglu) tma_prefetch_l2_2d(tmB, (k_begin + kb) * 64, n0 + p.geglu_offset);
        }
    }
    wait_for_prior_grid();

    if (warp == 0) {
        if (elect_one()) {
            const uint32_t bytes = kGemmABytes + (geglu ? 2u : 1u) * static_cast<uint32_t>(p.n_tile) * 128u;
            bool ok = true;
            int issued = 0;
            int slot = 0;
            uint32_t phase = 1;          // parity that a fresh barrier passes
            for (int kb = 0; kb < k_blocks; ++kb) {
                ok = mbar_wait(&empty[slot], phase);
                if (!ok) break;
                uint8_t* st = smem + slot * kGemmStageBytes;
                mbar_arrive_expect_tx(&full[slot], bytes);
                const int x = (k_begin + kb) * 64;
                tma_load_2d(st, tmA, &full[slot], x, m0);
                tma_load_2d(st + kGemmABytes, tmB, &full[slot], x, n0);
                if (geglu) tma_load_2d(st + kGemmABytes + kGemmBBytes, tmB, &full[slot], x, n0 + p.geglu_offset);
                issued = kb + 1;
                if (++slot == kGemmStages) { slot = 0; phase ^= 1; }
            }
            if (!ok) {
                for (int kb = max(0, issued - kGemmStages); kb < issued; ++kb)
                    mbar_wait(&full[kb % kGemmStages], static_cast<uint32_t>((kb / kGemmStages) & 1));
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // One elected thread runs the whole loop (with the warp in step and the lane elected for each
        // block 576 x 1280 x 1280 takes 7.3 us, this way 6.5).  The slot and its parity are counted on, a
        // division by the runtime ring size cost more than the four MMAs.
        const uint32_t idesc = make_idesc_f16(kBf16 ? 1 : 0, 128, p.n_tile, 0, 0);
        const uint64_t a0 = make_smem_desc_sw128(smem_u32(smem), 16, 1024);
        const uint64_t b0 = make_smem_desc_sw128(smem_u32(smem) + kGemmABytes, 16, 1024);
        const uint32_t stage_units = static_cast<uint32_t>(kGemmStageBytes) >> 4;   // descriptors count 16 bytes
        const uint32_t gate_units = static_cast<uint32_t>(kGemmBBytes) >> 4;
        if (elect_one()) {
            int slot = 0;
            uint32_t phase = 0;
            for (int kb = 0; kb < k_blocks; ++kb) {
                if (!mbar_wait(&full[slot], phase)) break;
                tc_fence_after();
                const uint64_t ad = a0 + slot * stage_units, bd = b0 + slot * stage_units;
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    umma_ss(tmem_base, ad + 2 * kk, bd + 2 * kk, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
                    if (geglu) umma_ss(tmem_base + 128, ad + 2 * kk, bd + gate_units + 2 * kk, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
                }
                umma_commit(&empty[slot]);
                if (kb == k_blocks - 1) umma_commit(acc_done);
                if (++slot == kGemmStages) { slot = 0; phase ^= 1; }
            }
        }
        __syncwarp();
    } else {
        // epilogue: warp w reads TMEM lanes 32 * (w % 4) ..
        const int q = warp & 3;
        const int row = m0 + q * 32 + lane;
        if (!kNormRope || !p.norm_rope) {
            // the tile's bias, zero where there is none, while the tile is computed
            const int t = static_cast<int>(threadIdx.x) - 64;
            const bool on = p.bias != nullptr && t < p.n_tile && n0 + t < p.N;
            bias_s[t] = on ? gemm_ld16<kBf16>(p.bias, n0 + t) : 0.0f;
            if constexpr (kGeglu)
                bias_s[128 + t] = on && geglu ? gemm_ld16<kBf16>(p.bias, static_cast<long long>(n0) + p.geglu_offset + t) : 0.0f;
            asm volatile("bar.sync 1, 128;" ::: "memory");
        }
        bool ok = mbar_wait(acc_done, 0);
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
        const uint32_t tacc = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
        uint16_t* crow0 = reinterpret_cast<uint16_t*>(p.C) + static_cast<long long>(m0 + q * 32) * p.ldc + n0;
        uint16_t* crow = crow0 + static_cast<long long>(lane) * p.ldc;
        const int n_valid = min(p.n_tile, p.N - n0);      // a ragged last tile stops at the matrix edge
        if constexpr (kSplit) {
            // partial sums to shared memory: the ring is at rest, its last MMA has completed
            float* rrow = reinterpret_cast<float*>(smem) + (q * 32 + lane) * gemm_red_ld(p.n_tile);
#pragma unroll 1
            for (int c = 0; ok && c < p.n_tile; c += 32) {
                uint32_t v[32];
                tmem_ld32(tacc + c, v);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    *reinterpret_cast<uint4*>(rrow + c + 4 * i) = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            }
        } else if (kNormRope && ok && p.norm_rope) {
            // The tile is one head and this thread holds one token's row of it:
            // RMSNorm over the head and the rotary embedding are thread-local
            // (src/dit/flux.cpp:462-469 + src/dit/common.cpp:192-193 fused into
            // the projection, so Q and K never travel to HBM un-normalised).
            float f[128];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (c * 32 < p.n_tile) {
                    uint32_t v[32];
                    tmem_ld32(tacc + c * 32, v);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        float x = __uint_as_float(v[i]);
                        if (p.bias != nullptr) {
                            const uint16_t b = reinterpret_cast<const uint16_t*>(p.bias)[n0 + c * 32 + i];
                            x += kBf16 ? __uint_as_float(static_cast<uint32_t>(b) << 16)
                                       : __half2float(*reinterpret_cast<const __half*>(&b));
                        }
                        f[c * 32 + i] = x;
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) f[c * 32 + i] = 0.0f;
                }
            }
            if (p.gain != nullptr) {
                float ss = 0.0f;
#pragma unroll
                for (int i = 0; i < 128; ++i) ss = fmaf(f[i], f[i], ss);
                const float inv = rsqrtf(ss / static_cast<float>(p.n_tile) + p.eps);
#pragma unroll
                for (int i = 0; i < 128; ++i) {
                    if (i < p.n_tile) {
                        float gv;
                        if (p.gain_is_f32) gv = __ldg(reinterpret_cast<const float*>(p.gain) + i);
                        else {
                            const uint16_t b = reinterpret_cast<const uint16_t*>(p.gain)[i];
                            gv = kBf16 ? __uint_as_float(static_cast<uint32_t>(b) << 16)
                                       : __half2float(*reinterpret_cast<const __half*>(&b));
                        }
                        f[i] *= inv * gv;
                    }
                }
            }
            if (p.cos != nullptr && row < p.M) {
                const long long t = static_cast<long long>(p.rope_row0 + row) * (p.n_tile / 2);
#pragma unroll
                for (int i = 0; i < 64; ++i) {
                    if (2 * i < p.n_tile) {
                        const float cv = __ldg(p.cos + t + i), sv = __ldg(p.sin + t + i);
                        const float a0 = f[2 * i], b0 = f[2 * i + 1];
                        f[2 * i] = a0 * cv - b0 * sv;
                        f[2 * i + 1] = a0 * sv + b0 * cv;
                    }
                }
            }
            if (row < p.M) {
#pragma unroll
                for (int v8 = 0; v8 < 16; ++v8) {
                    if (v8 * 8 < p.n_tile) {
                        uint4 w;
                        w.x = pack2<kBf16>(f[v8 * 8 + 0], f[v8 * 8 + 1]);
                        w.y = pack2<kBf16>(f[v8 * 8 + 2], f[v8 * 8 + 3]);
                        w.z = pack2<kBf16>(f[v8 * 8 + 4], f[v8 * 8 + 5]);
                        w.w = pack2<kBf16>(f[v8 * 8 + 6], f[v8 * 8 + 7]);
                        *reinterpret_cast<uint4*>(crow + v8 * 8) = w;
                    }
                }
            }
        } else if (ok) {
            for (int c = 0; c < n_valid; c += 32) {
                uint32_t v[32], gt[32];
                tmem_ld32(tacc + c, v);
                if (geglu) tmem_ld32(tacc + 128 + c, gt);
                tmem_wait_ld();
                float f[32];
                add_bias(v, bias_s + c, f);
                if constexpr (kGeglu) {
                    if (geglu) {
                        float gate[32];
                        add_bias(gt, bias_s + 128 + c, gate);
#pragma unroll
                        for (int i = 0; i < 32; ++i) f[i] *= gelu_exact(gate[i]);
                    }
                }
                // (the ring is at rest, its last MMA has completed: it holds the staging)
                store_tile32<kBf16>(f, smem + q * 2048, lane, crow0 + c, p.ldc, p.M - m0 - q * 32, n_valid - c);
            }
        }
    }

    if constexpr (kSplit) {
        namespace cg = cooperative_groups;
        cg::cluster_group cluster = cg::this_cluster();
        cluster_sync();
        if (warp >= 2)
            epilogue_split<kBf16>(p, cluster, reinterpret_cast<float*>(smem), bias_s, split, part,
                                  static_cast<int>(threadIdx.x) - 64, m0, n0);
        cluster_sync_relaxed();      // the peers' shared memory stays until everyone has read it
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

}  // namespace

cudaError_t launch_gemm_tc05(const GemmLaunch& L, cudaStream_t stream) {
    int tn = 0, tm = 0, nt_max = 16, any_geglu = 0, any_norm_rope = 0, k_max = 0;
    // a CTA without a K block would wait for an accumulator that nobody computes; the epilogues of GEGLU and
    // norm + RoPE take whole tiles
    for (int i = 0; i < L.n_problems; ++i) {
        const GemmProblem& p = L.args.p[i];
        if (L.args.split > gemm_k_blocks(p.K) || (L.args.split > 1 && (p.geglu_offset > 0 || p.norm_rope != 0)))
            return cudaErrorInvalidValue;
    }
    for (int i = 0; i < L.n_problems; ++i) {
        const GemmProblem& p = L.args.p[i];
        tn = p.tiles_n > tn ? p.tiles_n : tn;
        tm = p.tiles_m > tm ? p.tiles_m : tm;
        nt_max = p.n_tile > nt_max ? p.n_tile : nt_max;
        k_max = p.K > k_max ? p.K : k_max;
        any_geglu |= p.geglu_offset > 0 ? 1 : 0;
        any_norm_rope |= p.norm_rope ? 1 : 0;
    }
    GemmArgs args = L.args;
    args.n_tile_max = nt_max;
    args.any_geglu = any_geglu;
    const long long ctas = static_cast<long long>(tn) * tm * L.n_problems * args.split;
    // With norm + RoPE the CTAs of Q and K are the slow ones and come first, those of V fill up; the next
    // kernel's CTAs in the slots of the first finishers would undo that order for a kernel of this
    // kind (4096 rows, 2 heads of 64, K = 1024: 28.8 us a launch, 20.7 kept back).
    args.one_wave = ctas <= sm_count();
    const int stage = gemm_stage_bytes(nt_max, any_geglu != 0);
    // three stages with the gate tile: the stage ring stays below 114 KB and two CTAs fit per SM
    args.stages = any_geglu ? 3 : 4;
    if (ctas <= sm_count()) {
        // a CTA has its SM to itself: the ring may take all of the shared memory
        args.stages = 192 * 1024 / stage < kGemmMaxStages ? 192 * 1024 / stage : kGemmMaxStages;
    } else if (!any_geglu && k_max <= 512 && args.split == 1) {
        // Short K and more tiles than SMs: a ring of two (64 KB) lets up to three CTAs share an SM,
        // so that one CTA's epilogue runs under the others' loads (4096 x 320 -> 960: 18.1 -> 12.2 us).
        args.stages = 2;
    }
    const int smem = args.stages * stage + 256 + 1024 + 1024;    // barriers, bias, alignment
    const dim3 grid(static_cast<unsigned>(tn), static_cast<unsigned>(tm),
                    static_cast<unsigned>(L.n_problems * args.split));
    cudaError_t e = cudaSuccess;
    auto go = [&](auto kern) {
        e = set_max_smem_once(kern, 227 * 1024);
        if (e != cudaSuccess) return;
        e = launch_dependent_cluster(kern, grid, dim3(kGemmThreads), smem, stream, dim3(1, 1, args.split), L.tmA[0],
                                     L.tmA[1], L.tmA[2], L.tmB[0], L.tmB[1], L.tmB[2], args);
    };
    auto pick = [&](auto bf16) {
        constexpr bool kB = decltype(bf16)::value;
        if (any_norm_rope) go(gemm_tc05_kernel<kB, false, true, false>);        // never split
        else if (any_geglu) go(gemm_tc05_kernel<kB, true, false, false>);
        else if (args.split > 1) go(gemm_tc05_kernel<kB, false, false, true>);
        else go(gemm_tc05_kernel<kB, false, false, false>);
    };
    if (L.bf16) pick(std::true_type{});
    else pick(std::false_type{});
    return e;
}

}  // namespace bdattn
