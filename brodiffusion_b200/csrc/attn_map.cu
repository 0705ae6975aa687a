// Head-averaged softmax map for traced attention.
//
// The reference's trace mode recomputes attention on the host to expose the
// softmax (dit::joint_attention_traced, src/dit/common.cpp:198-329, keeps the
// image-query x text-key block, src/dit/flux.cpp:505-508; the U-Net uses
// brotensor::cross_attention_forward_with_attn, src/unet_blocks.cpp:282-290).
// Here the attention kernel writes each row's softmax statistics (reference
// maximum and row sum) and this kernel evaluates only the requested block of
// the map from them:  avg_h exp2((q.k * scale + bias) * log2e - m) / l.
//
// One cluster of CTAs owns 128 query rows x 64 keys of the map; its CTAs take the
// heads in turn, so that a small block (32 such tiles at 1024 rows x 256 keys) still
// fills the SMs, and add up their sums through distributed shared memory.  Per head:
// TMA brings the Q and K tile of the head (zero-filled past head_dim), one lane issues
// S = Q.K^T into one of two tensor-memory buffers, and eight warps (two threads per query
// row) turn the scores into weights and add them to 32 registers each; the bias of the tile
// and its visibility bits are fetched once, not per head.
// A tile is a chain of latencies: with four warps, bias rows fetched in eight batches, a test per key for its
// visibility and remote sums read by four bytes it took 35000 cycles at 1024 x 256, 24 heads of 128 (bias 9000, bits
// 4000, six heads 11000, sums and stores 10000), 21 of the 54 us of a traced call; now 10 of 40.
#include <cooperative_groups.h>

#include "sdpa_internal.h"
#include "tc05.cuh"

namespace bdattn {
namespace {

constexpr int kMapRows = 128;
constexpr int kMapKeys = 64;
constexpr int kMapStages = 3;
constexpr int kMapThreads = 320;          // TMA warp, MMA warp, eight warps for the rows: 32 rows x 32 keys each
constexpr uint32_t kMapTmemCols = 128;    // two score buffers of 64 columns
constexpr int kMapQChunk = kMapRows * 128;   // 64 head columns of the Q tile
constexpr int kMapKChunk = kMapKeys * 128;

template <int HD>
struct MapCfg {
    static constexpr int kChunks = HD / 64;
    static constexpr int kStageBytes = kChunks * (kMapQChunk + kMapKChunk);
    // the ring also holds the CTA's 128 x 64 sums on their way out
    static constexpr int kSmemBytes = kMapStages * kStageBytes + 128 + kMapKeys * 4 + 1024;
    // with a bias: 32 x 32 values of it for each of the row warps
    static constexpr int kBiasBytes = 8 * 4096;
};

constexpr int kMapSumLd = kMapKeys + 4;       // floats of a row of sums: no bank conflicts, a thread per row or per 16 bytes

// The first n of 32 bits.
__device__ __forceinline__ uint32_t first_bits(int n) { return n >= 32 ? 0xffffffffu : (n <= 0 ? 0u : (1u << n) - 1u); }

template <int HD, bool kBf16>
__global__ void __launch_bounds__(kMapThreads, 1)
attn_map_kernel(const __grid_constant__ CUtensorMap tmQ0, const __grid_constant__ CUtensorMap tmQ1,
                const __grid_constant__ CUtensorMap tmK0, const __grid_constant__ CUtensorMap tmK1,
                const AttnMapArgs a) {
    using C = MapCfg<HD>;
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int cs = static_cast<int>(gridDim.z);         // the cluster spans the grid's z
    const int rank = static_cast<int>(blockIdx.z);
    extern __shared__ uint8_t map_raw[];
    // (the same offset in every CTA of the cluster: the sums are read at the peers' address)
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(map_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kMapStages * C::kStageBytes);
    uint64_t* full = bars;
    uint64_t* empty = full + kMapStages;
    uint64_t* s_full = empty + kMapStages;   // [2]
    uint64_t* s_free = s_full + 2;           // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(s_free + 2);
    float* ks_s = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + 128);   // [kMapKeys]

    const int warp = warp_index();
    const int lane = threadIdx.x & 31;
    const int kt = blockIdx.x, rt = blockIdx.y;
    const int kseg = kt >= a.key_tiles0 ? 1 : 0;
    const int key_local0 = (kseg ? kt - a.key_tiles0 : kt) * kMapKeys;
    const int key_base = (kseg ? a.kv_rows[0] : 0) + key_local0;               // global key index of column 0
    const int keys = min(kMapKeys, (kseg ? a.key_n[1] : a.key_n[0]) - key_local0);
    const int rseg = rt >= a.row_tiles0 ? 1 : 0;
    const int row_off = (rseg ? rt - a.row_tiles0 : rt) * kMapRows;
    const int rows = min(kMapRows, (rseg ? a.row_n[1] : a.row_n[0]) - row_off);
    const int row_local0 = (rseg ? a.row_lo[1] : a.row_lo[0]) + row_off;
    const int row_base = (rseg ? a.q_rows[0] : 0) + row_local0;                // global query index of row 0
    const int n_heads = rank < a.num_heads ? (a.num_heads - rank + cs - 1) / cs : 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kMapStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&s_full[b], 1);
            mbar_init(&s_free[b], 8);
        }
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, kMapTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // only now: a dependent CTA that took tensor memory first could keep this one from getting its own
    dependents_may_launch();
    wait_for_prior_grid();

    if (a.key_scale != nullptr) {
        if (threadIdx.x < kMapKeys)
            ks_s[threadIdx.x] = static_cast<int>(threadIdx.x) < keys ? __ldg(a.key_scale + key_base + threadIdx.x) : 1.0f;
        __syncthreads();
    }

    float acc[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) acc[c] = 0.0f;
    const int row = (warp & 3) * 32 + lane;
    const int col0 = ((warp - 2) >> 2) * 32;       // the keys of this warp (warps 2-9)
    const int qi = row_base + row;

    if (warp == 0) {
        if (elect_one()) {
            const CUtensorMap* tmQ = rseg ? &tmQ1 : &tmQ0;
            const CUtensorMap* tmK = kseg ? &tmK1 : &tmK0;
            bool ok = true;
            int issued = 0;
            for (int i = 0; i < n_heads; ++i) {
                const int s = i % kMapStages;
                if (i >= kMapStages) ok = mbar_wait(&empty[s], static_cast<uint32_t>((i / kMapStages - 1) & 1));
                if (!ok) break;
                const int h = rank + i * cs;
                uint8_t* st = smem + s * C::kStageBytes;
                mbar_arrive_expect_tx(&full[s], C::kStageBytes);
                for (int c = 0; c < C::kChunks; ++c) {
                    tma_load_4d(st + c * kMapQChunk, tmQ, &full[s], c * 64, h, row_local0, 0);
                    tma_load_4d(st + C::kChunks * kMapQChunk + c * kMapKChunk, tmK, &full[s], c * 64, h, key_local0, 0);
                }
                issued = i + 1;
            }
            if (!ok) {
                // a wait ran out: let the copies in flight land before the CTA ends
                for (int i = max(0, issued - kMapStages); i < issued; ++i)
                    mbar_wait(&full[i % kMapStages], static_cast<uint32_t>((i / kMapStages) & 1));
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        constexpr uint32_t idesc = make_idesc_f16(kBf16 ? 1 : 0, kMapRows, kMapKeys, 0, 0);
        if (elect_one()) {
            bool ok = true;
            for (int i = 0; ok && i < n_heads; ++i) {
                const int s = i % kMapStages, b = i & 1;
                if (i >= 2) ok = mbar_wait(&s_free[b], static_cast<uint32_t>((i / 2 - 1) & 1));
                if (ok) ok = mbar_wait(&full[s], static_cast<uint32_t>((i / kMapStages) & 1));
                if (!ok) break;
                tc_fence_after();
                const uint32_t qa = smem_u32(smem + s * C::kStageBytes);
                const uint32_t kb = qa + C::kChunks * kMapQChunk;
#pragma unroll
                for (int kk = 0; kk < HD / 16; ++kk) {
                    umma_ss(tmem_base + b * kMapKeys,
                            make_smem_desc_sw128(qa + (kk >> 2) * kMapQChunk + (kk & 3) * 32, 16, 1024),
                            make_smem_desc_sw128(kb + (kk >> 2) * kMapKChunk + (kk & 3) * 32, 16, 1024), idesc,
                            kk > 0 ? 1u : 0u);
                }
                umma_commit(&empty[s]);
                umma_commit(&s_full[b]);
            }
        }
        __syncwarp();
    } else {
        const uint32_t tS = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + static_cast<uint32_t>(col0);
        const bool row_ok = row < rows;
        // the row's bias in log2 units, and which of its 32 keys it sees (the attention kernel's
        // rules: a masked key has weight 0)
        const float log2e = 1.4426950408889634f;
        float bias[32];
        uint8_t* const bs = reinterpret_cast<uint8_t*>(ks_s + kMapKeys) + (warp - 2) * 4096;
        if (a.bias != nullptr) {
            const int kg = key_base + col0;
            copy_rows32(bs, a.bias + kg, a.bias_ld, row_base + (warp & 3) * 32 - a.bias_row0, a.bias_rows,
                        min(keys - col0, a.bias_cols - kg), lane);
        }
        uint32_t vis = first_bits(keys - col0);
        if (a.mask_mode == 1) vis &= first_bits(qi + a.q_offset - key_base - col0 + 1);
        if (a.key_mask != nullptr) {
            const float seen = col0 + lane < keys ? __ldg(a.key_mask + key_base + col0 + lane) : 0.0f;
            vis &= __ballot_sync(0xffffffffu, seen != 0.0f);
        }
        if (!row_ok) vis = 0u;
        const float* st = a.lse + (static_cast<long long>(rank) * a.lq_total + qi) * 2;
        const long long st_step = static_cast<long long>(cs) * a.lq_total * 2;
        float2 stat = make_float2(0.0f, 0.0f);
        if (row_ok && n_heads > 0) stat = make_float2(st[0], st[1]);
        if (a.bias != nullptr) {
            cp_async_wait_all();
            __syncwarp();
        }
#pragma unroll
        for (int c = 0; c < 32; c += 4) {
            const float4 b = a.bias != nullptr ? row_piece32(bs, lane, c >> 2) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            bias[c] = b.x * log2e; bias[c + 1] = b.y * log2e; bias[c + 2] = b.z * log2e; bias[c + 3] = b.w * log2e;
        }
        bool ok = true;
        for (int i = 0; i < n_heads; ++i) {
            const int b = i & 1;
            const float m2 = stat.x;
            const float inv_l = stat.y > 0.0f ? 1.0f / stat.y : 0.0f;
            st += st_step;
            if (row_ok && i + 1 < n_heads) stat = make_float2(st[0], st[1]);
            // a row whose reference maximum is -inf saw no key: its map row is zero
            const uint32_t bits = m2 != -INFINITY ? vis : 0u;
            ok = __all_sync(0xffffffffu, mbar_wait(&s_full[b], static_cast<uint32_t>((i >> 1) & 1)));
            if (!ok) break;
            tc_fence_after();
            uint32_t v[32];
            tmem_ld32(tS + b * kMapKeys, v);
            tmem_wait_ld();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_free[b]);
#pragma unroll
            for (int c = 0; c < 32; ++c) {
                float x = __uint_as_float(v[c]);
                if (a.key_scale != nullptr) x *= ks_s[col0 + c];
                const float p = fast_exp2(fmaf(x, a.scale_log2, bias[c]) - m2) * inv_l;
                acc[c] += ((bits >> c) & 1u) != 0u ? p : 0.0f;
            }
        }
    }

    // Sums to shared memory (the ring is at rest: every MMA that read it has completed); then every CTA of the
    // cluster adds up and stores its share of the columns, four to a thread.
    const float inv_h = 1.0f / static_cast<float>(a.num_heads);
    float* const out = a.map + static_cast<long long>(row_base - a.map_row0) * a.map_ld + key_base;
    float* const red = reinterpret_cast<float*>(smem);
    if (warp >= 2) {
#pragma unroll
        for (int c = 0; c < 32; c += 4)
            *reinterpret_cast<float4*>(red + row * kMapSumLd + col0 + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
    }
    if (cs > 1) cluster_sync();
    else __syncthreads();
    if (warp >= 2) {
        const float* src[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) src[k] = cs > 1 ? cluster.map_shared_rank(red, min(k, cs - 1)) : red;
        const int units = kMapKeys / 4 / cs;                                   // a power of two, as cs is
        const bool vec = (a.map_ld & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
#pragma unroll 2
        for (int i = static_cast<int>(threadIdx.x) - 64; i < kMapRows * units; i += 256) {
            const int r = i / units, c = (rank * units + (i & (units - 1))) * 4;
            if (r >= rows || c >= keys) continue;
            float4 u[8];
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (k < cs) u[k] = *reinterpret_cast<const float4*>(src[k] + r * kMapSumLd + c);
            float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (k < cs) { sum.x += u[k].x; sum.y += u[k].y; sum.z += u[k].z; sum.w += u[k].w; }
            sum.x *= inv_h; sum.y *= inv_h; sum.z *= inv_h; sum.w *= inv_h;
            float* const at = out + r * a.map_ld + c;
            if (vec && c + 4 <= keys) {
                *reinterpret_cast<float4*>(at) = sum;
            } else {
                at[0] = sum.x;
                if (c + 1 < keys) at[1] = sum.y;
                if (c + 2 < keys) at[2] = sum.z;
                if (c + 3 < keys) at[3] = sum.w;
            }
        }
    }
    if (cs > 1) cluster_sync_relaxed();      // the peers' shared memory stays until everyone has read it

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kMapTmemCols);
    }
}

template <int HD, bool kBf16>
cudaError_t launch_map_t(const AttnMapLaunch& L, cudaStream_t stream) {
    auto kern = attn_map_kernel<HD, kBf16>;
    const int smem = MapCfg<HD>::kSmemBytes + (L.args.bias != nullptr ? MapCfg<HD>::kBiasBytes : 0);
    cudaError_t e = set_max_smem_once(kern, smem);
    if (e != cudaSuccess) return e;
    // heads are spread over a cluster while the grid stays within one wave
    const long long tiles = static_cast<long long>(L.key_tiles) * L.row_tiles;
    unsigned cs = 1;
    while (cs < 8 && tiles * cs * 2 <= sm_count() && L.args.num_heads >= static_cast<int>(cs) * 2) cs *= 2;
    return launch_dependent_cluster(kern, dim3(static_cast<unsigned>(L.key_tiles), static_cast<unsigned>(L.row_tiles), cs),
                                    dim3(kMapThreads), smem, stream, dim3(1, 1, cs), L.tmQ[0], L.tmQ[1],
                                    L.tmK[0], L.tmK[1], L.args);
}

}  // namespace

cudaError_t launch_attn_map(const AttnMapLaunch& L, cudaStream_t stream) {
    if (L.head_dim == 128) return L.bf16 ? launch_map_t<128, true>(L, stream) : launch_map_t<128, false>(L, stream);
    if (L.head_dim == 64) return L.bf16 ? launch_map_t<64, true>(L, stream) : launch_map_t<64, false>(L, stream);
    return cudaErrorInvalidValue;
}

}  // namespace bdattn
