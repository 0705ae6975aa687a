// Softmax attention forward for head_dim 64 / 128 on the sm_100a tensor cores.
//
// One CTA owns two 128-row query tiles of one (batch, head), or in the last wave of a launch
// a single one (launch_t), and walks the key
// tiles (128 keys each).  Roles (12 warps, three warpgroups):
//   warps 0-3  : softmax of query tile 0   (one thread per query row)
//   warps 4-7  : softmax of query tile 1
//   warp  8    : issues the Q.K^T MMAs (one lane), owns the TMEM allocation
//   warp  9    : TMA producer for Q, K and V tiles (one lane)
//   warp  10   : issues the P.V MMAs (one lane)
//   warp  11   : idle (it completes the third warpgroup, so that registers can be moved
//                to the softmax warpgroups with setmaxnreg)
//   warps 12-15: only with per-key scale vectors (kScale): multiply the rows of a K or V
//                tile in shared memory by their factors before the MMAs read it, 32
//                rows each
// Tensor memory (512 columns) at head_dim 128:
//   P0 [0,64)  S [64,192)  P1 [192,256)  O0 [256,384)  O1 [384,512)
// and at 64: S0 [0,128) S1 [128,256) P0 [256,320) P1 [320,384) O0 [384,448)
// O1 [448,512).  P is the exponentiated score tile (16-bit, two per column),
// consumed from tensor memory as the A operand of the P.V MMA.
//
// What paces the kernel is the dependency chain of one query tile: scores ready ->
// softmax -> P ready -> P.V.  P has columns of its own, so the scores of step j+1
// are computed while step j is still exponentiated: Q.K^T of a tile is issued as
// soon as the S buffer's last user has fetched its scores into registers, and the
// softmax warps go from one step to the next without waiting for any MMA of their
// own step.  At head_dim 128 there is room for one S buffer only; the two tiles, half
// a step apart, take turns in it (it is occupied from the first MMA until the fetch
// is over, about 1100 cycles of a step per tile).  At 64 each tile has its own, and the
// scores are issued in turns all the same: two tiles in step want the exponential unit at
// the same time (4096 x 4096, 8 heads of 40, FP16: 57.9 us in step, 53.9 in turns).  A key step takes 2720 cycles (3550
// when P overwrote S and Q.K^T of step j+1 had to wait for P.V of step j): 4608 x 4608,
// 24 heads of 128, 224 -> 199 us before the power cap sets in; 16896 x 16896, two batch
// items, under the cap (SM clock 1.48 GHz instead of 1.85) 6.34 -> 5.77 ms.
// The running maximum is only raised when it grew by more than 2^8 (the factor
// is carried by P and cancels in O / l), which makes the O rescale rare; the
// rescale is done in tensor memory by the softmax warps themselves.
// The softmax arithmetic is packed two floats per instruction (fma/add .f32x2)
// and the row maximum uses the three-input max.
//
// Q, K and V are addressed through 4-D tensor maps (head element, head, row,
// batch): a head narrower than the 64 / 128 columns the kernel computes with
// (40, 72, 80, 112, ...) is zero-padded by the TMA unit itself, so such head
// dims run here without a padding pass; only the real columns are stored.
//
// Arithmetic follows the attention core of dit::joint_attention_traced
// (src/dit/common.cpp:246-305): scale 1/sqrt(hd), stable softmax,
// inv = denom > 0 ? 1/denom : 0, with FP32 scores and accumulation.
#include "sdpa_internal.h"
#include "tc05.cuh"

namespace bdattn {

namespace {

constexpr int kBM = 128;           // query rows per tile
constexpr int kBN = 128;           // keys per tile
constexpr int kChunkBytes = 128 * 128;  // one 64-column (128 B) x 128-row TMA box

constexpr int kMaxListed = 512;    // key tiles a list of the tiles with a visible key has room for
constexpr int kPartTile = 0x8000;  // set in its entries for tiles that have a masked key too

// kBias: the softmax warps have 4 KB of shared memory each for rows of a logit bias, at 128 columns in the place of the
// third K tile; at 64 columns 16 KB more for the CTAs with a single query tile.
template <int HD, bool kBias>
struct Cfg {
    static constexpr int kChunks = HD / 64;
    static constexpr int kTileBytes = kBN * HD * 2;
    static constexpr int kQBytes = kBM * HD * 2;
    // K and V tiles have a ring each: each ring is then read by one MMA warp only,
    // which sees every phase of its barriers.
    static constexpr int kKStages = HD == 128 ? (kBias ? 2 : 3) : 4;
    static constexpr int kVStages = HD == 128 ? 2 : 4;
    static constexpr int kBarBytes = 512;
    static constexpr int kListBytes = 2 * kMaxListed;      // key tiles to visit (calls with a key mask)
    static constexpr int kBiasBytes = kBias ? (HD == 128 ? 8 : 12) * 4096 : 0;
    static constexpr int kSmemBytes =
        2 * kQBytes + (kKStages + kVStages) * kTileBytes + kBarBytes + kListBytes + kBiasBytes + 1024;
    // Tensor memory columns (512 in all).  At 64 columns per head every tile has its
    // own S; at 128 the two tiles take turns in one S buffer between their P tiles.
    static constexpr uint32_t kColS0 = HD == 128 ? 64 : 0;
    static constexpr uint32_t kColS1 = HD == 128 ? 64 : 128;
    static constexpr uint32_t kColP0 = HD == 128 ? 0 : 256;
    static constexpr uint32_t kColP1 = HD == 128 ? 192 : 320;
    static constexpr uint32_t kColO0 = HD == 128 ? 256 : 384;
    static constexpr uint32_t kColO1 = kColO0 + HD;
};

// Threads of a CTA, and registers per thread after the hand-over (setmaxnreg), which stay within what the
// CTA is launched with: 8 x 216 + 4 x 64 within 12 x 168; with scaling warps 8 x 208 + 8 x 48 = 16 x 128.
// Scaling a tile costs one warp 5000 cycles beside the softmax warps, a key step has two tiles and
// 2790 cycles: four warps (256 + 1024 keys of which 256 are scaled, 24 heads of 128: 24.6 us; 31.5 with
// one warp, 21.9 without scales; all of 2048 + 512 keys 53.6, 106 and 35.2).
template <bool kScale>
struct Roles {
    static constexpr int kThreads = kScale ? 512 : 384;
    static constexpr int kRegsSoftmax = kScale ? 208 : 216;
    static constexpr int kRegsOther = kScale ? 48 : 64;
};

struct TileInfo {
    int seg;
    int row0;
    int valid;
    int kbase;
};

__device__ __forceinline__ TileInfo kv_tile(const SdpaDevArgs& a, int t) {
    TileInfo ti;
    if (t < a.kv_tiles0) {
        ti.seg = 0;
        ti.row0 = t * kBN;
        ti.valid = min(kBN, a.kv_rows[0] - ti.row0);
        ti.kbase = ti.row0;
    } else {
        ti.seg = 1;
        ti.row0 = (t - a.kv_tiles0) * kBN;
        ti.valid = min(kBN, a.kv_rows[1] - ti.row0);
        ti.kbase = a.kv_rows[0] + ti.row0;
    }
    return ti;
}

// ------------------------------------------------------- packed FP32 math
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// (d0, d1) = (a0, a1) * (b0, b1) + (c0, c1)
__device__ __forceinline__ void ffma2(float& d0, float& d1, float a0, float a1, float b0, float b1,
                                      float c0, float c1) {
    asm("{\n"
        ".reg .b64 ra, rb, rc, rd;\n"
        "mov.b64 ra, {%2, %3};\n"
        "mov.b64 rb, {%4, %5};\n"
        "mov.b64 rc, {%6, %7};\n"
        "fma.rn.f32x2 rd, ra, rb, rc;\n"
        "mov.b64 {%0, %1}, rd;\n"
        "}\n"
        : "=f"(d0), "=f"(d1)
        : "f"(a0), "f"(a1), "f"(b0), "f"(b1), "f"(c0), "f"(c1));
}
__device__ __forceinline__ void fadd2(float& d0, float& d1, float a0, float a1, float b0, float b1) {
    asm("{\n"
        ".reg .b64 ra, rb, rd;\n"
        "mov.b64 ra, {%2, %3};\n"
        "mov.b64 rb, {%4, %5};\n"
        "add.rn.f32x2 rd, ra, rb;\n"
        "mov.b64 {%0, %1}, rd;\n"
        "}\n"
        : "=f"(d0), "=f"(d1)
        : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}
template <int N>
__device__ __forceinline__ void setmaxnreg_inc() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void setmaxnreg_dec() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

// HOOKS: 0 = none; 1 = key_mask only; 2 = key_mask and the per-row softmax statistics; 3 = a logit
// bias besides (slower softmax path); 4 = a bias of a few rows, read without shared memory (launch_hd).
// SCALE: key_scale / val_scale are applied to the K / V tiles in shared memory by
// warps 12-15 (rounded to the storage type, as the reference's scale_inplace on its
// k_full_ / v_full_ copies does, src/dit/qwenimage21_forward.cpp:606-645); the
// softmax code does not change.
// kMixed: some CTAs of the launch have one query tile (launch_t); without it every CTA has two.
template <int HD, bool kBf16, int kHooks, bool kScale, bool kMixed>
__global__ void __launch_bounds__(Roles<kScale>::kThreads, 1)
sdpa_tc05_kernel(const __grid_constant__ CUtensorMap tmQ0, const __grid_constant__ CUtensorMap tmQ1,
                 const __grid_constant__ CUtensorMap tmK0, const __grid_constant__ CUtensorMap tmK1,
                 const __grid_constant__ CUtensorMap tmV0, const __grid_constant__ CUtensorMap tmV1,
                 const SdpaDevArgs a) {
    using C = Cfg<HD, kHooks == 3>;
    constexpr int KS = C::kKStages;
    constexpr int VS = C::kVStages;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
    uint8_t* smem_q = smem;
    uint8_t* smem_k = smem + 2 * C::kQBytes;
    uint8_t* smem_v = smem_k + KS * C::kTileBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem_v + VS * C::kTileBytes);
    uint64_t* q_full = bars;             // [2]
    uint64_t* s_full = bars + 2;         // [2]  scores of the tile are in tensor memory
    uint64_t* s_free = bars + 4;         // [2]  the tile's softmax warps hold them in registers
    uint64_t* p_full = bars + 6;         // [2]
    uint64_t* pv_done = bars + 8;        // [2]
    uint64_t* q_ready = bars + 10;       // [2]  Q tile normalised + rotated in place (fused Q path)
    uint64_t* k_full = bars + 12;        // [KS]
    uint64_t* k_empty = k_full + KS;     // [KS]
    uint64_t* k_ready = k_empty + KS;    // [KS] tile landed and, where needed, scaled (kScale)
    uint64_t* v_full = k_ready + KS;     // [VS]
    uint64_t* v_empty = v_full + VS;     // [VS]
    uint64_t* v_ready = v_empty + VS;    // [VS]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(v_ready + VS);
    uint16_t* tile_list = reinterpret_cast<uint16_t*>(reinterpret_cast<uint8_t*>(bars) + C::kBarBytes);   // [kMaxListed]

    const int warp = warp_index();
    const int lane = threadIdx.x & 31;
    // Work item of this CTA: two query tiles of one (batch, head), or one of them.
    int q_cta = static_cast<int>(blockIdx.x), head = static_cast<int>(blockIdx.y), batch = static_cast<int>(blockIdx.z);
    int tile0 = 0, n_tiles = 2;
    if constexpr (kMixed) {
        int item = static_cast<int>(blockIdx.x);
        if (item >= a.whole_items) {
            n_tiles = 1;
            tile0 = (item - a.whole_items) & 1;
            item = a.whole_items + ((item - a.whole_items) >> 1);
        }
        q_cta = item % a.q_ctas;
        head = item / a.q_ctas % a.num_heads;
        batch = item / a.q_ctas / a.num_heads;
    }
    const int qseg = q_cta >= a.q_ctas0 ? 1 : 0;
    const int qrow0 = ((qseg ? q_cta - a.q_ctas0 : q_cta) * 2 + tile0) * kBM;
    const int seg_rows = qseg ? a.q_rows[1] : a.q_rows[0];
    const int q_global0 = (qseg ? a.q_rows[0] : 0) + qrow0;
    if constexpr (kMixed) {
        if (qrow0 >= seg_rows) return;               // the second tile of a segment's last rows
        if (seg_rows - qrow0 <= kBM) n_tiles = 1;
    }
    const int n_t = kMixed ? n_tiles : 2;

    // Key tiles this CTA has to visit.
    int n_kv = a.kv_tiles;
    if (a.mask_mode == 1) {
        const int last = q_global0 + min(n_t * kBM, seg_rows - qrow0) - 1;
        const int max_key = last + a.q_offset;
        int n = 0;
        for (int t = 0; t < a.kv_tiles; ++t) {
            if (kv_tile(a, t).kbase <= max_key) n = t + 1;
        }
        n_kv = n;
    }

    if (threadIdx.x == 0) {
        for (int i = 0; i < KS; ++i) {
            mbar_init(&k_full[i], 1);
            mbar_init(&k_empty[i], 1);
            mbar_init(&k_ready[i], 4);
        }
        for (int i = 0; i < VS; ++i) {
            mbar_init(&v_full[i], 1);
            mbar_init(&v_empty[i], 1);
            mbar_init(&v_ready[i], 4);
        }
        for (int t = 0; t < 2; ++t) {
            mbar_init(&q_full[t], 1);
            mbar_init(&s_full[t], 1);
            mbar_init(&s_free[t], 4);          // one arrival per softmax warp of the tile
            mbar_init(&p_full[t], 4);
            mbar_init(&pv_done[t], 1);
            mbar_init(&q_ready[t], 4);
        }
        fence_mbar_init();
    }
    if (warp == 8) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    if (warp == 9 && lane == 0) {
        tma_prefetch_desc(qseg ? &tmQ1 : &tmQ0);
        tma_prefetch_desc(&tmK0);
        tma_prefetch_desc(&tmV0);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // only now: a dependent CTA that took tensor memory first could keep this one from getting its own
    dependents_may_launch();
    // barriers, tensor memory and descriptors are set up; from here on global memory is touched
    wait_for_prior_grid();

    // With a key mask, tiles without a visible key (the padding of a caption) are left out: they
    // would add nothing to any row.  The warps look at the tiles in turn, one load per lane
    // and 32 keys, and the flags become the list that all roles walk.  (512 text keys of
    // which 187 are visible and 1530 others, 24 heads: 67.5 -> 60.8 us; the query tiles travel
    // while the list is made.)
    auto load_q = [&](int t) {
        const CUtensorMap* mq = qseg ? &tmQ1 : &tmQ0;
        mbar_arrive_expect_tx(&q_full[t], C::kQBytes);
        for (int c = 0; c < C::kChunks; ++c) {
            tma_load_4d(smem_q + t * C::kQBytes + c * kChunkBytes, mq, &q_full[t],
                        c * 64, head, qrow0 + t * kBM, batch);
        }
    };
    bool listed = false;
    if constexpr (kHooks >= 1 && !kScale) {
        if (a.key_mask != nullptr && n_kv <= kMaxListed) {
            listed = true;
            if (warp == 9 && lane == 0) {      // the query tiles travel meanwhile
                load_q(0);
                if (n_t == 2) load_q(1);
            }
            __syncwarp();
#pragma unroll 2
            for (int t = warp; t < n_kv; t += Roles<kScale>::kThreads / 32) {
                const TileInfo ti = kv_tile(a, t);
                float mv[4];
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    const int c = lane + 32 * w;
                    mv[w] = c < ti.valid ? __ldg(a.key_mask + ti.kbase + c) : 0.0f;
                }
                const bool seen = __any_sync(0xffffffffu, mv[0] != 0.0f || mv[1] != 0.0f || mv[2] != 0.0f || mv[3] != 0.0f);
                bool hidden = false;
#pragma unroll
                for (int w = 0; w < 4; ++w) hidden = hidden || (mv[w] == 0.0f && lane + 32 * w < ti.valid);
                const bool part = __any_sync(0xffffffffu, hidden);
                if (lane == 0) tile_list[t] = seen ? (part ? kPartTile | 1 : 1) : 0;
            }
            __syncthreads();
            // every warp counts and one writes (in place: an entry is read before it is overwritten)
            int n = 0;
            for (int t0 = 0; t0 < n_kv; t0 += 32) {
                const int t = t0 + lane;
                const int f = t < n_kv ? tile_list[t] : 0;
                const bool on = f != 0;
                const uint32_t m = __ballot_sync(0xffffffffu, on);
                __syncthreads();
                if (warp == 0 && on) tile_list[n + __popc(m & ((1u << lane) - 1u))] = static_cast<uint16_t>(t | (f & kPartTile));
                n += __popc(m);
            }
            __syncthreads();
            n_kv = n;
        }
    }
    // the j-th key tile of this CTA
    auto tile_at = [&](int j) { return kv_tile(a, listed ? tile_list[j] & (kPartTile - 1) : j); };

    if (warp < 4 * n_t) {
        // ------------------------------------------------ softmax + epilogue
        setmaxnreg_inc<Roles<kScale>::kRegsSoftmax>();
        const int t = warp >> 2;
        const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const uint32_t tS = tmem_base + lane_base + (t ? C::kColS1 : C::kColS0);
        const uint32_t tP = tmem_base + lane_base + (t ? C::kColP1 : C::kColP0);
        const uint32_t tO = tmem_base + lane_base + (t ? C::kColO1 : C::kColO0);
        const int row_in_tile = (warp & 3) * 32 + lane;
        const int row_in_seg = qrow0 + t * kBM + row_in_tile;
        const int q_glob = q_global0 + t * kBM + row_in_tile;
        const float sl2 = a.scale_log2;
        float m_ref = -INFINITY;
        float l_sum = 0.0f;
        bool ok = true;

        if (a.q_fused && n_kv > 0) {
            // Per-head RMSNorm + RoPE of the query tile, in place in the (128-byte
            // swizzled) Q tile, before the first Q.K^T MMA (src/dit/flux.cpp:462-469 +
            // src/dit/common.cpp:192 applied to Q).  A warp takes its 32 rows one at a
            // time with the head's columns spread over the lanes, so that the cos / sin
            // rows are read coalesced (one row per load; a thread-per-row version
            // touched 32 cache lines per load and cost ten times as much).  Rows past
            // the segment are zero and stay zero.
            ok = __all_sync(0xffffffffu, mbar_wait(&q_full[t], 0));
            if (ok) {
                constexpr int kEpl = HD / 32;                 // elements per lane: 4 or 2
                const int hd = a.hd_out;
                const int c0 = lane * kEpl;                   // first column of this lane
                const bool live = c0 < hd;                    // hd is a multiple of 8
                const void* gain = qseg ? a.q_gain[1] : a.q_gain[0];
                float gv[kEpl];
#pragma unroll
                for (int i = 0; i < kEpl; ++i) gv[i] = 1.0f;
                if (gain != nullptr && live) {
#pragma unroll
                    for (int i = 0; i < kEpl; ++i) {
                        if (a.q_gain_is_f32) gv[i] = __ldg(reinterpret_cast<const float*>(gain) + c0 + i);
                        else {
                            const uint16_t b = __ldg(reinterpret_cast<const uint16_t*>(gain) + c0 + i);
                            gv[i] = kBf16 ? __uint_as_float(static_cast<uint32_t>(b) << 16)
                                          : __half2float(*reinterpret_cast<const __half*>(&b));
                        }
                    }
                }
                const int bofs = (c0 & 63) * 2;               // byte offset inside the 128-byte row piece
                uint8_t* qbase = smem_q + t * C::kQBytes + (c0 >> 6) * kChunkBytes + (bofs & 15);
                const int cidx = bofs >> 4;
                const float inv_hd = 1.0f / static_cast<float>(hd);
                // 16 rows at a time, every load of a batch issued before the first use:
                // a row-by-row loop is a chain of load and shuffle latencies
                constexpr int kRb = 16;
                const bool rope = a.q_cos != nullptr && live;
#pragma unroll 1
                for (int r0 = 0; r0 < 32; r0 += kRb) {
                    uint32_t w[kRb][kEpl / 2];
                    float cs[kRb][kEpl / 2], sn[kRb][kEpl / 2];
#pragma unroll
                    for (int k = 0; k < kRb; ++k) {
                        const int r = (warp & 3) * 32 + r0 + k;
                        const uint8_t* ptr = qbase + r * 128 + ((cidx ^ (r & 7)) << 4);
                        if constexpr (kEpl == 4) {
                            const uint2 u = *reinterpret_cast<const uint2*>(ptr);
                            w[k][0] = u.x; w[k][1] = u.y;
                        } else {
                            w[k][0] = *reinterpret_cast<const uint32_t*>(ptr);
                        }
#pragma unroll
                        for (int i = 0; i < kEpl / 2; ++i) { cs[k][i] = 1.0f; sn[k][i] = 0.0f; }
                        if (rope && qrow0 + t * kBM + r < seg_rows) {
                            const long long tb = static_cast<long long>(a.q_rope_row0 + q_global0 + t * kBM + r) * (hd >> 1) + (c0 >> 1);
                            if constexpr (kEpl == 4) {
                                const float2 cv = __ldg(reinterpret_cast<const float2*>(a.q_cos + tb));
                                const float2 sv = __ldg(reinterpret_cast<const float2*>(a.q_sin + tb));
                                cs[k][0] = cv.x; cs[k][1] = cv.y; sn[k][0] = sv.x; sn[k][1] = sv.y;
                            } else {
                                cs[k][0] = __ldg(a.q_cos + tb); sn[k][0] = __ldg(a.q_sin + tb);
                            }
                        }
                    }
                    float x[kRb][kEpl], ss[kRb];
#pragma unroll
                    for (int k = 0; k < kRb; ++k) {
#pragma unroll
                        for (int i = 0; i < kEpl / 2; ++i) {
                            if constexpr (kBf16) {
                                x[k][2 * i] = __uint_as_float(w[k][i] << 16);
                                x[k][2 * i + 1] = __uint_as_float(w[k][i] & 0xffff0000u);
                            } else {
                                const __half2 h = *reinterpret_cast<const __half2*>(&w[k][i]);
                                x[k][2 * i] = __low2float(h);
                                x[k][2 * i + 1] = __high2float(h);
                            }
                        }
                        ss[k] = 0.0f;
#pragma unroll
                        for (int i = 0; i < kEpl; ++i) ss[k] = fmaf(x[k][i], x[k][i], ss[k]);
                    }
                    if (gain != nullptr) {
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
                            for (int k = 0; k < kRb; ++k) ss[k] += __shfl_xor_sync(0xffffffffu, ss[k], o);
                        }
#pragma unroll
                        for (int k = 0; k < kRb; ++k) {
                            const float inv = rsqrtf(ss[k] * inv_hd + a.q_eps);
#pragma unroll
                            for (int i = 0; i < kEpl; ++i) x[k][i] *= inv * gv[i];
                        }
                    }
#pragma unroll
                    for (int k = 0; k < kRb; ++k) {
                        const int r = (warp & 3) * 32 + r0 + k;
                        uint8_t* ptr = qbase + r * 128 + ((cidx ^ (r & 7)) << 4);
#pragma unroll
                        for (int i = 0; i < kEpl / 2; ++i) {
                            const float a0 = x[k][2 * i], b0 = x[k][2 * i + 1];
                            x[k][2 * i] = a0 * cs[k][i] - b0 * sn[k][i];
                            x[k][2 * i + 1] = a0 * sn[k][i] + b0 * cs[k][i];
                        }
                        if constexpr (kEpl == 4) {
                            uint2 u;
                            u.x = pack2<kBf16>(x[k][0], x[k][1]);
                            u.y = pack2<kBf16>(x[k][2], x[k][3]);
                            *reinterpret_cast<uint2*>(ptr) = u;
                        } else {
                            *reinterpret_cast<uint32_t*>(ptr) = pack2<kBf16>(x[k][0], x[k][1]);
                        }
                    }
                }
                fence_proxy_async_smem();      // the MMA reads the tile through the async proxy
                __syncwarp();
                if (lane == 0) mbar_arrive(&q_ready[t]);
            }
        }

        // Logit bias: the warp's 32 rows, 32 columns at a time through shared memory; the first piece travels while
        // the scores are computed (a load with a row per lane: 256 + 1024 tokens, 24 heads, bias on two of ten tiles,
        // 33.1 us, now 29.4, 21.1 without a bias).  The others follow one by one, a latency each, as far as there are
        // columns.  A CTA with a single query tile has nothing to hide that behind, but the room of the other tile: there
        // all four pieces travel ahead of the scores (23 + 512 tokens, 24 heads of 40, bias on the 23: 22.3 us one by one, 16.3).
        constexpr int kOwn = C::kBiasBytes / (4 * 4096);             // pieces of a lone tile that the bias area holds
        const int lone = n_t == 1 ? 1 : 0;
        uint8_t* const bias_s = reinterpret_cast<uint8_t*>(tile_list + kMaxListed) + warp * 4096;
        const int w_row = q_global0 + t * kBM + (warp & 3) * 32 - a.bias_row0;      // the warp's first bias row
        auto bias_piece = [&](int i) {
            // (from the end of the bias area back to the second tile's Q buffer)
            constexpr int kBack = kOwn * 4 * 4096 + C::kListBytes + C::kBarBytes + (KS + VS) * C::kTileBytes + C::kQBytes;
            return bias_s + lone * (i * 4 * 4096 - (i < kOwn ? 0 : kBack));
        };
        auto load_bias = [&](int kbase, int lim, int i) {
            copy_rows32(bias_piece(i), a.bias + kbase + i * 32, a.bias_ld, w_row, a.bias_rows, lim - i * 32, lane);
        };

        for (int j = 0; j < n_kv; ++j) {
            // Key mask of this tile as 128 bits (four ballots over one coalesced load
            // per lane), fetched before the wait for S so that its latency is hidden.
            uint32_t mbits[4] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu};
            if constexpr (kHooks >= 1) {
                // (a list says which tiles have none, and they are passed over: 2042 keys of which 1717 are visible, 24 heads, 56.7 -> 54.2 us)
                if (a.key_mask != nullptr && (!listed || (tile_list[j] & kPartTile) != 0)) {
                    const TileInfo tm = tile_at(j);
                    float mv[4];
#pragma unroll
                    for (int w = 0; w < 4; ++w) {
                        const int c = 4 * lane + w;
                        mv[w] = c < tm.valid ? __ldg(a.key_mask + tm.kbase + c) : 1.0f;
                    }
#pragma unroll
                    for (int w = 0; w < 4; ++w) mbits[w] = __ballot_sync(0xffffffffu, mv[w] != 0.0f);
                }
            }
            const TileInfo ti = tile_at(j);
            int bias_lim = 0;              // columns of this tile that have a bias, none where the warp's rows have none
            if constexpr (kHooks >= 3)
                if (w_row + 32 > 0 && w_row < a.bias_rows) bias_lim = min(ti.valid, a.bias_cols - ti.kbase);
            if constexpr (kHooks == 3) {
                if (bias_lim > 0) {
                    const int ahead = lone ? (bias_lim + 31) >> 5 : 1;
#pragma unroll 1
                    for (int i = 0; i < ahead; ++i) load_bias(ti.kbase, bias_lim, i);
                }
            }
            int lim = ti.valid - 1;
            if (a.mask_mode == 1) lim = min(lim, q_glob + a.q_offset - ti.kbase);
            // A wait that runs out leaves `ok` false in its lane and the step goes on with
            // whatever is there; the vote on the row maximum below ends the loop for the
            // whole warp (one vote per step instead of one per wait).
            ok = mbar_wait(&s_full[t], static_cast<uint32_t>(j & 1)) && ok;
            tc_fence_after();
            float s[kBN];
#pragma unroll
            for (int c = 0; c < kBN / 32; ++c) {
                tmem_ld32(tS + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&s[c * 32]));
            }
            tmem_wait_ld();
            // the scores are in registers: the next Q.K^T may overwrite the buffer
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_free[t]);

            if constexpr (kHooks == 3) {
                if (bias_lim > 0) {
#pragma unroll
                    for (int c = 0; c < kBN; c += 32) {
                        cp_async_wait_all();
                        __syncwarp();
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float4 b = row_piece32(bias_piece(c >> 5), lane, i);
                            s[c + 4 * i] += b.x * a.bias_mul;
                            s[c + 4 * i + 1] += b.y * a.bias_mul;
                            s[c + 4 * i + 2] += b.z * a.bias_mul;
                            s[c + 4 * i + 3] += b.w * a.bias_mul;
                        }
                        __syncwarp();
                        if (c + 32 >= bias_lim) break;
                        if (!lone) load_bias(ti.kbase, bias_lim, (c >> 5) + 1);
                    }
                }
            }
            if constexpr (kHooks == 4) {
                // a thread reads its own row, all loads in flight at once
                const int br = q_glob - a.bias_row0;
                if (bias_lim > 0 && br >= 0 && br < a.bias_rows) {
                    const float* const brow = a.bias + static_cast<long long>(br) * a.bias_ld + ti.kbase;
                    if ((bias_lim & 3) == 0 && (a.bias_ld & 3) == 0 && (reinterpret_cast<uintptr_t>(a.bias + ti.kbase) & 15u) == 0) {
#pragma unroll
                        for (int c = 0; c < kBN; c += 4) {
                            if (c < bias_lim) {
                                const float4 b = __ldg(reinterpret_cast<const float4*>(brow + c));
                                s[c] += b.x * a.bias_mul;
                                s[c + 1] += b.y * a.bias_mul;
                                s[c + 2] += b.z * a.bias_mul;
                                s[c + 3] += b.w * a.bias_mul;
                            }
                        }
                    } else {
#pragma unroll
                        for (int c = 0; c < kBN; ++c)
                            if (c < bias_lim) s[c] += __ldg(brow + c) * a.bias_mul;
                    }
                }
            }
            // (uniform over the CTA without the causal rule: no vote on whole tiles)
            if (a.mask_mode == 1 ? __any_sync(0xffffffffu, lim < kBN - 1) : ti.valid < kBN) {
#pragma unroll
                for (int c = 0; c < kBN; ++c) s[c] = (c <= lim) ? s[c] : -INFINITY;
            }
            if constexpr (kHooks >= 1) {
                // (tiles without a masked key, the usual case away from the padded tail, skip this)
                if (a.key_mask != nullptr && (mbits[0] & mbits[1] & mbits[2] & mbits[3]) != 0xffffffffu) {
#pragma unroll
                    for (int c = 0; c < kBN; ++c) {
                        if (((mbits[c & 3] >> (c >> 2)) & 1u) == 0u) s[c] = -INFINITY;
                    }
                }
            }

            // row maximum: four independent chains of three-input max
            float mx0 = max3(s[0], s[1], s[2]), mx1 = max3(s[3], s[4], s[5]);
            float mx2 = max3(s[6], s[7], s[8]), mx3 = max3(s[9], s[10], s[11]);
#pragma unroll
            for (int c = 12; c + 7 < kBN; c += 8) {
                mx0 = max3(mx0, s[c], s[c + 1]);
                mx1 = max3(mx1, s[c + 2], s[c + 3]);
                mx2 = max3(mx2, s[c + 4], s[c + 5]);
                mx3 = max3(mx3, s[c + 6], s[c + 7]);
            }
            // 12 + 8*14 = 124: four scores left
            mx0 = max3(mx0, s[124], s[125]);
            mx1 = max3(mx1, s[126], s[127]);
            const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
            const float m_new = fmaxf(m_ref, mx);
            const bool grow = (m_new - m_ref) * sl2 > 8.0f;
            if (__any_sync(0xffffffffu, grow || !ok)) {
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                float alpha = 1.0f;
                if (grow) {
                    alpha = (m_ref == -INFINITY) ? 0.0f : fast_exp2((m_ref - m_new) * sl2);
                    m_ref = m_new;
                }
                l_sum *= alpha;
                if (j > 0) {
                    // the accumulator is at rest between P.V of step j-1 and that of step j
                    ok = __all_sync(0xffffffffu, mbar_wait(&pv_done[t], static_cast<uint32_t>((j - 1) & 1)));
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll
                    for (int c = 0; c < HD / 32; ++c) {
                        uint32_t o[32];
                        tmem_ld32(tO + c * 32, o);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        tmem_st32(tO + c * 32, o);
                    }
                }
            }
            const float m_use = (m_ref == -INFINITY) ? 0.0f : m_ref;
            const float neg_ms = -m_use * sl2;
            // P.V of step j-1 releases the tile's P columns; it was issued when this step's scores were
            // fetched, so the wait is over by then as a rule.  Ahead of the exponentials and not between their
            // halves: these then run in two unbroken stretches, which is worth 4.5 % (2499 x 2499, 24 heads of 128,
            // 74.2 -> 70.8 us; with the tile's bounds looked up before the scores come and the row sum
            // behind the hand-over).
            if (j > 0) {
                ok = mbar_wait(&pv_done[t], static_cast<uint32_t>((j - 1) & 1));
                tc_fence_after();
            }
            // p = 2^(s * scale_log2 - m * scale_log2); row sum in four packed chains
            float rs[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) rs[i] = 0.0f;
            auto exp_pairs = [&](int c_begin, int n, uint32_t* pk) {
#pragma unroll
                for (int i = 0; i < n; ++i) {
                    const int c0 = c_begin + 2 * i;
                    float x0, x1, p0, p1;
                    ffma2(x0, x1, s[c0], s[c0 + 1], sl2, sl2, neg_ms, neg_ms);
                    p0 = fast_exp2(x0);
                    p1 = fast_exp2(x1);
                    fadd2(rs[2 * (i & 3)], rs[2 * (i & 3) + 1], rs[2 * (i & 3)], rs[2 * (i & 3) + 1], p0, p1);
                    pk[i] = pack2<kBf16>(p0, p1);
                }
            };
#pragma unroll
            for (int ch = 0; ch < 2; ++ch) {
                uint32_t pk[32];
                exp_pairs(ch * 64, 32, pk);
                tmem_st32(tP + ch * 32, pk);
            }
            tmem_wait_st();
            tc_fence_before();
            // one elected arrival per warp: 32 lanes arriving on the same barrier
            // word serialise and delay the hand-over to the MMA warp
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[t]);
            l_sum += ((rs[0] + rs[1]) + (rs[2] + rs[3])) + ((rs[4] + rs[5]) + (rs[6] + rs[7]));
        }

        if (n_kv > 0) {
            ok = mbar_wait(&pv_done[t], static_cast<uint32_t>((n_kv - 1) & 1)) && ok;
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
        } else if (listed) {
            // no visible key: the query tile may still be on its way into the buffer that the epilogue
            // stages its zeros in
            ok = __all_sync(0xffffffffu, mbar_wait(&q_full[t], 0));
        }
        const float inv = (l_sum > 0.0f) ? 1.0f / l_sum : 0.0f;
        if constexpr (kHooks >= 2) {
            if (a.lse != nullptr && ok && row_in_seg < seg_rows) {
                float* st = a.lse + ((static_cast<long long>(batch) * a.num_heads + head) * a.lq_total + q_glob) * 2;
                st[0] = m_ref * sl2;
                st[1] = l_sum;
            }
        }
        // Epilogue: O / l goes through shared memory (this tile's Q buffer, no longer
        // read: all Q.K^T MMAs have completed) so that global stores are whole
        // rows: 16-byte chunk c of row r sits at chunk c ^ (r mod chunks) to keep
        // the row-per-thread writes and the row-major reads free of bank conflicts.
        // A warp stores the 32 rows it wrote (no CTA barrier), a lane the same chunk of every
        // row, eight loads in flight: a row-by-row loop over the tile took 5500 cycles of
        // a CTA's 11700 outside the key steps.
        constexpr int kRowChunks = HD / 8;
        uint8_t* stg = smem_q + t * C::kQBytes;
#pragma unroll
        for (int c = 0; c < HD / 32; ++c) {
            uint32_t o[32];
            if (ok && n_kv > 0) {
                tmem_ld32(tO + c * 32, o);
                tmem_wait_ld();
            } else {
#pragma unroll
                for (int i = 0; i < 32; ++i) o[i] = 0u;
            }
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                uint4 w;
                w.x = pack2<kBf16>(__uint_as_float(o[g * 8 + 0]) * inv, __uint_as_float(o[g * 8 + 1]) * inv);
                w.y = pack2<kBf16>(__uint_as_float(o[g * 8 + 2]) * inv, __uint_as_float(o[g * 8 + 3]) * inv);
                w.z = pack2<kBf16>(__uint_as_float(o[g * 8 + 4]) * inv, __uint_as_float(o[g * 8 + 5]) * inv);
                w.w = pack2<kBf16>(__uint_as_float(o[g * 8 + 6]) * inv, __uint_as_float(o[g * 8 + 7]) * inv);
                const int cg = c * 4 + g;
                *reinterpret_cast<uint4*>(stg + row_in_tile * (HD * 2) + ((cg ^ (row_in_tile & (kRowChunks - 1))) << 4)) = w;
            }
        }
        __syncwarp();
        const int cg = lane & (kRowChunks - 1);
        if (ok && cg < (a.hd_out >> 3)) {
            constexpr int kRowsPer = 32 / kRowChunks;           // rows of one access: 2 or 4
            const int r0 = (warp & 3) * 32 + lane / kRowChunks;
            const int rows_left = seg_rows - (qrow0 + t * kBM + r0);
            const long long o_ld = 2 * (qseg ? a.o_ld[1] : a.o_ld[0]);
            const long long off0 = 2 * (static_cast<long long>(batch) * (qseg ? a.o_bs[1] : a.o_bs[0]) +
                                        static_cast<long long>(head) * a.hd_out + cg * 8) +
                                   (qrow0 + t * kBM + r0) * o_ld;
            uint8_t* const obase = reinterpret_cast<uint8_t*>(qseg ? a.o[1] : a.o[0]);
            uint8_t* const mc = reinterpret_cast<uint8_t*>(qseg ? a.o_mc[1] : a.o_mc[0]);
            auto chunk = [&](int i) {
                const int r = r0 + i * kRowsPer;
                return *reinterpret_cast<const uint4*>(stg + r * (HD * 2) + ((cg ^ (r & (kRowChunks - 1))) << 4));
            };
            if (mc == nullptr) {
#pragma unroll
                for (int i0 = 0; i0 < kRowChunks; i0 += 8) {
                    uint4 w[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) w[i] = chunk(i0 + i);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        if ((i0 + i) * kRowsPer < rows_left)
                            *reinterpret_cast<uint4*>(obase + off0 + (i0 + i) * kRowsPer * o_ld) = w[i];
                    }
                }
                // fused all-gather: the same vectors go to every peer's copy of the
                // output (plain stores over NVLink; no TMA, no peer reads)
                for (int pi = 0; pi < a.n_peers; ++pi) {
                    uint8_t* const pb = reinterpret_cast<uint8_t*>(qseg ? a.o_peer[1][pi] : a.o_peer[0][pi]);
                    for (int i = 0; i < kRowChunks && i * kRowsPer < rows_left; ++i)
                        *reinterpret_cast<uint4*>(pb + off0 + i * kRowsPer * o_ld) = chunk(i);
                }
            } else {
                // fused all-gather through the switch: one store to the multicast
                // address lands in every GPU's copy of the output, this one's included
                for (int i = 0; i < kRowChunks && i * kRowsPer < rows_left; ++i) {
                    const uint4 w = chunk(i);
                    asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1, %2, %3, %4};"
                                 ::"l"(mc + off0 + i * kRowsPer * o_ld), "f"(__uint_as_float(w.x)), "f"(__uint_as_float(w.y)),
                                   "f"(__uint_as_float(w.z)), "f"(__uint_as_float(w.w))
                                 : "memory");
                }
            }
        }
    } else if (warp >= 8) {
        setmaxnreg_dec<Roles<kScale>::kRegsOther>();
        if (warp == 8) {
            // -------------------------------------------------- Q.K^T issuer
            // The queue between the issuing thread and the tensor pipe holds about sixteen MMAs, and
            // every commit and completed wait costs the thread 46-50 cycles: a single warp issuing both
            // products of both tiles could not keep the pipe fed, two warps can.  All lanes wait (a
            // wait that runs out is voted on behind the MMAs, where nothing waits for the vote) and one
            // elected lane of the converged warp issues: see elect_one.
            constexpr uint32_t idesc_qk = make_idesc_f16(kBf16 ? 1 : 0, kBM, kBN, 0, 0);
            const uint32_t q_base = smem_u32(smem_q);
            const uint32_t k_base = smem_u32(smem_k);
            uint64_t* const k_rdy = kScale ? k_ready : k_full;
            int slot = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int j = 0; ok && j < n_kv; ++j) {
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    if (t == 1 && n_t == 1) continue;
                    if (j == 0) {
                        ok = mbar_wait(&q_full[t], 0);
                        if (ok && a.q_fused) ok = mbar_wait(&q_ready[t], 0);
                    }
                    // the other tile holds the scores before these in registers: with one buffer it
                    // was that buffer's last user, with two this keeps the tiles in turns
                    if (ok && (j > 0 || t > 0)) ok = mbar_wait(&s_free[n_t == 2 ? t ^ 1 : 0], static_cast<uint32_t>((t ? j : j - 1) & 1));
                    if (ok && t == 0) ok = mbar_wait(&k_rdy[slot], phase);
                    tc_fence_after();
                    if (elect_one() && ok) {
                        const uint32_t qa = q_base + t * C::kQBytes;
                        const uint32_t kb = k_base + slot * C::kTileBytes;
                        const uint32_t d = tmem_base + (t ? C::kColS1 : C::kColS0);
#pragma unroll
                        for (int kk = 0; kk < HD / 16; ++kk) {
                            const uint32_t off = (kk >> 2) * kChunkBytes + (kk & 3) * 32;
                            umma_ss(d, make_smem_desc_sw128(qa + off, 16, 1024),
                                    make_smem_desc_sw128(kb + off, 16, 1024), idesc_qk, kk > 0 ? 1u : 0u);
                        }
                        umma_commit(&s_full[t]);
                        if (t == 1 || n_t == 1) umma_commit(&k_empty[slot]);
                    }
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                }
                if (++slot == KS) { slot = 0; phase ^= 1; }
            }
        } else if (warp == 10) {
            // -------------------------------------------------- P.V issuer
            constexpr uint32_t idesc_pv = make_idesc_f16(kBf16 ? 1 : 0, kBM, HD, 0, 1);
            const uint32_t v_base = smem_u32(smem_v);
            uint64_t* const v_rdy = kScale ? v_ready : v_full;
            int slot = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int j = 0; ok && j < n_kv; ++j) {
                ok = mbar_wait(&v_rdy[slot], phase);
                for (int t = 0; t < n_t; ++t) {
                    if (ok) ok = mbar_wait(&p_full[t], static_cast<uint32_t>(j & 1));
                    tc_fence_after();
                    if (elect_one() && ok) {
                        const uint32_t vb = v_base + slot * C::kTileBytes;
                        const uint32_t d = tmem_base + (t ? C::kColO1 : C::kColO0);
                        const uint32_t p = tmem_base + (t ? C::kColP1 : C::kColP0);
#pragma unroll
                        for (int kk = 0; kk < kBN / 16; ++kk) {
                            umma_ts(d, p + kk * 8, make_smem_desc_sw128(vb + kk * 2048, kChunkBytes, 1024), idesc_pv,
                                    (j > 0 || kk > 0) ? 1u : 0u);
                        }
                        umma_commit(&pv_done[t]);
                        if (t == 1 || n_t == 1) umma_commit(&v_empty[slot]);
                    }
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                }
                if (++slot == VS) { slot = 0; phase ^= 1; }
            }
        } else if (warp == 9) {
            // ------------------------------------------------ TMA producer
            if (lane == 0 && n_kv > 0) {
                if (!listed) load_q(0);        // (already under way with a list)
                const int kv_head = head / a.kv_group;
                int ks = 0, vs = 0, issued = 0;
                uint32_t kph = 1, vph = 1;             // parity that a fresh barrier passes
                bool ok = true;
                for (int j = 0; j < n_kv; ++j) {
                    const TileInfo ti = tile_at(j);
                    if (j >= KS) ok = mbar_wait(&k_empty[ks], kph);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&k_full[ks], C::kTileBytes);
                    for (int c = 0; c < C::kChunks; ++c) {
                        tma_load_4d(smem_k + ks * C::kTileBytes + c * kChunkBytes, ti.seg ? &tmK1 : &tmK0, &k_full[ks],
                                    c * 64, kv_head, ti.row0, batch);
                    }
                    if (j == 0 && !listed && n_t == 2) load_q(1);         // after what the first scores need
                    issued = 2 * j + 1;
                    if (++ks == KS) { ks = 0; kph ^= 1; }
                    if (j >= VS) ok = mbar_wait(&v_empty[vs], vph);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&v_full[vs], C::kTileBytes);
                    for (int c = 0; c < C::kChunks; ++c) {
                        tma_load_4d(smem_v + vs * C::kTileBytes + c * kChunkBytes, ti.seg ? &tmV1 : &tmV0, &v_full[vs],
                                    c * 64, kv_head, ti.row0, batch);
                    }
                    issued = 2 * j + 2;
                    if (++vs == VS) { vs = 0; vph ^= 1; }
                }
                if (!ok) {
                    // Unwinding after a wait ran out: let the copies already in
                    // flight land before the CTA gives its shared memory back.
                    mbar_wait(&q_full[0], 0);
                    if (n_t == 2) mbar_wait(&q_full[1], 0);
                    const int nk = (issued + 1) / 2, nv = issued / 2;
                    for (int i = max(0, nk - KS); i < nk; ++i) mbar_wait(&k_full[i % KS], static_cast<uint32_t>((i / KS) & 1));
                    for (int i = max(0, nv - VS); i < nv; ++i) mbar_wait(&v_full[i % VS], static_cast<uint32_t>((i / VS) & 1));
                }
            }
            __syncwarp();
        } else if (kScale && warp >= 12) {
            // ------------------------------------------- K / V row scaling
            // The four warps walk the K and V tiles in order (they see every phase of the barriers they
            // wait on); a lane has one row of a tile and its factor, fetched one tile ahead.  Rows none of
            // whose factors differs from one are passed on as they are, the others multiplied by
            // theirs (FP32 product rounded to the storage type).
            if constexpr (kScale) {
                bool ok = true;
                const int row = (warp - 12) * 32 + lane;
                auto fetch = [&](int i) {
                    const float* sc = (i & 1) ? a.val_scale : a.key_scale;
                    if (sc == nullptr || i >= 2 * n_kv) return 1.0f;
                    const TileInfo ti = kv_tile(a, i >> 1);
                    return row < ti.valid ? __ldg(sc + ti.kbase + row) : 1.0f;
                };
                float next = fetch(0);
                int kslot = 0, vslot = 0;
                uint32_t kphase = 0, vphase = 0;
                for (int i = 0; i < 2 * n_kv; ++i) {
                    const float f = next;
                    next = fetch(i + 1);
                    const bool is_v = (i & 1) != 0;
                    ok = is_v ? mbar_wait(&v_full[vslot], vphase) : mbar_wait(&k_full[kslot], kphase);
                    if (!ok) break;
                    if (__any_sync(0xffffffffu, f != 1.0f)) {
                        // Within a 64-column chunk a row is one 128-byte line whose 16-byte pieces the
                        // swizzle permutes; the factor is the same for all of them, so the pieces are
                        // walked in physical order, rotated by the lane's row so that the 32 rows of
                        // one access fall into different banks.
                        uint8_t* line = (is_v ? smem_v + vslot * C::kTileBytes : smem_k + kslot * C::kTileBytes) + row * 128;
#pragma unroll 1
                        for (int h = 0; h < 2 * C::kChunks; ++h) {
                            uint8_t* const half = line + (h >> 1) * kChunkBytes;
                            const int rot = (lane & 7) ^ ((h & 1) * 4);
                            uint4 v[4];
#pragma unroll
                            for (int b = 0; b < 4; ++b) v[b] = *reinterpret_cast<const uint4*>(half + ((b ^ rot) << 4));
#pragma unroll
                            for (int b = 0; b < 4; ++b) {
                                uint32_t* w32 = reinterpret_cast<uint32_t*>(&v[b]);
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    float lo, hi;
                                    if constexpr (kBf16) {
                                        lo = __uint_as_float(w32[e] << 16);
                                        hi = __uint_as_float(w32[e] & 0xffff0000u);
                                    } else {
                                        const __half2 hh = *reinterpret_cast<const __half2*>(&w32[e]);
                                        lo = __low2float(hh);
                                        hi = __high2float(hh);
                                    }
                                    // x * f + (-0) = x * f with the sign of a zero product kept
                                    ffma2(lo, hi, lo, hi, f, f, -0.0f, -0.0f);
                                    w32[e] = pack2<kBf16>(lo, hi);
                                }
                            }
#pragma unroll
                            for (int b = 0; b < 4; ++b) *reinterpret_cast<uint4*>(half + ((b ^ rot) << 4)) = v[b];
                        }
                        fence_proxy_async_smem();      // the MMA reads the tile through the async proxy
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(is_v ? &v_ready[vslot] : &k_ready[kslot]);
                    if (is_v) { if (++vslot == VS) { vslot = 0; vphase ^= 1; } }
                    else { if (++kslot == KS) { kslot = 0; kphase ^= 1; } }
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

template <int HD, bool kBf16, int kHooks, bool kScale>
cudaError_t launch_t(const SdpaLaunch& L, cudaStream_t stream) {
    using C = Cfg<HD, kHooks == 3>;
    // The CTAs of a last wave that fills no more than half of the SMs have one query tile each: a key step of
    // one tile takes about 1900 cycles, of two 2720, so that the wave ends after two thirds of the time.  A
    // row's arithmetic is the same in both.  1024 x 1024, 8 heads of 80 (32 items) 16.4 -> 13.7 us, 2042 x 2042,
    // 24 heads of 128 (192 items) 58.2 -> 53.6; a wave of 92 (2499 x 2499) would be two.  Calls without such a
    // wave keep the kernel whose CTAs all have two tiles: it issues its MMAs a little faster (4096 x 4096, 8 heads of
    // 40, 50.1 us against 53.1).
    const int sms = sm_count();
    const long long items = static_cast<long long>(L.q_ctas) * L.num_heads * L.batch, rest = items % sms;
    SdpaDevArgs args = L.args;
    args.q_ctas = L.q_ctas;
    args.num_heads = L.num_heads;
    args.whole_items = static_cast<int>(items - rest);
    const bool mixed = rest > 0 && 2 * rest <= sms && items < (1LL << 30);
    const dim3 grid = mixed ? dim3(static_cast<unsigned>(items + rest))
                            : dim3(static_cast<unsigned>(L.q_ctas), static_cast<unsigned>(L.num_heads), static_cast<unsigned>(L.batch));
    auto go = [&](auto kern) {
        cudaError_t e = set_max_smem_once(kern, C::kSmemBytes);
        if (e != cudaSuccess) return e;
        return launch_dependent(kern, grid, dim3(Roles<kScale>::kThreads), C::kSmemBytes, stream, L.tmQ[0], L.tmQ[1], L.tmK[0],
                                L.tmK[1], L.tmV[0], L.tmV[1], args);
    };
    return mixed ? go(sdpa_tc05_kernel<HD, kBf16, kHooks, kScale, true>) : go(sdpa_tc05_kernel<HD, kBf16, kHooks, kScale, false>);
}

template <int HD, bool kBf16>
cudaError_t launch_hd(const SdpaLaunch& L, cudaStream_t stream) {
    // 3: a logit bias and every other softmax hook; 2: key mask and statistics (a map), free of the bias's code
    // and with the third K tile that its rows take (mask and scales, 1033 x 1137, 24 heads of 128, 28.6 -> 27.1 us;
    // statistics 8.8 -> 8.1 at 344 tokens); 1: key mask only (the common case: padded captions; with the statistics'
    // store at its end 441 x 2365, 3 heads, takes 35.1 us instead of 32.9); 0: none.  The per-key scale vectors are
    // handled outside the softmax (kScale) and combine with 0, 2 and 3.
    const bool scale = L.args.key_scale != nullptr || L.args.val_scale != nullptr;
    if (L.args.bias != nullptr) {
        // A bias of few rows concerns a warp or two, and a piece of it behind the other through shared memory held up
        // the whole call: 32 rows x 1280 columns, 24 heads of 128, 49.2 us, a row per thread 37.4; 26 x 1096, 24 heads of 64, 31.7
        // and 27.4 (1024 rows x 256, 29.2 and 32.4).  Where every CTA has a single tile the pieces are all in flight
        // and the better choice (23 x 512, 24 heads of 40, 16.4 and 19.0) unless the rows are off 16 bytes (one row of 537, 25.7 and 22.1).
        const bool lone = 2LL * L.q_ctas * L.num_heads * L.batch <= sm_count();
        const bool rows16 = (L.args.bias_ld & 3) == 0 && (reinterpret_cast<uintptr_t>(L.args.bias) & 15u) == 0;
        if (L.args.bias_rows <= 32 && !(lone && rows16))
            return scale ? launch_t<HD, kBf16, 4, true>(L, stream) : launch_t<HD, kBf16, 4, false>(L, stream);
        return scale ? launch_t<HD, kBf16, 3, true>(L, stream) : launch_t<HD, kBf16, 3, false>(L, stream);
    }
    if (scale)
        return L.args.lse != nullptr || L.args.key_mask != nullptr ? launch_t<HD, kBf16, 2, true>(L, stream)
                                                                   : launch_t<HD, kBf16, 0, true>(L, stream);
    if (L.args.lse != nullptr) return launch_t<HD, kBf16, 2, false>(L, stream);
    if (L.args.key_mask != nullptr) return launch_t<HD, kBf16, 1, false>(L, stream);
    return launch_t<HD, kBf16, 0, false>(L, stream);
}

}  // namespace

cudaError_t launch_sdpa_tc05(const SdpaLaunch& L, cudaStream_t stream) {
    if (L.head_dim == 128) return L.bf16 ? launch_hd<128, true>(L, stream) : launch_hd<128, false>(L, stream);
    if (L.head_dim == 64) return L.bf16 ? launch_hd<64, true>(L, stream) : launch_hd<64, false>(L, stream);
    return cudaErrorInvalidValue;
}

}  // namespace bdattn
