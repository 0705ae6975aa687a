// Softmax attention forward for the head dims the tcgen05 kernel does not take (136
// to 256; SD1.5's deepest levels have 160), with the probabilities kept to FP32.
//
// These calls are small (64 to 576 queries, 8 heads): what counts is how many SMs a
// call reaches and how short a CTA's chain of loads and products is, so the tiles are
// far below a tcgen05 tile.  One CTA = 16 * MT query rows of one (batch, head); its
// four warps take the 16-key chunks of the sequence in turn, each with a ring of two
// K / V chunks of its own (cp.async, no CTA barrier in the loop) and a running
// maximum, sum and accumulator of its own, which are merged through shared memory at
// the end.  Products run on mma.sync m16n8k16 with FP32 accumulation; a probability is
// split into 16-bit parts, one product each, so that nothing is rounded to 16 bits before the
// output: three for BF16 (they add up to it exactly) and two for FP16 (23 of its 24 bits; the
// exponential itself is good to 2^-22.5).
// Two row tiles per CTA (MT = 2) halve the reads of K and V where there are still
// enough CTAs for that.
// 64 x 64 with 8 heads of 160: 4.2 us, 576 x 576: 22.3 us (97 and 840 on the CUDA-core kernel
// that stood here before).
// Same arithmetic as src/dit/common.cpp:246-305 with FP32 scores.
#include "sdpa_internal.h"
#include "tc05.cuh"

namespace bdattn {
namespace {

constexpr int kGWarps = 4;
constexpr int kGThreads = kGWarps * 32;
constexpr int kGKeys = 16;     // keys of a chunk

// Rows of HD elements, 16 bytes apart from a multiple of 32: an odd number of 16-byte
// units, so that the eight rows of an ldmatrix fall into different banks.
template <int HD>
struct GenCfg {
    static constexpr int kLd = HD + 8;                        // elements
    static constexpr int kChunk = kGKeys * kLd;               // elements of a K or V chunk
    static constexpr int kRing = kGWarps * 2 * 2 * kChunk * 2;   // bytes: two stages of K and V per warp
    static constexpr int kMergeLd = HD + 4;                   // floats
    static constexpr int smem(int mt) {
        const int q = 16 * mt * kLd * 2;
        const int merge = kGWarps * 16 * mt * (kMergeLd + 2) * 4;
        return q + (kRing > merge ? kRing : merge);
    }
};

__device__ __forceinline__ void gen_ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void gen_ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
template <bool kBf16>
__device__ __forceinline__ void gen_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    if constexpr (kBf16)
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
            "{%0, %1, %2, %3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
            "{%0, %1, %2, %3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// 16 bytes global -> shared; zeros where `live` is false (the source is not read then)
__device__ __forceinline__ void gen_cp16(uint32_t dst, const void* src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
// Takes the 16-bit part off a pair of floats: returns it packed, leaves the remainder.
template <bool kBf16>
__device__ __forceinline__ uint32_t gen_part(float& x, float& y) {
    const uint32_t w = pack2<kBf16>(x, y);
    if constexpr (kBf16) {
        x -= __uint_as_float(w << 16);
        y -= __uint_as_float(w & 0xffff0000u);
    } else {
        const __half2 h = *reinterpret_cast<const __half2*>(&w);
        x -= __low2float(h);
        y -= __high2float(h);
    }
    return w;
}

// Eight 16-bit values as floats.
template <bool kBf16>
__device__ __forceinline__ void gen_wide8(const uint16_t* src, float (&out)[8]) {
    const uint4 w = *reinterpret_cast<const uint4*>(src);
    const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if constexpr (kBf16) {
            out[2 * e] = __uint_as_float(ws[e] << 16);
            out[2 * e + 1] = __uint_as_float(ws[e] & 0xffff0000u);
        } else {
            const __half2 h = *reinterpret_cast<const __half2*>(&ws[e]);
            out[2 * e] = __low2float(h);
            out[2 * e + 1] = __high2float(h);
        }
    }
}

// The output of a CTA again, with plain FP32 products, when some value of it was not finite (an infinity
// or NaN among the inputs): a weight split into parts has parts that are zero or negative, whose
// product with an infinite value is NaN.  Q rows in Qs; the four warps' row maxima and sums of the first
// pass in the merge area.  `boost`: the factor those sums carry.
// A function of its own that is not inlined: in line it changed how the loop of the first pass
// was compiled (576 x 576, 24 heads of 160: 53.9 -> 65.6 us); called, it costs that pass nothing.
template <int HD, int MT, bool kBf16>
__device__ __noinline__ void gen_plain(const SdpaGeneralArgs& a, int q_ctas0, float boost, const uint16_t* Qs, uint8_t* ring) {
    using C = GenCfg<HD>;
    constexpr int kRows = 16 * MT;
    const int hd = a.head_dim, vecs = hd >> 3;
    const int head = blockIdx.y, batch = blockIdx.z;
    const int qseg = static_cast<int>(blockIdx.x) >= q_ctas0 ? 1 : 0;
    const int qrow0 = (qseg ? static_cast<int>(blockIdx.x) - q_ctas0 : static_cast<int>(blockIdx.x)) * kRows;
    const int seg_rows = qseg ? a.q_rows[1] : a.q_rows[0];
    const int q_glob0 = (qseg ? a.q_rows[0] : 0) + qrow0;
    const int Lk = a.kv_rows[0] + a.kv_rows[1];
    int k_end = Lk;
    if (a.mask_mode == 1) k_end = max(0, min(Lk, q_glob0 + min(kRows, seg_rows - qrow0) + a.q_offset));
    const long long kv_col = static_cast<long long>(head / a.kv_group) * hd;
    const float sl2 = a.scale * 1.4426950408889634f;

    float* Om = reinterpret_cast<float*>(ring);
    const float* Sm = Om + kGWarps * kRows * C::kMergeLd;
    float* const Ms = Om;                        // [kRows] maximum, [kRows] 1 / sum
    float* const Ps = Om + 2 * kRows;            // [kRows][33]
    if (threadIdx.x < kRows) {
        float m = -INFINITY, l = 0.0f;
        for (int w = 0; w < kGWarps; ++w) m = fmaxf(m, Sm[(w * kRows + threadIdx.x) * 2]);
        for (int w = 0; w < kGWarps; ++w) {
            const float mw = Sm[(w * kRows + threadIdx.x) * 2];
            l += mw == -INFINITY ? 0.0f : fast_exp2(mw - m) * Sm[(w * kRows + threadIdx.x) * 2 + 1];
        }
        Ms[threadIdx.x] = m == -INFINITY ? 0.0f : m;
        Ms[kRows + threadIdx.x] = l > 0.0f ? boost / l : 0.0f;
    }
    auto row_of = [&](const void* const (&p)[2], const long long (&ld)[2], const long long (&bs)[2], int kg) {
        const int seg = kg >= a.kv_rows[0] ? 1 : 0;
        const long long rr = seg ? kg - a.kv_rows[0] : kg;
        return static_cast<const uint16_t*>(seg ? p[1] : p[0]) + (batch * (seg ? bs[1] : bs[0]) + rr * (seg ? ld[1] : ld[0]) + kv_col);
    };
    constexpr int kItems = (kRows * (HD / 8) + kGThreads - 1) / kGThreads;    // output vectors of a thread
    float acc[kItems][8];
#pragma unroll
    for (int j = 0; j < kItems; ++j)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[j][e] = 0.0f;
#pragma unroll 1
    for (int k0 = 0; k0 < k_end; k0 += 32) {
        __syncthreads();
#pragma unroll 1
        for (int i = threadIdx.x; i < kRows * 32; i += kGThreads) {
            const int r = i >> 5, kg = k0 + (i & 31);
            const bool vis = kg < Lk && (a.mask_mode != 1 || kg <= q_glob0 + r + a.q_offset) &&
                             (a.key_mask == nullptr || __ldg(a.key_mask + kg) != 0.0f);
            float p = 0.0f;
            if (vis) {
                const uint16_t* kr = row_of(a.k, a.k_ld, a.k_bs, kg);
                float dot = 0.0f;
#pragma unroll 1
                for (int d = 0; d < hd; d += 8) {
                    float qv[8], kv[8];
                    gen_wide8<kBf16>(Qs + r * C::kLd + d, qv);
                    gen_wide8<kBf16>(kr + d, kv);
#pragma unroll
                    for (int e = 0; e < 8; ++e) dot = fmaf(qv[e], kv[e], dot);
                }
                p = fast_exp2(dot * (sl2 * (a.key_scale != nullptr ? __ldg(a.key_scale + kg) : 1.0f)) - Ms[r]) * Ms[kRows + r];
            }
            Ps[r * 33 + (i & 31)] = p;
        }
        __syncthreads();
#pragma unroll 1
        for (int kk = 0; kk < min(32, Lk - k0); ++kk) {
            const uint16_t* vr = row_of(a.v, a.v_ld, a.v_bs, k0 + kk);
            const float sc = a.val_scale != nullptr ? __ldg(a.val_scale + k0 + kk) : 1.0f;
#pragma unroll
            for (int j = 0; j < kItems; ++j) {
                const int i = threadIdx.x + j * kGThreads, r = i / vecs;
                if (r < kRows) {
                    const float p = Ps[r * 33 + kk];
                    float vv[8];
                    gen_wide8<kBf16>(vr + (i - r * vecs) * 8, vv);
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[j][e] = fmaf(p, vv[e] * sc, acc[j][e]);
                }
            }
        }
    }
    uint16_t* op = static_cast<uint16_t*>(qseg ? a.o[1] : a.o[0]) + batch * (qseg ? a.o_bs[1] : a.o_bs[0]) +
                   static_cast<long long>(head) * hd;
    const long long o_ld = qseg ? a.o_ld[1] : a.o_ld[0];
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const int i = threadIdx.x + j * kGThreads, r = i / vecs;
        if (r < kRows && qrow0 + r < seg_rows) {
            uint4 w4;
            w4.x = pack2<kBf16>(acc[j][0], acc[j][1]); w4.y = pack2<kBf16>(acc[j][2], acc[j][3]);
            w4.z = pack2<kBf16>(acc[j][4], acc[j][5]); w4.w = pack2<kBf16>(acc[j][6], acc[j][7]);
            *reinterpret_cast<uint4*>(op + static_cast<long long>(qrow0 + r) * o_ld + (i - r * vecs) * 8) = w4;
        }
    }
}

// kWide (FP16 with value scales): a weight, the probability times its scale, has the range of FP32, which
// FP16 parts do not.  Weights are split into BF16 parts as with BF16 values, and a value of FP16 into
// two BF16 parts that add up to it.
template <int HD, int MT, bool kBf16, bool kWide>
__global__ void __launch_bounds__(kGThreads)
sdpa_general_kernel(const __grid_constant__ SdpaGeneralArgs a, int q_ctas0) {
    using C = GenCfg<HD>;
    constexpr bool kBf16Parts = kBf16 || kWide;
    constexpr int kParts = kBf16Parts ? 3 : 2;
    extern __shared__ __align__(16) uint8_t gsm[];
    uint16_t* Qs = reinterpret_cast<uint16_t*>(gsm);                                    // [16 * MT][kLd]
    uint8_t* ring = gsm + 16 * MT * C::kLd * 2;

    dependents_may_launch();
    wait_for_prior_grid();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, q4 = lane & 3;
    const int hd = a.head_dim, vecs = hd >> 3;
    const int head = blockIdx.y, batch = blockIdx.z;
    const int qseg = static_cast<int>(blockIdx.x) >= q_ctas0 ? 1 : 0;
    const int qrow0 = (qseg ? static_cast<int>(blockIdx.x) - q_ctas0 : static_cast<int>(blockIdx.x)) * (16 * MT);
    const int seg_rows = qseg ? a.q_rows[1] : a.q_rows[0];
    const int q_glob0 = (qseg ? a.q_rows[0] : 0) + qrow0;
    const int Lk = a.kv_rows[0] + a.kv_rows[1];
    int k_end = Lk;
    if (a.mask_mode == 1) {
        const int last = q_glob0 + min(16 * MT, seg_rows - qrow0) - 1;
        k_end = max(0, min(Lk, last + a.q_offset + 1));
    }
    const int n_chunks = (k_end + kGKeys - 1) / kGKeys;
    const long long kv_col = static_cast<long long>(head / a.kv_group) * hd;

    // K / V chunk `ch` into stage `st` of this warp's ring.  Columns past head_dim and keys past
    // the sequence read as zero.
    uint16_t* wring = reinterpret_cast<uint16_t*>(ring) + warp * 4 * C::kChunk;
    auto fetch = [&](int ch, int st) {
        const uint32_t kd = smem_u32(wring + st * 2 * C::kChunk);
#pragma unroll 2
        for (int i = lane; i < kGKeys * (HD / 8); i += 32) {
            const int kk = i / (HD / 8), v = i - kk * (HD / 8);
            const int kg = ch * kGKeys + kk;
            const bool live = kg < Lk && v < vecs;
            const int seg = live && kg >= a.kv_rows[0] ? 1 : 0;
            const long long rr = live ? (seg ? kg - a.kv_rows[0] : kg) : 0;
            const long long col = live ? kv_col + v * 8 : 0;
            const uint16_t* kp = static_cast<const uint16_t*>(seg ? a.k[1] : a.k[0]) +
                                 (batch * (seg ? a.k_bs[1] : a.k_bs[0]) + rr * (seg ? a.k_ld[1] : a.k_ld[0]) + col);
            const uint16_t* vp = static_cast<const uint16_t*>(seg ? a.v[1] : a.v[0]) +
                                 (batch * (seg ? a.v_bs[1] : a.v_bs[0]) + rr * (seg ? a.v_ld[1] : a.v_ld[0]) + col);
            const uint32_t d = kd + (kk * C::kLd + v * 8) * 2;
            gen_cp16(d, kp, live);
            gen_cp16(d + C::kChunk * 2, vp, live);
        }
    };

    // Q rows (zero past the segment and past head_dim)
    {
        const uint16_t* qp = static_cast<const uint16_t*>(qseg ? a.q[1] : a.q[0]) + batch * (qseg ? a.q_bs[1] : a.q_bs[0]) +
                             static_cast<long long>(head) * hd;
        const long long q_ld = qseg ? a.q_ld[1] : a.q_ld[0];
        for (int i = threadIdx.x; i < 16 * MT * (HD / 8); i += kGThreads) {
            const int r = i / (HD / 8), v = i - r * (HD / 8);
            const bool live = qrow0 + r < seg_rows && v < vecs;
            gen_cp16(smem_u32(Qs + r * C::kLd + v * 8), qp + (live ? static_cast<long long>(qrow0 + r) * q_ld + v * 8 : 0), live);
        }
    }
    if (warp < n_chunks) fetch(warp, 0);
    asm volatile("cp.async.commit_group;" ::: "memory");

    // FP16: probabilities carry a factor of 2^15, which keeps the parts of small ones out of the subnormals
    // and cancels in O / l.  It is multiplied on, exactly: added to the exponent it costs the argument
    // of a probability near one its last three bits.
    constexpr float kBoost = kBf16Parts ? 1.0f : 32768.0f;

    float o[MT][HD / 8][4];
    float m_run[MT][2], l_run[MT][2];
#pragma unroll
    for (int t = 0; t < MT; ++t) {
        m_run[t][0] = m_run[t][1] = -INFINITY;
        l_run[t][0] = l_run[t][1] = 0.0f;
#pragma unroll
        for (int n = 0; n < HD / 8; ++n) o[t][n][0] = o[t][n][1] = o[t][n][2] = o[t][n][3] = 0.0f;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                             // Q from all warps

    const float sl2 = a.scale * 1.4426950408889634f;
    const uint32_t q_addr = smem_u32(Qs + (lane & 15) * C::kLd + (lane >> 4) * 8);
    int st = 0;
    for (int ch = warp; ch < n_chunks; ch += kGWarps, st ^= 1) {
        if (ch + kGWarps < n_chunks) fetch(ch + kGWarps, st ^ 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");      // this chunk (all but the newest group)
        __syncwarp();
        const uint16_t* Kc = wring + st * 2 * C::kChunk;
        // B fragments: K is (key, d) = (n, k) row-major; matrices keys 0-7 | 8-15 x d 0-7 | 8-15
        const uint32_t k_addr = smem_u32(Kc + ((lane & 7) + ((lane >> 4) << 3)) * C::kLd + ((lane >> 3) & 1) * 8);
        const uint32_t v_addr = smem_u32(Kc + C::kChunk + (lane & 15) * C::kLd + (lane >> 4) * 8);

        float s[MT][2][4];
#pragma unroll
        for (int t = 0; t < MT; ++t)
#pragma unroll
            for (int n = 0; n < 2; ++n) s[t][n][0] = s[t][n][1] = s[t][n][2] = s[t][n][3] = 0.0f;
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
            uint32_t b[4];
            gen_ldsm4(b, k_addr + kk * 32);
#pragma unroll
            for (int t = 0; t < MT; ++t) {
                uint32_t qa[4];
                gen_ldsm4(qa, q_addr + t * 16 * C::kLd * 2 + kk * 32);
                gen_mma<kBf16>(s[t][0], qa, b[0], b[1]);
                gen_mma<kBf16>(s[t][1], qa, b[2], b[3]);
            }
        }

        // this thread's four keys: 2 * q4 + {0, 1} and the same + 8
        float ks[4], vs[4];
        bool seen[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int kg = ch * kGKeys + (i >> 1) * 8 + q4 * 2 + (i & 1);
            const bool in = kg < Lk;
            seen[i] = in && (a.key_mask == nullptr || __ldg(a.key_mask + kg) != 0.0f);
            ks[i] = sl2 * (in && a.key_scale != nullptr ? __ldg(a.key_scale + kg) : 1.0f);
            vs[i] = kBf16Parts && in && a.val_scale != nullptr ? __ldg(a.val_scale + kg) : 1.0f;
        }
        uint32_t pa[MT][kParts][4];
#pragma unroll
        for (int t = 0; t < MT; ++t) {
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {                      // row g, row g + 8
                const int q_glob = q_glob0 + t * 16 + hf * 8 + g;
                float x[4];
                float mx = -INFINITY;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int kg = ch * kGKeys + (i >> 1) * 8 + q4 * 2 + (i & 1);
                    const bool vis = seen[i] && (a.mask_mode != 1 || kg <= q_glob + a.q_offset);
                    x[i] = vis ? s[t][i >> 1][hf * 2 + (i & 1)] * ks[i] : -INFINITY;
                    mx = fmaxf(mx, x[i]);
                }
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                const float m_new = fmaxf(m_run[t][hf], mx);
                const float m_use = m_new == -INFINITY ? 0.0f : m_new;
                if (m_new != m_run[t][hf]) {
                    const float alpha = m_run[t][hf] == -INFINITY ? 0.0f : fast_exp2(m_run[t][hf] - m_use);
                    l_run[t][hf] *= alpha;
#pragma unroll
                    for (int n = 0; n < HD / 8; ++n) {
                        o[t][n][hf * 2] *= alpha;
                        o[t][n][hf * 2 + 1] *= alpha;
                    }
                    m_run[t][hf] = m_new;
                }
                float p[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    p[i] = fast_exp2(x[i] - m_use) * kBoost;
                    l_run[t][hf] += p[i];
                    if constexpr (kBf16Parts) p[i] *= vs[i];
                }
#pragma unroll
                for (int k = 0; k < kParts; ++k) {
                    pa[t][k][hf] = gen_part<kBf16Parts>(p[0], p[1]);          // keys 2 q4, 2 q4 + 1
                    pa[t][k][2 + hf] = gen_part<kBf16Parts>(p[2], p[3]);      // the same + 8
                }
            }
        }
#pragma unroll
        for (int n = 0; n < HD / 16; ++n) {
            uint32_t b[4];
            gen_ldsm4_t(b, v_addr + n * 32);
            if constexpr (kWide) {
                uint32_t rest[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const __half2 h = *reinterpret_cast<const __half2*>(&b[i]);
                    float lo = __low2float(h), hi = __high2float(h);
                    b[i] = gen_part<true>(lo, hi);
                    rest[i] = pack2<true>(lo, hi);
                }
#pragma unroll
                for (int t = 0; t < MT; ++t) {
#pragma unroll
                    for (int k = kParts - 1; k >= 0; --k) {
                        gen_mma<true>(o[t][2 * n], pa[t][k], rest[0], rest[1]);
                        gen_mma<true>(o[t][2 * n + 1], pa[t][k], rest[2], rest[3]);
                    }
                }
            }
#pragma unroll
            for (int t = 0; t < MT; ++t) {
#pragma unroll
                for (int k = kParts - 1; k >= 0; --k) {                  // smallest part first
                    gen_mma<kBf16Parts>(o[t][2 * n], pa[t][k], b[0], b[1]);
                    gen_mma<kBf16Parts>(o[t][2 * n + 1], pa[t][k], b[2], b[3]);
                }
            }
        }
        __syncwarp();                            // the stage is refilled in the next step
    }

    // merge of the four warps' results (the ring is at rest)
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    constexpr int kRows = 16 * MT;
    float* Om = reinterpret_cast<float*>(ring);                          // [warps][kRows][kMergeLd]
    float* Sm = Om + kGWarps * kRows * C::kMergeLd;                      // [warps][kRows][2]
#pragma unroll
    for (int t = 0; t < MT; ++t) {
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int r = t * 16 + hf * 8 + g;
            float l = l_run[t][hf];
            l += __shfl_xor_sync(0xffffffffu, l, 1);
            l += __shfl_xor_sync(0xffffffffu, l, 2);
            if (q4 == 0) {
                Sm[(warp * kRows + r) * 2] = m_run[t][hf];
                Sm[(warp * kRows + r) * 2 + 1] = l;
            }
            float* orow = Om + (warp * kRows + r) * C::kMergeLd + q4 * 2;
#pragma unroll
            for (int n = 0; n < HD / 8; ++n)
                *reinterpret_cast<float2*>(orow + n * 8) = make_float2(o[t][n][hf * 2], o[t][n][hf * 2 + 1]);
        }
    }
    __syncthreads();
    uint16_t* op = static_cast<uint16_t*>(qseg ? a.o[1] : a.o[0]) + batch * (qseg ? a.o_bs[1] : a.o_bs[0]) +
                   static_cast<long long>(head) * hd;
    const long long o_ld = qseg ? a.o_ld[1] : a.o_ld[0];
    bool finite = true;
    for (int i = threadIdx.x; i < kRows * vecs; i += kGThreads) {
        const int r = i / vecs, v = i - r * vecs;
        if (qrow0 + r >= seg_rows) break;        // rows only grow from here on
        float m = -INFINITY;
#pragma unroll
        for (int w = 0; w < kGWarps; ++w) m = fmaxf(m, Sm[(w * kRows + r) * 2]);
        float l = 0.0f, f[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = 0.0f;
#pragma unroll
        for (int w = 0; w < kGWarps; ++w) {
            const float mw = Sm[(w * kRows + r) * 2];
            const float c = mw == -INFINITY ? 0.0f : fast_exp2(mw - m);
            l = fmaf(c, Sm[(w * kRows + r) * 2 + 1], l);
            const float* src = Om + (w * kRows + r) * C::kMergeLd + v * 8;
            const float4 u0 = *reinterpret_cast<const float4*>(src), u1 = *reinterpret_cast<const float4*>(src + 4);
            f[0] = fmaf(c, u0.x, f[0]); f[1] = fmaf(c, u0.y, f[1]); f[2] = fmaf(c, u0.z, f[2]); f[3] = fmaf(c, u0.w, f[3]);
            f[4] = fmaf(c, u1.x, f[4]); f[5] = fmaf(c, u1.y, f[5]); f[6] = fmaf(c, u1.z, f[6]); f[7] = fmaf(c, u1.w, f[7]);
        }
        const float inv = l > 0.0f ? 1.0f / l : 0.0f;
        float t = 0.0f;                          // NaN once a value is not finite
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            f[e] *= inv;
            t = fmaf(f[e], 0.0f, t);
        }
        finite = finite && t == 0.0f;
        uint4 w4;
        w4.x = pack2<kBf16>(f[0], f[1]); w4.y = pack2<kBf16>(f[2], f[3]);
        w4.z = pack2<kBf16>(f[4], f[5]); w4.w = pack2<kBf16>(f[6], f[7]);
        *reinterpret_cast<uint4*>(op + static_cast<long long>(qrow0 + r) * o_ld + v * 8) = w4;
    }
    if (__syncthreads_or(!finite)) gen_plain<HD, MT, kBf16>(a, q_ctas0, kBoost, Qs, ring);
}

template <int HD, int MT, bool kBf16, bool kWide>
cudaError_t launch_general_t(const SdpaGeneralArgs& a, int num_heads, int batch, cudaStream_t stream) {
    auto kern = sdpa_general_kernel<HD, MT, kBf16, kWide>;
    constexpr int smem = GenCfg<HD>::smem(MT);
    cudaError_t e = set_max_smem_once(kern, smem);
    if (e != cudaSuccess) return e;
    const int q_ctas0 = (a.q_rows[0] + 16 * MT - 1) / (16 * MT);
    const int q_ctas1 = (a.q_rows[1] + 16 * MT - 1) / (16 * MT);
    dim3 grid(static_cast<unsigned>(q_ctas0 + q_ctas1), static_cast<unsigned>(num_heads),
              static_cast<unsigned>(batch));
    return launch_dependent(kern, grid, dim3(kGThreads), smem, stream, a, q_ctas0);
}

template <int HD, int MT>
cudaError_t launch_general_hd(const SdpaGeneralArgs& a, int num_heads, int batch, bool bf16, cudaStream_t stream) {
    if (bf16) return launch_general_t<HD, MT, true, false>(a, num_heads, batch, stream);
    return a.val_scale != nullptr ? launch_general_t<HD, MT, false, true>(a, num_heads, batch, stream)
                                  : launch_general_t<HD, MT, false, false>(a, num_heads, batch, stream);
}

}  // namespace

cudaError_t launch_sdpa_general(const SdpaGeneralArgs& a, int num_heads, int batch, bool bf16,
                                cudaStream_t stream) {
    if (a.head_dim > 160) return launch_general_hd<256, 1>(a, num_heads, batch, bf16, stream);
    // two row tiles per CTA once that still leaves one CTA per SM
    const long long rows = static_cast<long long>(a.q_rows[0]) + a.q_rows[1];
    if ((rows + 31) / 32 * num_heads * batch >= sm_count())
        return launch_general_hd<160, 2>(a, num_heads, batch, bf16, stream);
    return launch_general_hd<160, 1>(a, num_heads, batch, bf16, stream);
}

}  // namespace bdattn
