// attention_prefill_f32.cuh -- attention of a block of 128 query rows on the f32 FMA pipe, head size 128.
//
// What lux_attn_prefill_mma_f32 does with a block in which it met values that its bf16 parts cannot carry (2^60 and
// more, infinities, NaN; outputs below 2^-100): the block starts over here, in the same CTA, before anything of it was written, and
// no other block notices.  lux_attn_prefill_f32 runs it for every block (no scratch to be had; tunable attn_prefill = 3: the tests).
//
// What bounds it.  Both contractions are f32 products of f32 operands, so the FMA pipe is the floor: 128 lanes x 148
// SMs (72 TFLOP/s at 1.9 GHz).  A 16-byte shared-memory read costs the SM four cycles however many lanes read
// the same bytes, so the floor in practice is set by FMAs per read: 8 in lux_attn_stream_f32, 16 (scores) and
// 26 (weighted sum) here.  2048 causal tokens, Llama-3-8B heads, all blocks: 956 us (36 TFLOP/s; streaming kernel 1679).
// The contractions are register-tiled like a matrix product:
//   * a CTA of 256 threads owns 128 queries of one head and walks 64-key tiles;
//   * a thread owns rows tr + 32 i (i < 4) with tr = tid / 8.  Scores: keys tc + 8 j (j < 8, tc = tid % 8),
//     four keys at a time: 8 16-byte reads per 64 FMAs.  Weighted sum: columns 32 j + 4 tc .. + 3;
//   * FMAs go through fma.rn.f32x2 (two IEEE f32 FMAs per instruction, the same rounding as fmaf).  The
//     pairs are neighbouring head columns, as they lie in memory: a score is kept as its even- and its
//     odd-column half;
//   * rows of Q and K are 132 floats apart in shared memory: the four rows and eight keys that a warp
//     reads in one instruction then lie in different banks.  K arrives by one bulk copy per row, V (read
//     along its rows) by one per tile;
//   * a warp owns its 16 rows (four values of tr) through the softmax, so the weights pass from the score layout to the
//     weighted-sum layout through a warp-private piece of shared memory, 32 keys at a time;
//   * the next K tile is requested when the scores are done, the next V tile when the weighted sum is.
// Long sums are cut so that no rounding chain is longer than in the streaming kernel's lanes: scores
// are folded every 32 columns (chains of 16 per half), the weighted sum every 32 keys, the denominator
// every tile.
// A masked (row, key) pair takes no part in the sums at all (a predicated FMA, not a zero weight): an
// infinite or NaN value at a position that a row must not see does not reach it.
#pragma once

#include "common.cuh"
#include "tc_ptx.cuh"

#include <type_traits>

namespace luxcuda {
namespace {
namespace prefill {

using namespace tcptx;

constexpr int PF_D = 128;                 // head size
constexpr int PF_BM = 128;                // queries per CTA
constexpr int PF_BN = 64;                 // keys per tile
constexpr int PF_THREADS = 256;
constexpr int PF_PITCH = PF_D + 4;        // floats between rows of Q and K in shared memory
constexpr int PF_PW = 32;                 // keys whose weights are passed on at a time
constexpr int PF_PPITCH = PF_PW + 8;      // floats between rows of the weights
constexpr int PF_Q_FLOATS = PF_BM * PF_PITCH, PF_K_FLOATS = PF_BN * PF_PITCH, PF_V_FLOATS = PF_BN * PF_D,
              PF_P_FLOATS = PF_BM * PF_PPITCH;
// Q, K, V, weights, then two mbarriers and the abort flag: 151 KB
constexpr int PF_SMEM = (PF_Q_FLOATS + PF_K_FLOATS + PF_V_FLOATS + PF_P_FLOATS) * 4 + 32;

__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// c + a * b where `take`, c elsewhere
__device__ __forceinline__ uint64_t fma2_if(bool take, uint64_t a, uint64_t b, uint64_t c) {
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p fma.rn.f32x2 %0, %1, %2, %0;\n\t}" : "+l"(c) : "l"(a), "l"(b), "r"((uint32_t)take));
    return c;
}
__device__ __forceinline__ uint64_t pair(float lo, float hi) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ void unpair(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
struct Pair2 { uint64_t a, b; };          // 16 bytes of shared memory: two pairs of neighbouring floats
__device__ __forceinline__ Pair2 lds_pairs(uint32_t addr) {
    Pair2 r;
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(r.a), "=l"(r.b) : "r"(addr));
    return r;
}
__device__ __forceinline__ float4 lds4(uint32_t addr) {
    float4 r;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "r"(addr));
    return r;
}


__device__ __forceinline__ float ex2(float x) {                // as in the streaming kernel
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

constexpr float PF_NEG = -3.0e38f;        // "no key seen yet" in the base-2 score domain
constexpr float PF_LN2 = 0.6931471805599453f;

// The block's own barrier: its 256 threads may be part of a larger CTA.
__device__ __forceinline__ void block_sync() { named_bar_sync_c<1>(PF_THREADS); }
__device__ __forceinline__ bool block_or(bool v) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(r) : "r"((uint32_t)v), "n"(PF_THREADS) : "memory");
    return r != 0u;
}

// Block qb of head h of sequence b.  The first 256 threads of the CTA call it, with 128-byte aligned shared memory that no copy
// in flight still writes.
__device__ __forceinline__ void attend_f32(const PrefillArgs& p, unsigned char* smem, uint32_t qb, uint32_t h, uint32_t b) {
    float* qs = reinterpret_cast<float*>(smem);
    float* ks = qs + PF_Q_FLOATS;
    float* vs = ks + PF_K_FLOATS;
    float* ps = vs + PF_V_FLOATS;
    uint64_t* bars = reinterpret_cast<uint64_t*>(ps + PF_P_FLOATS);
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(bars + 2);
    const uint32_t bar_k = smem_u32(bars), bar_v = bar_k + 8u;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tr = tid >> 3, tc = tid & 7;

    fence_proxy_async_smem();             // copies are about to land where this thread may have written
    block_sync();
    if (tid == 0) {
        mbar_init(bar_k, 1u);
        mbar_init(bar_v, 1u);
        *abort_flag = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    block_sync();
    const uint32_t g = h / p.group;
    const uint32_t q0 = qb * PF_BM;
    const uint32_t rows = min((uint32_t)PF_BM, p.seq_q - q0);
    auto row_len = [&](uint32_t qi) { return p.causal ? min(p.causal_base + qi + 1u, p.kv_len) : p.kv_len; };
    const uint32_t lmax = row_len(q0 + rows - 1u);
    const uint32_t tiles = (lmax + PF_BN - 1u) / PF_BN;
    const float* kbase = p.k + ((size_t)b * p.kv_heads + g) * p.kv_stride * PF_D;
    const float* vbase = p.v + ((size_t)b * p.kv_heads + g) * p.kv_stride * PF_D;

    // warp 0 requests tiles: one copy per row of K (padded rows), one for all of V
    auto load_k = [&](uint32_t t) {
        const uint32_t t0 = t * PF_BN, nk = min((uint32_t)PF_BN, lmax - t0);
        if (lane == 0) mbar_expect_tx(bar_k, nk * PF_D * 4u);
        __syncwarp();
        for (uint32_t r = lane; r < nk; r += 32) bulk_g2s(smem_u32(ks + r * PF_PITCH), kbase + (size_t)(t0 + r) * PF_D, PF_D * 4u, bar_k);
    };
    auto load_v = [&](uint32_t t) {
        const uint32_t t0 = t * PF_BN, nk = min((uint32_t)PF_BN, lmax - t0);
        if (lane == 0) {
            mbar_expect_tx(bar_v, nk * PF_D * 4u);
            bulk_g2s(smem_u32(vs), vbase + (size_t)t0 * PF_D, nk * PF_D * 4u, bar_v);
        }
    };
    if (warp == 0 && tiles) {
        load_k(0);
        load_v(0);
    }
    {
        const float* qsrc = p.q + (((size_t)b * p.heads + h) * p.seq_q + q0) * PF_D;
#pragma unroll 4
        for (int e = tid; e < PF_BM * (PF_D / 4); e += PF_THREADS) {
            const int r = e / (PF_D / 4), c = e % (PF_D / 4);
            float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
            if ((uint32_t)r < rows) t = __ldg(reinterpret_cast<const float4*>(qsrc + (size_t)r * PF_D) + c);
            *reinterpret_cast<float4*>(qs + r * PF_PITCH + c * 4) = make_float4(t.x * p.qscale, t.y * p.qscale, t.z * p.qscale, t.w * p.qscale);
        }
    }
    block_sync();

    uint64_t o[4][8];                     // row tr + 32 i, columns 32 (j / 2) + 4 tc + 2 (j % 2) and the next
    float m[4], l[4];
    uint32_t len[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t qi = q0 + tr + 32 * i;
        len[i] = tr + 32 * i < (int)rows ? row_len(qi) : 0u;        // a padding row sees nothing and is not written
        m[i] = PF_NEG;
        l[i] = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; j++) o[i][j] = 0ull;
    }
    const uint32_t min_len = row_len(q0);
    const uint32_t qaddr = smem_u32(qs) + (uint32_t)(tr * PF_PITCH * 4), kaddr = smem_u32(ks) + (uint32_t)(tc * PF_PITCH * 4);
    const uint32_t vaddr = smem_u32(vs) + (uint32_t)tc * 16u, paddr = smem_u32(ps) + (uint32_t)(tr * PF_PPITCH * 4);

    // weighted sum over PF_PW keys of the tile whose weights lie in `ps`; MASKED skips pairs past a row's length
    auto weighted = [&](auto masked, uint32_t key0, uint32_t t0) {
        constexpr bool MASKED = decltype(masked)::value;
        uint64_t acc[4][8];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) acc[i][j] = 0ull;
#pragma unroll 1
        for (uint32_t kk = 0; kk < PF_PW; kk += 4) {
            float w[4][4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float4 t = lds4(paddr + (uint32_t)(32 * i * PF_PPITCH * 4) + kk * 4u);
                w[i][0] = t.x; w[i][1] = t.y; w[i][2] = t.z; w[i][3] = t.w;
            }
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const uint32_t va = vaddr + (key0 + kk + e) * (PF_D * 4u);
                Pair2 v[4];
#pragma unroll
                for (int j = 0; j < 4; j++) v[j] = lds_pairs(va + (uint32_t)j * 128u);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const uint64_t ww = pair(w[i][e], w[i][e]);
                    const bool take = !MASKED || t0 + key0 + kk + e < len[i];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        if (MASKED) {
                            acc[i][2 * j] = fma2_if(take, ww, v[j].a, acc[i][2 * j]);
                            acc[i][2 * j + 1] = fma2_if(take, ww, v[j].b, acc[i][2 * j + 1]);
                        } else {
                            acc[i][2 * j] = fma2(ww, v[j].a, acc[i][2 * j]);
                            acc[i][2 * j + 1] = fma2(ww, v[j].b, acc[i][2 * j + 1]);
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) o[i][j] = add2(o[i][j], acc[i][j]);
    };

    bool ok = true;
    for (uint32_t t = 0; t < tiles; t++) {
        const uint32_t t0 = t * PF_BN;
        const bool edge = t0 + PF_BN > min_len;          // some row of the CTA does not see the whole tile
        float s[4][8];
        ok = warp_wait(bar_k, t & 1u, abort_flag, lane);
        if (ok) {
#pragma unroll
            for (int hf = 0; hf < 2; hf++) {
                uint64_t tot[4][4];
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) tot[i][j] = 0ull;
#pragma unroll 1
                for (int d0 = 0; d0 < PF_D; d0 += 32) {
                    uint64_t acc[4][4];
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int j = 0; j < 4; j++) acc[i][j] = 0ull;
#pragma unroll
                    for (int d = 0; d < 32; d += 4) {
                        Pair2 qv[4], kv[4];
#pragma unroll
                        for (int i = 0; i < 4; i++) qv[i] = lds_pairs(qaddr + (uint32_t)(32 * i * PF_PITCH * 4 + (d0 + d) * 4));
#pragma unroll
                        for (int j = 0; j < 4; j++) kv[j] = lds_pairs(kaddr + (uint32_t)(8 * (4 * hf + j) * PF_PITCH * 4 + (d0 + d) * 4));
#pragma unroll
                        for (int i = 0; i < 4; i++)
#pragma unroll
                            for (int j = 0; j < 4; j++) {
                                acc[i][j] = fma2(qv[i].a, kv[j].a, acc[i][j]);
                                acc[i][j] = fma2(qv[i].b, kv[j].b, acc[i][j]);
                            }
                    }
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int j = 0; j < 4; j++) tot[i][j] = add2(tot[i][j], acc[i][j]);
                }
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        float lo, hi;
                        unpair(tot[i][j], lo, hi);
                        s[i][4 * hf + j] = lo + hi;
                    }
            }
        }
        // K has been read by every warp: the next tile may land
        if (block_or(!ok)) { ok = false; break; }
        if (warp == 0 && t + 1 < tiles) load_k(t + 1);

        // running maximum per row (the 8 lanes of a row agree on it), raised only when a score passes it
        // by more than 8 in the base-2 domain, so that weights stay below 2^8 and most tiles rescale nothing
        float mt[4];
        bool up = false;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            mt[i] = PF_NEG;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                if (edge && t0 + tc + 8 * j >= len[i]) s[i][j] = -__int_as_float(0x7f800000);
                mt[i] = fmaxf(mt[i], s[i][j]);
            }
            mt[i] = fmaxf(mt[i], __shfl_xor_sync(0xffffffffu, mt[i], 1));
            mt[i] = fmaxf(mt[i], __shfl_xor_sync(0xffffffffu, mt[i], 2));
            mt[i] = fmaxf(mt[i], __shfl_xor_sync(0xffffffffu, mt[i], 4));
            up |= mt[i] > m[i] + 8.0f;
        }
        if (__any_sync(0xffffffffu, up)) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float mn = fmaxf(m[i], mt[i]), alpha = ex2(m[i] - mn);
                const uint64_t aa = pair(alpha, alpha);
                m[i] = mn;
                l[i] *= alpha;
#pragma unroll
                for (int j = 0; j < 8; j++) o[i][j] = mul2(o[i][j], aa);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
#pragma unroll
            for (int j = 0; j < 8; j++) s[i][j] = ex2(s[i][j] - m[i]);
            l[i] += ((s[i][0] + s[i][1]) + (s[i][2] + s[i][3])) + ((s[i][4] + s[i][5]) + (s[i][6] + s[i][7]));
        }

        ok = warp_wait(bar_v, t & 1u, abort_flag, lane);
        if (ok) {
#pragma unroll
            for (int hf = 0; hf < 2; hf++) {
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) ps[(tr + 32 * i) * PF_PPITCH + tc + 8 * j] = s[i][4 * hf + j];
                __syncwarp();
                if (edge) weighted(std::true_type{}, hf * PF_PW, t0);
                else weighted(std::false_type{}, hf * PF_PW, t0);
                __syncwarp();
            }
        }
        if (block_or(!ok)) { ok = false; break; }
        if (warp == 0 && t + 1 < tiles) load_v(t + 1);
    }
    if (!ok) {
        // a bounded wait gave up: report it, give copies in flight time to land, write nothing
        if (tid == 0 && p.status) atomicOr(p.status, p.status_wait);
        for (int i = 0; i < 64; i++) __nanosleep(1000);
        block_sync();
        return;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 4);
        const int r = tr + 32 * i;
        if (r >= (int)rows) continue;
        const size_t orow = ((size_t)b * p.heads + h) * p.seq_q + q0 + r;
        const bool any = l[i] > 0.0f;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            float4 t;
            unpair(o[i][2 * j], t.x, t.y);
            unpair(o[i][2 * j + 1], t.z, t.w);
            t = any ? make_float4(t.x / l[i], t.y / l[i], t.z / l[i], t.w / l[i]) : make_float4(0.f, 0.f, 0.f, 0.f);
            *reinterpret_cast<float4*>(p.out + orow * PF_D + 32 * j + 4 * tc) = t;
        }
        if (tc == 0 && p.lse) p.lse[orow] = l[i] > 0.0f ? fmaf(m[i], PF_LN2, logf(l[i])) : -3.402823e+38f;
    }
}

}  // namespace prefill
}  // namespace
}  // namespace luxcuda
