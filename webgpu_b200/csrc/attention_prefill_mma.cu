// attention_prefill_mma.cu -- attention of many query rows per head on the tensor cores, f32 in and out, head size 128.
//
// The f32 FMA pipe (72 TFLOP/s) is not what a prompt has to be bound by: an f32 number split into two f16 parts,
// h = f16(x) and l = f16(x - h), keeps 22 bits and the sign, and  a b = ah bh + (ah bl + al bh)  leaves out only
// al bl <= 2^-22 |a b|.  Three m16n8k16 products replace one f32 product, and mma.sync does 1011 of those multiply-
// adds per clock and SM (measured: 8.1 cycles each per sub-core) where the FMA pipe does 128.
//
// Range.  f16 has five exponent bits, so the operands are scaled by powers of two (exact) first: a row of Q or K by
// its own largest magnitude, a column of V by that of the tile's 64 keys, so that the largest lies in [2^14, 2^15);
// the weights by 2^10.  A part is then a normal f16 down to 2^-28 of the row's (column's) largest magnitude, and
// smaller ones lose at most 2^-39 of it.  The products' scales come off the f32 sums.
//
// Accumulation.  The tensor core sums a step of 16 exactly and cuts the f32 result off (measured: mean loss 3.8e-8,
// otherwise no more than rounding's error).  Every step of 16 columns (scores) or keys (weighted sum) therefore
// starts from zero, small products first, and is added to the running f32 sum by an ordinary rounded
// addition; the mean loss of the output is put back with its division.  Relative error against 64 bits (2-norm, N(0, 1)
// inputs, Llama-3-8B heads; streaming kernel / this one): causal, 150 tokens 1.36e-7 / 1.35e-7, 512 1.64 / 1.50,
// 2048 2.24 / 1.73; unmasked, 700 x 3 3.04 / 2.14, 1448 4.07 / 2.51.  With the fourth product it gains 3 % of that
// for 17 % more time.
//
// Non-finite inputs.  NaN and infinities do not survive the scaling, so a CTA that meets one writes nothing and leaves
// this call's number in a word of the context; lux_attn_prefill_f32, launched behind this kernel, returns at
// once unless it finds that number there, and otherwise does the whole call.
//
// Work.  A CTA of eight warps owns 128 queries of one head and walks 64-key tiles: bulk copies bring a tile as f32,
// all warps convert it (K row by row, V column by column) into hi / lo f16 tiles that ldmatrix reads
// without conflicts, double-buffered; in each sub-core one warp converts the next tile before it works on the
// current one and the other after it, so that conversion runs beside the tensor core.  A warp owns 16 rows from
// the scores to the output; Q's fragments and the output stay in its registers, the weights go from
// accumulator to operand layout without leaving them.  Causal, Llama-3-8B heads, against the streaming kernel:
// 2048 tokens 1684 -> 453 us (76 TFLOP/s of f32 products, 228 of the tensor core's 568 at this instruction), 512
// tokens 153 -> 65, 150 tokens 29.9 -> 22.5; unmasked 1448 tokens 1570 -> 512.  What is left is the tensor pipe (half
// the time) and the softmax, conversion and fragment loads beside it.
#include "common.cuh"
#include "tc_ptx.cuh"

#include <algorithm>

namespace luxcuda {

namespace {
namespace pmma {

using namespace tcptx;

constexpr int D = 128;                    // head size
constexpr int BM = 128;                   // queries per CTA: 16 per warp
constexpr int BN = 64;                    // keys per tile
constexpr int WARPS = 8, THREADS = WARPS * 32;
constexpr int HALF_TILE = BN * D * 2;     // a tile's hi or lo part: 64 rows of 256 bytes, 16-byte chunks ^ (row & 7)
// f32 K and V, then two buffers of {K hi, K lo, V hi, V lo}, then the scales and barriers
constexpr int OFF_FK = 0, OFF_FV = BN * D * 4, OFF_BUF = 2 * BN * D * 4, BUF_BYTES = 4 * HALF_TILE;
constexpr int OFF_KINV = OFF_BUF + 2 * BUF_BYTES;            // [2][64] floats
constexpr int OFF_VINV = OFF_KINV + 2 * BN * 4;              // [2][128] floats
constexpr int OFF_VMAX = OFF_VINV + 2 * D * 4;               // [2][4][128] words: column maxima of 16 keys each
constexpr int OFF_BAR = OFF_VMAX + 2 * 4 * D * 4;            // two mbarriers, abort flag, bad flag
constexpr int SMEM = OFF_BAR + 64 + 128;
constexpr float NEG = -3.0e38f, LN2 = 0.6931471805599453f;
constexpr float P_SCALE = 1024.0f;        // weights are split times 2^10 (taken off with V's scales)
constexpr double UNBIAS = 3.8e-8;         // mean relative loss of one cut-off f32 sum (measured: 3.7e-8 .. 3.85e-8)
constexpr float RAISE = 4.0f;             // the running maximum is raised when a score passes it by more: weights below 2^14

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldm4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldm4t(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// two values as (hi, hi) and (lo, lo) pairs, the first in the low half
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
__device__ __forceinline__ uint32_t abs_bits(float x) { return __float_as_uint(x) & 0x7fffffffu; }
// largest magnitude (as bits; an infinity or a NaN is at least 0x7f800000) -> the power of two that brings it into
// [2^14, 2^15), and its reciprocal; anything below 2^-76 counts as that (the reciprocal less P_SCALE stays a normal number)
__device__ __forceinline__ void scale_of(uint32_t max_bits, float& s, float& inv) {
    const int e = min(max((int)(max_bits >> 23), 51), 254);      // biased exponent
    s = __uint_as_float((uint32_t)(127 + 14 + 127 - e) << 23);   // 2^(14 - (e - 127))
    inv = __uint_as_float((uint32_t)(e - 14) << 23);
}

__global__ void __launch_bounds__(THREADS, 1) lux_attn_prefill_mma_f32(const PrefillArgs p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
    const uint32_t sb = smem_u32(smem);
    const uint32_t bar_k = sb + OFF_BAR, bar_v = bar_k + 8u;
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + OFF_BAR + 16);
    volatile uint32_t* bad_flag = abort_flag + 1;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;

    pdl_launch_dependents();
    // blocks of late queries see the most keys under a causal mask: they come first, so that the last
    // wave is made of short ones.  Neighbouring CTAs are heads of one KV head and share its tiles in L2.
    const uint32_t bh = p.batch * p.heads;
    const uint32_t qb = p.q_blocks - 1u - blockIdx.x / bh, rest = blockIdx.x % bh;
    const uint32_t h = rest % p.heads, b = rest / p.heads, kvh = h / p.group;
    const uint32_t q0 = qb * BM, rows = min((uint32_t)BM, p.seq_q - q0);
    auto row_len = [&](uint32_t qi) { return p.causal ? min(p.causal_base + qi + 1u, p.kv_len) : p.kv_len; };
    const uint32_t lmax = row_len(q0 + rows - 1u);
    const uint32_t tiles = (lmax + BN - 1u) / BN;
    const float* kbase = p.k + ((size_t)b * p.kv_heads + kvh) * p.kv_stride * D;
    const float* vbase = p.v + ((size_t)b * p.kv_heads + kvh) * p.kv_stride * D;

    auto load_tile = [&](uint32_t t) {
        const uint32_t t0 = t * BN, bytes = min((uint32_t)BN, lmax - t0) * D * 4u;
        mbar_expect_tx(bar_k, bytes);
        bulk_g2s(sb + OFF_FK, kbase + (size_t)t0 * D, bytes, bar_k);
        mbar_expect_tx(bar_v, bytes);
        bulk_g2s(sb + OFF_FV, vbase + (size_t)t0 * D, bytes, bar_v);
    };
    if (tid == 0) {
        mbar_init(bar_k, 1u);
        mbar_init(bar_v, 1u);
        *abort_flag = 0u;
        *bad_flag = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();                              // the flags are clear before a warp may raise one over its rows of Q
    pdl_wait();
    if (tid == 0 && tiles) load_tile(0);

    // ---- Q: this lane's fragments of rows g and g + 8 of the warp's 16, scaled and split ------------------
    uint32_t qh[8][4], ql[8][4];
    float qinv[2], m[2], l[2];
    uint32_t len[2];
    {
        float2 x[2][16];                              // row half r: columns 8 j + 2 t4 and the next
        uint32_t mx[2] = {0u, 0u};
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const uint32_t row = (uint32_t)(warp * 16 + g + 8 * r);
            len[r] = row < rows ? row_len(q0 + row) : 0u;            // a padding row sees nothing and is not written
            const float* src = p.q + (((size_t)b * p.heads + h) * p.seq_q + q0 + min(row, rows - 1u)) * D + 2 * t4;
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const float2 v = __ldg(reinterpret_cast<const float2*>(src + 8 * j));
                x[r][j] = make_float2(v.x * p.qscale, v.y * p.qscale);
                mx[r] = max(mx[r], max(abs_bits(x[r][j].x), abs_bits(x[r][j].y)));
            }
            mx[r] = max(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
            mx[r] = max(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
            float s;
            scale_of(mx[r], s, qinv[r]);
            if (mx[r] >= 0x7f800000u) *bad_flag = 1u;
#pragma unroll
            for (int j = 0; j < 16; j++) split2(x[r][j].x * s, x[r][j].y * s, qh[j >> 1][2 * (j & 1) + r], ql[j >> 1][2 * (j & 1) + r]);
            m[r] = NEG;
            l[r] = 0.0f;
        }
    }
    float o[16][4];                                   // columns 8 n + 2 t4 (+ 1) of rows g (0, 1) and g + 8 (2, 3)
#pragma unroll
    for (int n = 0; n < 16; n++)
#pragma unroll
        for (int e = 0; e < 4; e++) o[n][e] = 0.0f;

    // ---- tile t, f32 -> hi / lo f16 in buffer t & 1 -------------------------------------------------
    // The column maxima of V come in two steps: vmax() leaves those of 16 keys per thread, the barrier that ends
    // a round publishes them, convert() uses them.
    auto vmax = [&](uint32_t t) {
        const uint32_t nk = min((uint32_t)BN, lmax - t * BN);
        const int c2 = tid & 63, kg = tid >> 6;       // columns 2 c2, 2 c2 + 1; keys 16 kg ..
        const float2* src = reinterpret_cast<const float2*>(smem + OFF_FV) + c2;
        uint32_t m0 = 0u, m1 = 0u;
#pragma unroll
        for (int k = 0; k < 16; k++)
            if ((uint32_t)(16 * kg + k) < nk) {
                const float2 v = src[(16 * kg + k) * (D / 2)];
                m0 = max(m0, abs_bits(v.x));
                m1 = max(m1, abs_bits(v.y));
            }
        *reinterpret_cast<uint2*>(smem + OFF_VMAX + ((t & 1u) * 4 + kg) * (D * 4) + c2 * 8) = make_uint2(m0, m1);
        if (max(m0, m1) >= 0x7f800000u) *bad_flag = 1u;
    };
    auto convert = [&](uint32_t t) {
        const uint32_t nk = min((uint32_t)BN, lmax - t * BN);
        unsigned char* buf = smem + OFF_BUF + (t & 1u) * BUF_BYTES;
        float* kinv = reinterpret_cast<float*>(smem + OFF_KINV) + (t & 1u) * BN;
        // K: rows 8 warp .. + 7, a lane holds four columns
#pragma unroll 4
        for (int i = 0; i < 8; i++) {
            const int key = warp * 8 + i;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if ((uint32_t)key < nk) v = *(reinterpret_cast<const float4*>(smem + OFF_FK + key * (D * 4)) + lane);
            const uint32_t mx = __reduce_max_sync(0xffffffffu, max(max(abs_bits(v.x), abs_bits(v.y)), max(abs_bits(v.z), abs_bits(v.w))));
            float s, inv;
            scale_of(mx, s, inv);
            if (mx >= 0x7f800000u) *bad_flag = 1u;
            uint2 hi, lo;
            split2(v.x * s, v.y * s, hi.x, lo.x);
            split2(v.z * s, v.w * s, hi.y, lo.y);
            const int at = key * 256 + (((lane >> 1) ^ (key & 7)) << 4) + (lane & 1) * 8;
            *reinterpret_cast<uint2*>(buf + at) = hi;
            *reinterpret_cast<uint2*>(buf + HALF_TILE + at) = lo;
            if (lane == 0) kinv[key] = inv;
        }
        // V: columns 2 c2, 2 c2 + 1 of keys 16 kg ..
        const int c2 = tid & 63, kg = tid >> 6;
        uint2 mm = make_uint2(0u, 0u);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint2 w = *reinterpret_cast<const uint2*>(smem + OFF_VMAX + ((t & 1u) * 4 + q) * (D * 4) + c2 * 8);
            mm = make_uint2(max(mm.x, w.x), max(mm.y, w.y));
        }
        float s0, s1, i0, i1;
        scale_of(mm.x, s0, i0);
        scale_of(mm.y, s1, i1);
        if (kg == 0) *reinterpret_cast<float2*>(smem + OFF_VINV + (t & 1u) * (D * 4) + c2 * 8) = make_float2(i0 * (1.0f / P_SCALE), i1 * (1.0f / P_SCALE));
        const float2* src = reinterpret_cast<const float2*>(smem + OFF_FV) + c2;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const int key = 16 * kg + k;
            float2 v = make_float2(0.f, 0.f);
            if ((uint32_t)key < nk) v = src[key * (D / 2)];
            uint32_t hi, lo;
            split2(v.x * s0, v.y * s1, hi, lo);
            const int at = 2 * HALF_TILE + key * 256 + (((c2 >> 2) ^ (key & 7)) << 4) + (c2 & 3) * 4;
            *reinterpret_cast<uint32_t*>(buf + at) = hi;
            *reinterpret_cast<uint32_t*>(buf + HALF_TILE + at) = lo;
        }
    };

    // ---- one tile's work of a warp ---------------------------------------------------------------
    const uint32_t last_len = row_len(q0 + min((uint32_t)(warp * 16 + 15), rows - 1u));
    const uint32_t first_len = row_len(q0 + min((uint32_t)(warp * 16), rows - 1u));
    const bool live = (uint32_t)(warp * 16) < rows;
    auto work = [&](uint32_t t) {
        const uint32_t t0 = t * BN;
        if (!live || t0 >= last_len) return;            // no row of the warp sees the tile
        const uint32_t buf = sb + OFF_BUF + (t & 1u) * BUF_BYTES;
        // scores: B fragments of 8 keys x 32 columns per ldmatrix (rows = keys, four 16-byte chunks)
        float s[8][4];
        const uint32_t krow = (uint32_t)(lane & 7) * 256u, kchunk = (uint32_t)(lane >> 3), kx = (uint32_t)(lane & 7);
#pragma unroll
        for (int n = 0; n < 8; n++) {
#pragma unroll
            for (int e = 0; e < 4; e++) s[n][e] = 0.0f;
#pragma unroll
            for (int d = 0; d < 4; d++) {
                uint32_t kh[4], kl[4];
                const uint32_t at = buf + (uint32_t)(n * 8 * 256) + krow + (((kchunk + 4u * d) ^ kx) << 4);
                ldm4(at, kh);
                ldm4(at + HALF_TILE, kl);
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    float c[4] = {0.f, 0.f, 0.f, 0.f};
                    mma(c, ql[2 * d + k], kh[2 * k], kh[2 * k + 1]);
                    mma(c, qh[2 * d + k], kl[2 * k], kl[2 * k + 1]);
                    mma(c, qh[2 * d + k], kh[2 * k], kh[2 * k + 1]);
#pragma unroll
                    for (int e = 0; e < 4; e++) s[n][e] += c[e];
                }
            }
        }
        const float* kinv = reinterpret_cast<const float*>(smem + OFF_KINV) + (t & 1u) * BN + 2 * t4;
        const bool edge = t0 + BN > first_len;
        float mt[2] = {NEG, NEG};
#pragma unroll
        for (int n = 0; n < 8; n++) {
            const float2 ki = *reinterpret_cast<const float2*>(kinv + 8 * n);
#pragma unroll
            for (int e = 0; e < 4; e++) {
                s[n][e] = s[n][e] * qinv[e >> 1] * (e & 1 ? ki.y : ki.x);
                if (edge && t0 + 8 * n + 2 * t4 + (e & 1) >= len[e >> 1]) s[n][e] = -__int_as_float(0x7f800000);
                mt[e >> 1] = fmaxf(mt[e >> 1], s[n][e]);
            }
        }
        bool up = false;
#pragma unroll
        for (int r = 0; r < 2; r++) {
            mt[r] = fmaxf(mt[r], __shfl_xor_sync(0xffffffffu, mt[r], 1));
            mt[r] = fmaxf(mt[r], __shfl_xor_sync(0xffffffffu, mt[r], 2));
            up |= mt[r] > m[r] + RAISE;
        }
        if (__any_sync(0xffffffffu, up)) {
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const float mn = fmaxf(m[r], mt[r]), alpha = ex2(m[r] - mn);
                m[r] = mn;
                l[r] *= alpha;
#pragma unroll
                for (int n = 0; n < 16; n++) {
                    o[n][2 * r] *= alpha;
                    o[n][2 * r + 1] *= alpha;
                }
            }
        }
        uint32_t ph[4][4], pl[4][4];
        float sum[2] = {0.f, 0.f};
#pragma unroll
        for (int n = 0; n < 8; n++) {
#pragma unroll
            for (int e = 0; e < 4; e++) s[n][e] = ex2(s[n][e] - m[e >> 1]);
            sum[0] += s[n][0] + s[n][1];
            sum[1] += s[n][2] + s[n][3];
            split2(s[n][0] * P_SCALE, s[n][1] * P_SCALE, ph[n >> 1][2 * (n & 1)], pl[n >> 1][2 * (n & 1)]);
            split2(s[n][2] * P_SCALE, s[n][3] * P_SCALE, ph[n >> 1][2 * (n & 1) + 1], pl[n >> 1][2 * (n & 1) + 1]);
        }
        l[0] += sum[0];
        l[1] += sum[1];
        // weighted sum: B fragments of 16 keys x 16 columns per transposing ldmatrix
        const float* vinv = reinterpret_cast<const float*>(smem + OFF_VINV) + (t & 1u) * D + 2 * t4;
        const uint32_t vkey = (uint32_t)(lane & 15), vchunk = (uint32_t)(lane >> 4);
        const uint32_t vbase_s = buf + 2 * HALF_TILE + vkey * 256u, vx = vkey & 7u;
#pragma unroll
        for (int kc = 0; kc < 2; kc++) {               // 32 keys
            if (t0 + 32 * kc >= last_len) break;
#pragma unroll
            for (int n2 = 0; n2 < 8; n2++) {           // 16 columns
                uint32_t vh[2][4], vl[2][4];
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const uint32_t at = vbase_s + (uint32_t)((32 * kc + 16 * k) * 256) + (((vchunk + 2u * n2) ^ vx) << 4);
                    ldm4t(at, vh[k]);
                    ldm4t(at + HALF_TILE, vl[k]);
                }
#pragma unroll
                for (int c2 = 0; c2 < 2; c2++) {
                    const int n = 2 * n2 + c2;
                    const float2 vi = *reinterpret_cast<const float2*>(vinv + 8 * n);
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        float c[4] = {0.f, 0.f, 0.f, 0.f};
                        mma(c, pl[2 * kc + k], vh[k][2 * c2], vh[k][2 * c2 + 1]);
                        mma(c, ph[2 * kc + k], vl[k][2 * c2], vl[k][2 * c2 + 1]);
                        mma(c, ph[2 * kc + k], vh[k][2 * c2], vh[k][2 * c2 + 1]);
                        o[n][0] = fmaf(c[0], vi.x, o[n][0]);
                        o[n][1] = fmaf(c[1], vi.y, o[n][1]);
                        o[n][2] = fmaf(c[2], vi.x, o[n][2]);
                        o[n][3] = fmaf(c[3], vi.y, o[n][3]);
                    }
                }
            }
        }
    };

    // ---- rounds: in round t the warps convert tile t + 1 and work on tile t -----------------------------
    __syncthreads();
    bool ok = true;
    if (tiles) {
        ok = warp_wait(bar_k, 0u, abort_flag, lane) && warp_wait(bar_v, 0u, abort_flag, lane);
        if (ok) vmax(0);
        if (!__syncthreads_or(!ok)) {
            convert(0);
            ok = !__syncthreads_or(*bad_flag != 0u);
            if (ok && tid == 0 && tiles > 1) load_tile(1);
            for (uint32_t t = 0; ok && t < tiles; t++) {
                const bool more = t + 1 < tiles;
                bool landed = true;
                if (more) {
                    landed = warp_wait(bar_k, (t + 1) & 1u, abort_flag, lane) && warp_wait(bar_v, (t + 1) & 1u, abort_flag, lane);
                    if (landed) vmax(t + 1);
                }
                if (__syncthreads_or(!landed)) { ok = false; break; }
                if (more && warp < WARPS / 2) convert(t + 1);
                work(t);
                if (more && warp >= WARPS / 2) convert(t + 1);
                if (__syncthreads_or(*bad_flag != 0u)) { ok = false; break; }
                if (tid == 0 && t + 2 < tiles) load_tile(t + 2);
            }
        } else {
            ok = false;
        }
    } else {
        ok = !__syncthreads_or(*bad_flag != 0u);
    }
    if (!ok) {
        // non-finite inputs: the kernel behind this one does the call; or a bounded wait gave up: report it, and give
        // copies in flight time to land.  Nothing is written.  (No copy is in flight when a round ends on bad_flag.)
        if (*abort_flag) {
            if (tid == 0 && p.status) atomicOr(p.status, p.status_wait);
            for (int i = 0; i < 64; i++) __nanosleep(1000);
            __syncthreads();
        } else if (tid == 0) {
            atomicExch(p.redo, p.call);
        }
        return;
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
        const uint32_t row = (uint32_t)(warp * 16 + g + 8 * r);
        if (row >= rows) continue;
        const size_t orow = ((size_t)b * p.heads + h) * p.seq_q + q0 + row;
        const bool any = l[r] > 0.0f;                  // a row without keys is zero
        // the tensor core cuts its f32 results off instead of rounding them: the sums are short by UNBIAS on average
        const double inv = any ? (1.0 + UNBIAS) / (double)l[r] : 0.0;
#pragma unroll
        for (int n = 0; n < 16; n++)
            *reinterpret_cast<float2*>(p.out + orow * D + 8 * n + 2 * t4) =
                any ? make_float2((float)(o[n][2 * r] * inv), (float)(o[n][2 * r + 1] * inv)) : make_float2(0.f, 0.f);
        if (t4 == 0 && p.lse) p.lse[orow] = any ? fmaf(m[r], LN2, logf(l[r])) : -3.402823e+38f;
    }
}

}  // namespace pmma
}  // namespace

LuxBackendError launch_attn_prefill_mma(Context* ctx, PrefillArgs p) {
    using namespace pmma;
    static std::atomic<bool> configured[64];
    const int dev = ctx->device & 63;
    if (!configured[dev].load(std::memory_order_relaxed)) {
        cudaError_t e = cudaFuncSetAttribute(lux_attn_prefill_mma_f32, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) return map_cuda(e, "lux_attn_prefill_mma_f32");
        configured[dev].store(true, std::memory_order_relaxed);
    }
    p.q_blocks = (p.seq_q + pmma::BM - 1) / pmma::BM;
    cudaError_t e = launch_pdl(g_tune.pdl != 2, lux_attn_prefill_mma_f32, dim3(p.q_blocks * p.heads * p.batch), dim3(THREADS), (size_t)SMEM, ctx->stream, 1, p);
    if (e != cudaSuccess) return map_cuda(e, "lux_attn_prefill_mma_f32");
    count_launch("lux_attn_prefill_mma_f32");
    return LUX_BACKEND_OK;
}

const void* kernel_addr_attn_prefill_mma_f32() { return (const void*)pmma::lux_attn_prefill_mma_f32; }

}  // namespace luxcuda
