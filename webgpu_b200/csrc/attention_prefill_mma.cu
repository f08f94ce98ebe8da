// attention_prefill_mma.cu -- attention of many query rows per head on the tensor cores, f32 in and out, head size 128.
//
// The f32 FMA pipe (72 TFLOP/s) is not what a prompt has to be bound by.  An f32 number is the exact sum of three bf16
// parts, h = bf16(x), m = bf16(x - h), l = x - h - m, and
//     a b = ah bh + (ah bm + am bh) + (am bm + ah bl + al bh)
// leaves out only am bl + al bm + al bl <= 2^-24 |a b|, what rounding the product to f32 would cost.  Six m16n8k16
// products replace one f32 product, and mma.sync does 1011 of those multiply-adds per clock and SM (measured: 8.1 cycles
// each per sub-core) where the FMA pipe does 128.
//
// Range.  bf16 has f32's exponents, so a part depends on its own element alone: no scale is shared along a row, a
// column or a tile, and a masked key weighs exactly nothing however large its values.  A part below 2^-126 may be
// lost.  Weights are split times 2^30 (a weight is 2^-126 at least, or 0) and so keep their 24 bits; in a score
// 2^-126 x 2^60 x 128 is nothing; and V can lose 2^-126 of an output, which matters to outputs below 2^-100 alone:
// if V had non-zero values below 2^-100 and such an output comes out, the block is done on the f32 pipe.
// So is one that meets a magnitude of 2^60 or more (after Q's scale), an infinity or a NaN: with all below 2^60
// no score, no sum (2^120 x 128; 2^(8 + 30 + 60) a key) and no bf16 rounding overflows.
//
// Accumulation.  The tensor core sums a step of 16 exactly and cuts the f32 result off (measured: mean loss 3.8e-8 of
// it, otherwise no more than rounding's error).  Every step's h h products, of 16 bits each, therefore start from zero
// and are added to the running f32 sum by an ordinary rounded addition; the other products, 2^-8 of these and less,
// run in a chain of their own, where the cut is 2^-8 as large, and are added once per tile.  Relative error against
// 64 bits (2-norm, N(0, 1) inputs, Llama-3-8B heads; streaming kernel / this one): causal, 150 tokens 1.34e-7 /
// 1.04e-7, 512 1.65 / 1.22, 2048 2.25 / 1.42; unmasked, 700 x 3 3.06 / 1.76, 1448 4.06 / 2.03.
//
// Out-of-range inputs.  A CTA that meets one starts its block over on the f32 pipe (attention_prefill_f32.cuh); it has written
// nothing by then, so this holds with out == q, and no other block, call or replay of a captured one takes part.
//
// Work.  A CTA of eight warps owns 128 queries of one head and walks 32-key tiles (three parts of 64 would not fit
// shared memory twice): bulk copies bring a tile as f32, two tiles ahead; all warps split it into three bf16
// tiles each of K and V that ldmatrix reads without conflicts, double-buffered; in each sub-core one warp splits the next tile
// before it works on the current one and the other after it, so that the splitting runs beside the tensor core.  A warp
// owns 16 rows from the scores to the output; Q's fragments and the output stay in its registers, the weights go from
// accumulator to operand layout without leaving them.  Causal, Llama-3-8B heads, against the streaming kernel:
// 2048 tokens 1679 -> 673 us (51 TFLOP/s of f32 products, 307 of the tensor core's 568 at this instruction), 512
// tokens 152 -> 93, 150 tokens 29.5 -> 28.3; unmasked 1448 tokens 1567 -> 774.  What is left is the tensor pipe (more
// than half the time) and the softmax, splitting and fragment loads beside it.
#include "attention_prefill_f32.cuh"

namespace luxcuda {

namespace {
namespace pmma {

using namespace tcptx;

constexpr int D = 128;                    // head size
constexpr int BM = 128;                   // queries per CTA: 16 per warp
constexpr int BN = 32;                    // keys per tile
constexpr int WARPS = 8, THREADS = WARPS * 32;
constexpr int F32_TILE = BN * D * 4;      // K or V of a tile as it arrives
constexpr int PART = BN * D * 2;          // one part of it: 32 rows of 256 bytes, 16-byte chunks ^ (row & 7)
// two slots of {K, V} in f32, two buffers of {K h, m, l, V h, m, l}, two mbarriers, abort flag, bad flag, tiny flag
constexpr int OFF_F32 = 0, SLOT = 2 * F32_TILE, OFF_BUF = 2 * SLOT, BUF_BYTES = 6 * PART;
constexpr int OFF_BAR = OFF_BUF + 2 * BUF_BYTES;
constexpr int SMEM = OFF_BAR + 64 + 128;
constexpr float NEG = -3.0e38f, LN2 = 0.6931471805599453f;
constexpr float RAISE = 8.0f;             // the running maximum is raised when a score passes it by more: weights below 2^8
constexpr float P_SCALE = 0x1p30f;        // of the weights before they are split
constexpr uint32_t TOO_LARGE = (127u + 60u) << 23;           // |x| >= 2^60, infinity or NaN, as bits
constexpr uint32_t TOO_SMALL = (127u - 100u) << 23;          // 0 < |v| < 2^-100

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldm4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldm4t(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// two values as pairs of their parts, the first in the low half; the two differences are exact
__device__ __forceinline__ void split3(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    auto pack = [](float x, float y) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
        return *reinterpret_cast<const uint32_t*>(&v);
    };
    h = pack(a, b);
    a -= __uint_as_float(h << 16);
    b -= __uint_as_float(h & 0xffff0000u);
    m = pack(a, b);
    l = pack(a - __uint_as_float(m << 16), b - __uint_as_float(m & 0xffff0000u));
}
__device__ __forceinline__ uint32_t abs_bits(float x) { return __float_as_uint(x) & 0x7fffffffu; }

__global__ void __launch_bounds__(THREADS, 1) lux_attn_prefill_mma_f32(const PrefillArgs p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
    const uint32_t sb = smem_u32(smem);
    const uint32_t bars = sb + OFF_BAR;           // one per slot
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + OFF_BAR + 16);
    volatile uint32_t* bad_flag = abort_flag + 1;
    volatile uint32_t* tiny_flag = abort_flag + 2;
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

    auto load_tile = [&](uint32_t t) {            // tile t goes to slot t & 1
        const uint32_t t0 = t * BN, bytes = min((uint32_t)BN, lmax - t0) * D * 4u, bar = bars + 8u * (t & 1u);
        const uint32_t dst = sb + OFF_F32 + (t & 1u) * SLOT;
        mbar_expect_tx(bar, 2u * bytes);
        bulk_g2s(dst, kbase + (size_t)t0 * D, bytes, bar);
        bulk_g2s(dst + F32_TILE, vbase + (size_t)t0 * D, bytes, bar);
    };
    if (tid == 0) {
        mbar_init(bars, 1u);
        mbar_init(bars + 8u, 1u);
        *abort_flag = 0u;
        *bad_flag = 0u;
        *tiny_flag = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();                              // the flags are clear before a warp may raise one over its rows of Q
    pdl_wait();
    if (tid == 0) {
        if (tiles > 0) load_tile(0);
        if (tiles > 1) load_tile(1);
    }
    auto landed = [&](uint32_t t) { return warp_wait(bars + 8u * (t & 1u), (t >> 1) & 1u, abort_flag, lane); };

    // ---- Q: this lane's fragments of rows g and g + 8 of the warp's 16, scaled and split ------------------
    uint32_t qp[3][8][4];
    float m[2], l[2];
    uint32_t len[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {                     // row half r: columns 8 j + 2 t4 and the next
        const uint32_t row = (uint32_t)(warp * 16 + g + 8 * r);
        len[r] = row < rows ? row_len(q0 + row) : 0u;                // a padding row sees nothing and is not written
        const float* src = p.q + (((size_t)b * p.heads + h) * p.seq_q + q0 + min(row, rows - 1u)) * D + 2 * t4;
        float2 x[16];
        uint32_t top = 0u;
#pragma unroll
        for (int j = 0; j < 16; j++) x[j] = __ldg(reinterpret_cast<const float2*>(src + 8 * j));
#pragma unroll
        for (int j = 0; j < 16; j++) {
            x[j] = make_float2(x[j].x * p.qscale, x[j].y * p.qscale);
            top = max(top, max(abs_bits(x[j].x), abs_bits(x[j].y)));
            const int f = j >> 1, e = 2 * (j & 1) + r;
            split3(x[j].x, x[j].y, qp[0][f][e], qp[1][f][e], qp[2][f][e]);
        }
        if (top >= TOO_LARGE) *bad_flag = 1u;
        m[r] = NEG;
        l[r] = 0.0f;
    }
    float o[16][4];                                   // columns 8 n + 2 t4 (+ 1) of rows g (0, 1) and g + 8 (2, 3)
#pragma unroll
    for (int n = 0; n < 16; n++)
#pragma unroll
        for (int e = 0; e < 4; e++) o[n][e] = 0.0f;

    // ---- tile t, f32 -> parts in buffer t & 1: warps 0..3 take eight rows of K each, 4..7 of V -----------------
    auto convert = [&](uint32_t t) {
        const uint32_t nk = min((uint32_t)BN, lmax - t * BN);
        const unsigned char* src = smem + OFF_F32 + (t & 1u) * SLOT + warp * 8 * (D * 4) + lane * 16;
        unsigned char* buf = smem + OFF_BUF + (t & 1u) * BUF_BYTES + (warp >> 2) * (3 * PART);
        uint32_t top = 0u, low = 0xffffffffu;         // largest magnitude; smallest non-zero one, less 1
#pragma unroll 4
        for (int i = 0; i < 8; i++) {
            const int key = (warp & 3) * 8 + i;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if ((uint32_t)key < nk) v = *reinterpret_cast<const float4*>(src + i * (D * 4));
            const uint32_t b0 = abs_bits(v.x), b1 = abs_bits(v.y), b2 = abs_bits(v.z), b3 = abs_bits(v.w);
            top = max(top, max(max(b0, b1), max(b2, b3)));
            low = min(low, min(min(b0 - 1u, b1 - 1u), min(b2 - 1u, b3 - 1u)));
            uint2 w[3];
            split3(v.x, v.y, w[0].x, w[1].x, w[2].x);
            split3(v.z, v.w, w[0].y, w[1].y, w[2].y);
            const int at = key * 256 + (((lane >> 1) ^ (key & 7)) << 4) + (lane & 1) * 8;
#pragma unroll
            for (int c = 0; c < 3; c++) *reinterpret_cast<uint2*>(buf + c * PART + at) = w[c];
        }
        if (top >= TOO_LARGE) *bad_flag = 1u;
        if (low < TOO_SMALL - 1u && warp >= WARPS / 2) *tiny_flag = 1u;
    };
    // c += a b without its h h part, for two independent pairs at once (their chains of five are interleaved)
    auto mma_rest = [&](float (&c0)[4], float (&c1)[4], const uint32_t (&ah)[4], const uint32_t (&am)[4], const uint32_t (&al)[4],
                        const uint32_t (&b0)[3][2], const uint32_t (&b1)[3][2]) {
        mma(c0, al, b0[0][0], b0[0][1]);
        mma(c1, al, b1[0][0], b1[0][1]);
        mma(c0, ah, b0[2][0], b0[2][1]);
        mma(c1, ah, b1[2][0], b1[2][1]);
        mma(c0, am, b0[1][0], b0[1][1]);
        mma(c1, am, b1[1][0], b1[1][1]);
        mma(c0, am, b0[0][0], b0[0][1]);
        mma(c1, am, b1[0][0], b1[0][1]);
        mma(c0, ah, b0[1][0], b0[1][1]);
        mma(c1, ah, b1[1][0], b1[1][1]);
    };

    // ---- one tile's work of a warp ---------------------------------------------------------------
    const uint32_t last_len = row_len(q0 + min((uint32_t)(warp * 16 + 15), rows - 1u));
    const uint32_t first_len = row_len(q0 + min((uint32_t)(warp * 16), rows - 1u));
    const bool live = (uint32_t)(warp * 16) < rows;
    auto work = [&](uint32_t t) {
        const uint32_t t0 = t * BN;
        if (!live || t0 >= last_len) return;            // no row of the warp sees the tile
        const uint32_t buf = sb + OFF_BUF + (t & 1u) * BUF_BYTES;
        // scores: B fragments of 8 keys x 32 columns per ldmatrix (rows = keys, four 16-byte chunks), two groups of
        // 8 keys at a time
        float s[4][4];
        const uint32_t krow = buf + (uint32_t)(lane & 7) * 256u, kchunk = (uint32_t)(lane >> 3), kx = (uint32_t)(lane & 7);
#pragma unroll
        for (int n = 0; n < 4; n += 2) {
            float rest[2][4];
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int e = 0; e < 4; e++) s[n + i][e] = rest[i][e] = 0.0f;
#pragma unroll
            for (int d = 0; d < 4; d++) {
                uint32_t kf[2][3][4];
#pragma unroll
                for (int i = 0; i < 2; i++)
#pragma unroll
                    for (int c = 0; c < 3; c++) ldm4(krow + (uint32_t)(c * PART + (n + i) * 8 * 256) + (((kchunk + 4u * d) ^ kx) << 4), kf[i][c]);
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const int f = 2 * d + k;
                    float c[2][4] = {};
                    uint32_t bf[2][3][2];
#pragma unroll
                    for (int i = 0; i < 2; i++) {
#pragma unroll
                        for (int part = 0; part < 3; part++) {
                            bf[i][part][0] = kf[i][part][2 * k];
                            bf[i][part][1] = kf[i][part][2 * k + 1];
                        }
                        mma(c[i], qp[0][f], bf[i][0][0], bf[i][0][1]);
                    }
                    mma_rest(rest[0], rest[1], qp[0][f], qp[1][f], qp[2][f], bf[0], bf[1]);
#pragma unroll
                    for (int i = 0; i < 2; i++)
#pragma unroll
                        for (int e = 0; e < 4; e++) s[n + i][e] += c[i][e];
                }
            }
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int e = 0; e < 4; e++) s[n + i][e] += rest[i][e];
        }
        const bool edge = t0 + BN > first_len;
        float mt[2] = {NEG, NEG};
#pragma unroll
        for (int n = 0; n < 4; n++) {
#pragma unroll
            for (int e = 0; e < 4; e++) {
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
        uint32_t wp[3][2][4];                          // the weights' parts as A fragments of 16 keys
        float sum[2] = {0.f, 0.f};
#pragma unroll
        for (int n = 0; n < 4; n++) {
#pragma unroll
            for (int e = 0; e < 4; e++) s[n][e] = ex2(s[n][e] - m[e >> 1]);
            sum[0] += s[n][0] + s[n][1];
            sum[1] += s[n][2] + s[n][3];
            const int f = n >> 1, e = 2 * (n & 1);
            split3(s[n][0] * P_SCALE, s[n][1] * P_SCALE, wp[0][f][e], wp[1][f][e], wp[2][f][e]);
            split3(s[n][2] * P_SCALE, s[n][3] * P_SCALE, wp[0][f][e + 1], wp[1][f][e + 1], wp[2][f][e + 1]);
        }
        l[0] += sum[0];
        l[1] += sum[1];
        // weighted sum: B fragments of 16 keys x 16 columns per transposing ldmatrix
        const uint32_t vrow = buf + (uint32_t)(3 * PART) + (uint32_t)(lane & 15) * 256u, vchunk = (uint32_t)(lane >> 4), vx = (uint32_t)(lane & 7);
#pragma unroll
        for (int n2 = 0; n2 < 8; n2++) {               // 16 columns
            float c[2][2][4] = {}, rest[2][4] = {};
#pragma unroll
            for (int k = 0; k < 2; k++) {              // 16 keys
                uint32_t vf[3][4], bf[2][3][2];
#pragma unroll
                for (int part = 0; part < 3; part++) ldm4t(vrow + (uint32_t)(part * PART + 16 * k * 256) + (((vchunk + 2u * n2) ^ vx) << 4), vf[part]);
#pragma unroll
                for (int i = 0; i < 2; i++) {
#pragma unroll
                    for (int part = 0; part < 3; part++) {
                        bf[i][part][0] = vf[part][2 * i];
                        bf[i][part][1] = vf[part][2 * i + 1];
                    }
                    mma(c[i][k], wp[0][k], bf[i][0][0], bf[i][0][1]);
                }
                mma_rest(rest[0], rest[1], wp[0][k], wp[1][k], wp[2][k], bf[0], bf[1]);
            }
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int e = 0; e < 4; e++) o[2 * n2 + i][e] += c[i][0][e] + (c[i][1][e] + rest[i][e]);
        }
    };

    // ---- rounds: in round t the warps split tile t + 1 and work on tile t, and tile t + 2 is on its way ---------
    bool ok = true;
    uint32_t asked = min(2u, tiles);                   // tiles requested so far
    if (tiles) {
        bool here = landed(0);
        if (here) convert(0);
        ok = !__syncthreads_or(!here || *bad_flag != 0u);
        for (uint32_t t = 0; ok && t < tiles; t++) {
            const bool more = t + 1 < tiles;
            if (t + 2 < tiles) {                       // slot t & 1 was split in the last round
                if (tid == 0) load_tile(t + 2);
                asked = t + 3;
            }
            here = true;
            if (more && warp < WARPS / 2 && (here = landed(t + 1))) convert(t + 1);
            work(t);
            if (more && warp >= WARPS / 2 && (here = landed(t + 1))) convert(t + 1);
            if (__syncthreads_or(!here || *bad_flag != 0u)) ok = false;
        }
    } else {
        ok = !__syncthreads_or(*bad_flag != 0u);
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
    }
    if (ok && *tiny_flag) {                            // the same for all: last written before the last round's barrier
        bool low = false;
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int n = 0; n < 16; n++) {
                const float least = l[r] * (P_SCALE * 0x1p-100f);
                low |= fabsf(o[n][2 * r]) < least || fabsf(o[n][2 * r + 1]) < least;
            }
        ok = !__syncthreads_or(low);
    }
    if (!ok) {
        // values out of range: the block starts over on the f32 pipe; or a bounded wait gave up: report it, and give
        // copies in flight time to land.  Nothing has been written.
        for (uint32_t t = asked > 2u ? asked - 2u : 0u; t < asked; t++) landed(t);
        __syncthreads();
        if (*abort_flag) {
            if (tid == 0 && p.status) atomicOr(p.status, p.status_wait);
            for (int i = 0; i < 64; i++) __nanosleep(1000);
            __syncthreads();
        } else {
            prefill::attend_f32(p, smem, qb, h, b);
        }
        return;
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const uint32_t row = (uint32_t)(warp * 16 + g + 8 * r);
        if (row >= rows) continue;
        const size_t orow = ((size_t)b * p.heads + h) * p.seq_q + q0 + row;
        const bool any = l[r] > 0.0f;                  // a row without keys is zero
#pragma unroll
        for (int n = 0; n < 16; n++)
            *reinterpret_cast<float2*>(p.out + orow * D + 8 * n + 2 * t4) =
                any ? make_float2(o[n][2 * r] / l[r] * (1.0f / P_SCALE), o[n][2 * r + 1] / l[r] * (1.0f / P_SCALE)) : make_float2(0.f, 0.f);
        if (t4 == 0 && p.lse) p.lse[orow] = any ? fmaf(m[r], LN2, logf(l[r])) : -3.402823e+38f;
    }
}

// Every block on the f32 pipe.
__global__ void __launch_bounds__(prefill::PF_THREADS, 1) lux_attn_prefill_f32(const PrefillArgs p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t bh = p.batch * p.heads, rest = blockIdx.x % bh;
    prefill::attend_f32(p, smem, p.q_blocks - 1u - blockIdx.x / bh, rest % p.heads, rest / p.heads);
}

static_assert(THREADS == prefill::PF_THREADS && BM == prefill::PF_BM && SMEM >= prefill::PF_SMEM + 128, "a block can change over");

}  // namespace pmma
}  // namespace

LuxBackendError launch_attn_prefill(Context* ctx, PrefillArgs p, bool f32_only) {
    using namespace pmma;
    auto kfn = f32_only ? lux_attn_prefill_f32 : lux_attn_prefill_mma_f32;
    const char* name = f32_only ? "lux_attn_prefill_f32" : "lux_attn_prefill_mma_f32";
    static std::atomic<bool> configured[2][64];
    std::atomic<bool>& done = configured[f32_only][ctx->device & 63];
    if (!done.load(std::memory_order_relaxed)) {
        cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) return map_cuda(e, name);
        done.store(true, std::memory_order_relaxed);
    }
    p.q_blocks = (p.seq_q + pmma::BM - 1) / pmma::BM;
    cudaError_t e = launch_pdl(g_tune.pdl != 2, kfn, dim3(p.q_blocks * p.heads * p.batch), dim3(THREADS), (size_t)SMEM, ctx->stream, 1, p);
    if (e != cudaSuccess) return map_cuda(e, name);
    count_launch(name);
    return LUX_BACKEND_OK;
}

const void* kernel_addr_attn_prefill_mma_f32() { return (const void*)pmma::lux_attn_prefill_mma_f32; }
const void* kernel_addr_attn_prefill_f32() { return (const void*)pmma::lux_attn_prefill_f32; }

}  // namespace luxcuda
