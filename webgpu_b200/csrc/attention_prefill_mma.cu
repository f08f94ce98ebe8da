// attention_prefill_mma.cu -- attention of many query rows per head on the tensor cores, f32 in and out, head size 128.
//
// The f32 FMA pipe (72 TFLOP/s) is not what a prompt has to be bound by.  An f32 number is the exact sum of three bf16
// parts, h = bf16(x), m = bf16(x - h), l = x - h - m, and
//     a b = ah bh + (ah bm + am bh) + (am bm + ah bl + al bh)
// leaves out only am bl + al bm + al bl <= 2^-24 |a b|, what rounding the product to f32 would cost.  Six bf16 products
// on tcgen05 (8192 flop per clock and SM) replace one f32 product.
//
// Range.  bf16 has f32's exponents, so a part depends on its own element alone: no scale is shared along a row, a
// column or a tile, and a masked key weighs exactly nothing however large its values.  A part below 2^-126 may be
// lost.  Weights are split times 2^30 (a weight is 2^-126 at least, or 0) and so keep their 24 bits; in a score
// 2^-126 x 2^60 x 128 is nothing; and V can lose 2^-126 of an output, which matters to outputs below 2^-100 alone:
// if V had non-zero values below 2^-100 and such an output comes out, the block is done on the f32 pipe.
// So is one that meets a magnitude of 2^60 or more (after Q's scale), an infinity or a NaN: with all below 2^60
// no score, no sum (2^120 x 128; 2^(8 + 30 + 60) a key) and no bf16 rounding overflows.  A block (a CTA: 128 queries of
// one head) starts over by itself (attention_prefill_f32.cuh), before it has written anything: this holds with
// out == q, and no other block, call or replay of a captured one takes part.
//
// Two kernels.  (Where the parts of all keys do not fit the scratch, a pair of them per pass, attention_passes.h: blocks then carry their
// outputs, maxima and denominators from one range of keys to the next, merged by the running-maximum rule.)  lux_attn_split_kv writes the parts of K and V once per call, tile by tile as the tensor core wants them in
// shared memory, into the context's scratch (split in every CTA instead, an element would be converted 64 times in a
// 2048-token prompt, and the parts' way through shared memory would take as long as the products).
// lux_attn_prefill_mma_f32 is a pair of CTAs (two heads that share a KV head and their 128 queries, or two
// blocks of queries of one head where heads do not pair up) that works on 64-key tiles with cta_group::2 products of
// 256 rows: each CTA holds one half of every tile, so a tile crosses L2 -> SM once per pair (48 KB per CTA and 3.2 k cycles).
//   warp 9      bulk copies of the pair's K and V halves, seven slots of 24 KB
//   warp 8      issues: scores of tile t + 1, then the weighted sum of tile t (in the pair's second CTA it passes on
//               "my half has landed" instead)
//   warps 0..3  a thread per row: scores from tensor memory, softmax without any exchange, weights back as operand
//   warps 4..7  a thread per row: the running output in registers; adds each tile's 128 columns
// Tensor memory (512 columns): Q's h and m parts 128, scores 2 x 64, weights 96, weighted sum 128.  Q's l part, one
// product in six, is read from shared memory.
//
// Accumulation.  The tensor core cuts its f32 sums off at every step of 16 (measured on chains of 1 / 2 / 4 / 8 steps:
// mean loss 1.1 / 2.4 / 4.9 / 9.4e-8 of the sum, in rms 2.5 / 3.9 / 6.5 / 11.6e-8), so chains are four steps of the large products, after
// the small ones: a score is the f32 sum of two such chains, and the output is kept in f32 registers, to which each
// tile of 64 keys is added by an ordinary rounded addition.  What the weighted sum of a tile loses on average (signed, N(0, 1) inputs:
// 3.6e-8 of it with 2 keys, 4.1 with 16, 5.2 with 32, 6.5 with 48, 7.8 with 64; scores six times as large give the same) is added to the
// quotient before its one rounding, which leaves at most 0.9e-8; a row with a single weight loses nothing and is its value bit for bit.
// The log-sum-exp takes the denominator as it is.
// Relative error against 64 bits, in 1e-7 (2-norm, N(0, 1) inputs, Llama-3-8B heads; streaming kernel / mma.sync form of this
// one / this one): causal, 64 tokens 1.22 / 0.96 / 0.84, 150 1.36 / 1.08 / 0.92, 512 1.68 / 1.23 / 1.05, 2048 2.25 / 1.42 / 1.20; unmasked,
// 700 x 3 3.12 / 1.82 / 1.50, 1448 4.05 / 2.05 / 1.70.  The log-sum-exp (rms, a unit in its last place being 4.8): 1.69 / 1.48 / 1.62 at 150,
// 2.47 / 2.13 / 2.22 at 2048, 2.49 / 2.05 / 2.16 at 1448 (scores of both signs are cut towards zero, which takes 0.6 off it on average).
//
// Measured, Llama-3-8B heads, against the form with mma.sync products and the splitting in every CTA (bound by that instruction,
// 568 TFLOP/s, and by the splitting): causal, 2048 tokens 674 -> 167 us (206 TFLOP/s of f32 products, 1.24 PFLOP/s of
// bf16 ones), 192 where a call follows others under the power cap, 512 tokens 95 -> 32, 150 tokens 28.7 -> 15.4; unmasked
// 700 tokens x 3 511 -> 138.  The tensor pipe is busy for 62 % of the time, at 1.63 GHz; two softmax warps per row instead of one
// gave 1 %.
#include "attention_passes.h"
#include "attention_prefill_f32.cuh"
#include "attention_ring.h"

#include <algorithm>
#include <cstddef>
#include <new>

namespace luxcuda {

namespace {
namespace pmma {

using namespace tcptx;

constexpr int D = 128;                    // head size
constexpr int BM = 128;                   // queries per CTA
constexpr int BN = 64;                    // keys per tile
constexpr int THREADS = 384;              // three warpgroups
// registers per thread of the softmax, output and copy / issue warpgroups; their sum is three times the 168 of the launch
constexpr int REGS_S = 208, REGS_O = 216, REGS_C = 80, REGS = 168;
constexpr int PART = 64 * D;              // bytes of one part of a CTA's half tile: K 32 keys x 128, V 64 keys x 64 columns
constexpr int SLOT = 3 * PART;            // K or V of a tile, one CTA's half
constexpr int SLOTS = 7;
constexpr size_t TILE_BYTES = 4 * SLOT;   // scratch per tile: K of rank 0, 1, V of rank 0, 1
constexpr size_t SCRATCH = 131072 / BN * TILE_SCRATCH;       // 201 MB
// Q's l part, ring, two rows of factors, denominators, maxima and losses, barriers and flags
constexpr int OFF_QL = 0, OFF_RING = BM * D * 2, OFF_ALPHA = OFF_RING + SLOTS * SLOT, OFF_STAT = OFF_ALPHA + 2 * BM * 4;
constexpr int OFF_BAR = OFF_STAT + 3 * BM * 4, OFF_FLAG = OFF_BAR + 256;
constexpr int SMEM = OFF_FLAG + 64 + 1024;
constexpr int OUT_PITCH = D + 4;          // floats between the rows of the output in shared memory (over the ring)
// tensor memory columns
constexpr uint32_t T_QH = 0, T_QM = 64, T_S = 128, T_P = 256, T_O = 384;
constexpr float NEG = -3.0e38f, LN2 = 0.6931471805599453f;
constexpr float RAISE = 8.0f;             // the running maximum is raised when a score passes it by more: weights below 2^8
constexpr float P_SCALE = 0x1p30f;        // of the weights before they are split
constexpr float LOSS_CHAIN = 2.2e-8f, LOSS_STEP = 1.4e-8f;   // what a weighted sum of one tile loses on average: per chain, per step of 16 keys
constexpr float LOSS = LOSS_CHAIN + LOSS_STEP * (BN / 16);
constexpr uint32_t TOO_LARGE = (127u + 60u) << 23;           // |x| >= 2^60, infinity or NaN, as bits
constexpr uint32_t TOO_SMALL = (127u - 100u) << 23;          // 0 < |v| < 2^-100
constexpr uint32_t FLAG_BAD = 1u, FLAG_TINY = 2u;            // of a tile of K or V

using prefill::add2;
using prefill::ex2;
using prefill::mul2;
using prefill::pair;
using prefill::unpair;

__device__ __forceinline__ uint32_t pack(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
// two values as pairs of their parts, the first in the low half; the two differences are exact
__device__ __forceinline__ void split3(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = pack(a, b);
    a -= __uint_as_float(h << 16);
    b -= __uint_as_float(h & 0xffff0000u);
    m = pack(a, b);
    l = pack(a - __uint_as_float(m << 16), b - __uint_as_float(m & 0xffff0000u));
}
__device__ __forceinline__ uint32_t abs_bits(float x) { return __float_as_uint(x) & 0x7fffffffu; }

template <int N> __device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// ---- cta_group::2 wrappers: 256 rows, 128 of each CTA --------------------------------------------------
__host__ __device__ constexpr uint32_t idesc2(int n, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | (16u << 24);
}
__device__ __forceinline__ void mma2_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void mma2_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives on the barrier of this offset in both CTAs when all products issued so far are complete
__device__ __forceinline__ void commit2(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// the same offset in the pair's first CTA
__device__ __forceinline__ uint32_t in_leader(uint32_t addr) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
    return r;
}
// Only tensor-memory reads and writes, already waited for, are ordered by it: a release at cluster scope would
// first wait for every store of the thread (600 cycles and more, three times a tile: 235 -> 184 us at 2048 tokens without).
__device__ __forceinline__ void arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Passes on to the leader what this thread has waited for: copies that have landed in this CTA's shared memory.
__device__ __forceinline__ void arrive_release_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// mbar_wait that takes over what such an arrival passes on
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag) {
    for (uint32_t it = 0; it < WAIT_LIMIT; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
        if ((it & 31u) == 31u && *abort_flag) return false;
    }
    *abort_flag = 1u;
    return false;
}

// The parts of a tile of K (blockIdx.z 0) or V (1), rows past the end as zeros, in the layout of the ring's slots:
//   K, rank r (keys 32 r ..): [part][64 columns][32 keys] rows of 128 bytes      (K-major operand, 128-byte swizzle)
//   V, rank r (columns 64 r ..): [part][64 keys] rows of 128 bytes               (MN-major operand, 128-byte swizzle)
// 4 bytes are read and 6 written per element: 2048 keys x 8 heads 42 MB.
__global__ void __launch_bounds__(256) lux_attn_split_kv(const float* __restrict__ k, const float* __restrict__ v, unsigned char* __restrict__ parts,
                                                         uint32_t* __restrict__ flags, uint32_t bk0, uint32_t kv_len, uint32_t kv_stride) {
    __shared__ uint32_t seen;
    const uint32_t t = blockIdx.x, bk = blockIdx.y, is_v = blockIdx.z, tid = threadIdx.x;
    if (tid == 0) seen = 0u;
    __syncthreads();
    pdl_wait();
    pdl_launch_dependents();                          // after the wait: what comes next starts behind everything before this kernel
    const float* src = (is_v ? v : k) + ((size_t)(bk0 + bk) * kv_stride + (size_t)t * BN) * D;
    unsigned char* dst = parts + ((size_t)bk * gridDim.x + t) * TILE_BYTES + (is_v ? 2 * SLOT : 0);
    const uint32_t nk = min((uint32_t)BN, kv_len - t * BN);
    uint32_t top = 0u, low = 0xffffffffu;             // largest magnitude; smallest non-zero one, less 1
    const bool wide = (reinterpret_cast<uintptr_t>(src) & 31u) == 0;
    float4 x[4][2];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t e = tid + 256u * i, key = e >> 4, c = e & 15u;      // 16-byte chunk c of a row's parts: columns 8 c ..
        x[i][0] = x[i][1] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (key < nk) {
            const float* at = src + (size_t)key * D + 8 * c;
            if (wide) {
                load32(at, x[i][0], x[i][1]);
            } else {
                x[i][0] = __ldg(reinterpret_cast<const float4*>(at));
                x[i][1] = __ldg(reinterpret_cast<const float4*>(at) + 1);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t e = tid + 256u * i, key = e >> 4, c = e & 15u;
        uint32_t w[3][4];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const float4 f = x[i][j];
            const uint32_t b0 = abs_bits(f.x), b1 = abs_bits(f.y), b2 = abs_bits(f.z), b3 = abs_bits(f.w);
            top = max(top, max(max(b0, b1), max(b2, b3)));
            low = min(low, min(min(b0 - 1u, b1 - 1u), min(b2 - 1u, b3 - 1u)));
            split3(f.x, f.y, w[0][2 * j], w[1][2 * j], w[2][2 * j]);
            split3(f.z, f.w, w[0][2 * j + 1], w[1][2 * j + 1], w[2][2 * j + 1]);
        }
        const uint32_t at = is_v ? (c >> 3) * SLOT + key * 128u : (key >> 5) * SLOT + (c >> 3) * (PART / 2) + (key & 31u) * 128u;
#pragma unroll
        for (int q = 0; q < 3; q++)
            *reinterpret_cast<uint4*>(dst + at + q * PART + (((c & 7u) ^ (key & 7u)) << 4)) = make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]);
    }
    const uint32_t f = (top >= TOO_LARGE ? FLAG_BAD : 0u) | (is_v && low < TOO_SMALL - 1u ? FLAG_TINY : 0u);
    if (f) atomicOr(&seen, f);
    __syncthreads();
    if (tid == 0) flags[((size_t)bk * gridDim.x + t) * 2 + is_v] = seen;
}

struct Geometry {
    const unsigned char* parts;  // of the KV heads bk0 .. bk0 + nbk (batch x kv_heads), all_tiles tiles each
    const uint32_t* flags;
    uint32_t bk0, nbk, all_tiles;
    uint32_t by_head;            // pairs are two heads (their number per KV head is even), else two blocks of queries
    uint32_t units, levels;      // pairs per KV head and block of queries; blocks of queries (pairs of them),
    uint32_t level0;             // from this one on
    // A pass over the keys key0 .. key0 + keys.  Unless it is the first and the last, blocks carry what they have so far:
    // CARRY_ROW floats a row, at the same block of the grid in every pass, and CARRY_BAD, FLAG_TINY.
    uint32_t key0, keys, first, last;
    float* carry;
    uint32_t* carry_flags;
};
constexpr int CARRY_ROW = D + 4;          // the outputs, maximum, denominator, loss; whole 16 bytes
static_assert(TILE_SCRATCH == TILE_BYTES + 8 && CARRY == BM * CARRY_ROW * 4 + 16, "tiles and carried blocks with their flags");
constexpr uint32_t CARRY_BAD = 1u;

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1) lux_attn_prefill_mma_f32(const PrefillArgs p, const Geometry geo) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t sb = smem_u32(smem);
    float* alpha_s = reinterpret_cast<float*>(smem + OFF_ALPHA);
    float* stat = reinterpret_cast<float*>(smem + OFF_STAT);
    const uint32_t bars = sb + OFF_BAR;
    auto kv_full = [&](uint32_t s) { return bars + 8u * s; };
    auto kv_empty = [&](uint32_t s) { return bars + 8u * (SLOTS + s); };
    const uint32_t s_full = bars + 8u * (2 * SLOTS), s_free = s_full + 8u, p_ready = s_full + 16u, o_full = s_full + 24u, o_free = s_full + 32u,
                   alpha_ready = s_full + 40u;    // two of these
    volatile uint32_t* flag = reinterpret_cast<volatile uint32_t*>(smem + OFF_FLAG);
    volatile uint32_t* abort_flag = flag;
    volatile uint32_t* seen = flag + 1;           // FLAG_BAD, FLAG_TINY of what this CTA reads
    volatile uint32_t* peer_bad = flag + 2;
    uint32_t* tmem_slot = const_cast<uint32_t*>(flag + 3);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_ctarank();

    pdl_launch_dependents();
    // blocks of late queries see the most keys under a causal mask: they come first, so that the last
    // wave is made of short ones.  Neighbouring pairs are heads of one KV head and share its tiles in L2.
    const uint32_t per_level = geo.nbk * geo.units;
    const uint32_t level = geo.level0 + geo.levels - 1u - (blockIdx.x >> 1) / per_level, rest = (blockIdx.x >> 1) % per_level;
    const uint32_t unit = rest % geo.units, bkl = rest / geo.units, bk = geo.bk0 + bkl, b = bk / p.kv_heads;
    const uint32_t h = bk % p.kv_heads * p.group + (geo.by_head ? 2u * unit + rank : unit);
    const uint32_t qb = geo.by_head ? level : 2u * level + rank;
    const uint32_t q0 = qb * BM, rows = q0 < p.seq_q ? min((uint32_t)BM, p.seq_q - q0) : 0u;
    auto row_len = [&](uint32_t qi) {             // of the keys of this pass
        const uint32_t n = p.causal ? min(p.causal_base + qi + 1u, p.kv_len) : p.kv_len;
        return min(max(n, geo.key0) - geo.key0, geo.keys);
    };
    const uint32_t lmax = rows ? row_len(q0 + rows - 1u) : 0u, own_tiles = (lmax + BN - 1u) / BN;
    const uint32_t pair_last = min(p.seq_q, (geo.by_head ? level + 1u : 2u * level + 2u) * BM) - 1u;
    const uint32_t tiles = (row_len(pair_last) + BN - 1u) / BN;            // the pair walks them together
    const unsigned char* tile0 = geo.parts + (size_t)bkl * geo.all_tiles * TILE_BYTES + rank * SLOT;

    if (tid == 0) {
        for (uint32_t s = 0; s < SLOTS; s++) {
            mbar_init(kv_full(s), rank == 0 ? 2u : 1u);         // the first CTA's: both halves
            mbar_init(kv_empty(s), 1u);
        }
        mbar_init(s_full, 1u);
        mbar_init(s_free, 8u);                    // four warps of each CTA
        mbar_init(p_ready, 8u);
        mbar_init(o_full, 1u);
        mbar_init(o_free, 8u);
        mbar_init(alpha_ready, 4u);
        mbar_init(alpha_ready + 8u, 4u);
        *abort_flag = 0u;
        *seen = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot, quad = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    // Q comes from kernels before lux_attn_split_kv, which has waited for them before it let this one start: it may be read
    // while K and V are still being split (from L2: this SM may have read an earlier call's; 512 tokens 33.4 -> 30.3 us).  Without keys nothing is split, and the wait comes first.
    if (!geo.all_tiles) pdl_wait();

    // the ring: K0, K1, V0, K2, V1, ... in both CTAs, in the order in which the products read them
    auto slot_at = [&](uint32_t i) { return sb + OFF_RING + (i % SLOTS) * SLOT; };
    const uint32_t entries = 2u * tiles;
    auto request = [&](uint32_t i) {
        const RingEntry e = ring_entry(i, tiles);
        const uint32_t bar = kv_full(i % SLOTS);
        mbar_expect_tx(bar, SLOT);
        bulk_g2s(slot_at(i), tile0 + (size_t)e.tile * TILE_BYTES + (e.is_v ? 2 * SLOT : 0), SLOT, bar);
    };
    if (warp == 9) {
        pdl_wait();
        if (lane == 0)
            for (uint32_t i = 0; i < min(entries, (uint32_t)SLOTS); i++) request(i);
    }

    // ---- Q: rows on lanes, scaled and split; warps 0..3 take columns 0..63, warps 4..7 the others ---------
    const uint32_t row = (uint32_t)((warp & 3) * 32 + lane);
    uint32_t found = 0u;
    if (warp < 8) {
        const int half = warp >> 2;
        uint32_t qh[32], qm[32];
        const float* src = p.q + (((size_t)b * p.heads + h) * p.seq_q + q0 + min(row, max(rows, 1u) - 1u)) * D + half * 64;
        float4 x[16];
#pragma unroll
        for (int j = 0; j < 16; j++) x[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (rows && (reinterpret_cast<uintptr_t>(p.q) & 31u) == 0) {         // whole sectors at a time, as L1 does not keep them (2048 tokens 178 -> 168 us)
#pragma unroll
            for (int j = 0; j < 16; j += 2)
                asm volatile("ld.global.cg.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                             : "=f"(x[j].x), "=f"(x[j].y), "=f"(x[j].z), "=f"(x[j].w), "=f"(x[j + 1].x), "=f"(x[j + 1].y), "=f"(x[j + 1].z), "=f"(x[j + 1].w)
                             : "l"(src + 4 * j) : "memory");
        } else if (rows) {
#pragma unroll
            for (int j = 0; j < 16; j++) x[j] = __ldcg(reinterpret_cast<const float4*>(src) + j);
        }
        uint32_t top = 0u;
        unsigned char* ql = smem + OFF_QL + half * (BM * 128) + row * 128u;
#pragma unroll
        for (int c = 0; c < 8; c++) {
            uint32_t l[4];
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const float4 v = x[2 * c + j];
                const float4 y = make_float4(v.x * p.qscale, v.y * p.qscale, v.z * p.qscale, v.w * p.qscale);
                top = max(top, max(max(abs_bits(y.x), abs_bits(y.y)), max(abs_bits(y.z), abs_bits(y.w))));
                const int e = 4 * c + 2 * j;
                split3(y.x, y.y, qh[e], qm[e], l[2 * j]);
                split3(y.z, y.w, qh[e + 1], qm[e + 1], l[2 * j + 1]);
            }
            *reinterpret_cast<uint4*>(ql + (((uint32_t)c ^ (row & 7u)) << 4)) = make_uint4(l[0], l[1], l[2], l[3]);
        }
        tmem_st32(quad + T_QH + half * 32, qh);
        tmem_st32(quad + T_QM + half * 32, qm);
        tmem_st_wait();
        if (top >= TOO_LARGE) found = FLAG_BAD;
    }
    pdl_wait();
    for (uint32_t i = tid; i < 2u * own_tiles; i += THREADS) found |= geo.flags[(size_t)bkl * geo.all_tiles * 2u + i];
    if (found) atomicOr(const_cast<uint32_t*>(seen), found);
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {                               // a CTA without rows has nothing to lose
        uint32_t there;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(smem_u32(const_cast<uint32_t*>(peer_bad))), "r"(rank ^ 1u));
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(there), "r"((*seen & FLAG_BAD) || !rows ? 1u : 0u) : "memory");
    }
    cluster_sync_all();
    tc_fence_after();
    const bool bad = (*seen & FLAG_BAD) || !rows;
    // both start over: no products.  One of them: the pair works on, for the other's sake.
    const uint32_t walk = bad && *peer_bad ? 0u : tiles;
    float* out_s = reinterpret_cast<float*>(smem + OFF_RING);
    bool low = false;                             // an output that V's lost parts could matter to
    static_assert(REGS_S + REGS_O + REGS_C <= 3 * REGS, "what the launch has");
    if (warp >= 8) {
        regs_dec<REGS_C>();
        if (warp == 9) {
            if (lane == 0) {
                for (uint32_t i = SLOTS; walk && i < entries; i++) {
                    if (!mbar_wait_relaxed(kv_empty(i % SLOTS), (i / SLOTS - 1u) & 1u, abort_flag)) break;
                    request(i);
                }
                // nobody else waits for what was requested above
                for (uint32_t i = 0; !walk && i < min(entries, (uint32_t)SLOTS); i++) mbar_wait(kv_full(i), 0u, abort_flag);
            }
        } else if (warp == 8 && rank == 0) {
            if (elect_one()) {
                constexpr uint32_t id_s = idesc2(BN, false), id_o = idesc2(D, true);
                uint32_t i = 0;                   // ring entry
                auto take = [&]() { return mbar_wait_cluster(kv_full(i % SLOTS), (i / SLOTS) & 1u, abort_flag); };
                // Only slots that are filled again are given back: an arrival in the second CTA that nobody there waits for
                // could come after that CTA has ended.
                auto give_back = [&]() {
                    if (ring_refilled(i, entries, SLOTS)) commit2(kv_empty(i % SLOTS));
                    i++;
                };
                auto scores = [&]() {
                    const uint64_t kd = make_kmajor_sw128_desc(slot_at(i)), ld = make_kmajor_sw128_desc(sb + OFF_QL);
                    tc_fence_after();
#pragma unroll
                    for (int c = 0; c < 2; c++) { // columns 64 c .. of the head
                        const uint32_t d = tmem + T_S + c * BN;
                        // l h, h l, m m, m h, h m, h h
#pragma unroll
                        for (int s = 0; s < 4; s++)
                            mma2_ss(d, ld + (uint64_t)(c * (BM * 128 / 16) + 2 * s), kd + (uint64_t)(c * (PART / 32) + 2 * s), id_s, s != 0);
#pragma unroll
                        for (int o = 1; o < 6; o++) {
                            const int a = o == 2 || o == 3 ? 1 : 0, w = o == 1 ? 2 : o == 2 || o == 4 ? 1 : 0;
#pragma unroll
                            for (int s = 0; s < 4; s++)
                                mma2_ts(d, tmem + (a ? T_QM : T_QH) + c * 32 + s * 8, kd + (uint64_t)(w * (PART / 16) + c * (PART / 32) + 2 * s), id_s, 1u);
                        }
                    }
                    commit2(s_full);
                    give_back();
                };
                auto weighted = [&]() {
                    // MN-major: rows of 128 bytes are keys, eight of them a swizzle atom, one atom column wide
                    const uint64_t vd = make_kmajor_sw128_desc(slot_at(i));
                    tc_fence_after();
#pragma unroll
                    for (int o = 0; o < 6; o++) {
                        const int a = o == 0 ? 2 : o == 2 || o == 3 ? 1 : 0, w = o == 1 ? 2 : o == 2 || o == 4 ? 1 : 0;
#pragma unroll
                        for (int s = 0; s < 4; s++)
                            mma2_ts(tmem + T_O, tmem + T_P + a * 32 + s * 8, vd + (uint64_t)(w * (PART / 16) + s * (16 * 128 / 16)), id_o, (o | s) != 0);
                    }
                    commit2(o_full);
                    give_back();
                };
                bool ok = walk > 0 && take();
                if (ok) scores();
                for (uint32_t t = 0; ok && t < walk; t++) {
                    if (t + 1 < walk) {
                        ok = take() && mbar_wait(s_free, t & 1u, abort_flag);
                        if (!ok) break;
                        scores();
                    }
                    ok = take() && mbar_wait(p_ready, t & 1u, abort_flag) && (t == 0 || mbar_wait(o_free, (t - 1u) & 1u, abort_flag));
                    if (!ok) break;
                    weighted();
                }
            }
        } else if (warp == 8) {
            if (lane == 0)
                for (uint32_t i = 0; i < (walk ? entries : min(entries, (uint32_t)SLOTS)); i++) {
                    if (!mbar_wait(kv_full(i % SLOTS), (i / SLOTS) & 1u, abort_flag)) break;
                    arrive_release_cluster(in_leader(kv_full(i % SLOTS)));
                }
        }
        __syncwarp();
        cluster_sync_all();
        regs_inc<REGS>();
    } else if (warp < 4) {
        // ---- softmax: this thread's row of every tile ------------------------------------------------
        regs_inc<REGS_S>();
        const uint32_t len = row < rows ? row_len(q0 + row) : 0u;        // a padding row sees nothing and is not written
        const uint32_t free_bar = in_leader(s_free), ready_bar = in_leader(p_ready);
        float m = NEG, l = 0.0f, kept = 0.0f;     // kept: of the loss that l stands for, what a tile's unseen keys leave out
        for (uint32_t t = 0; t < walk; t++) {
            if (!warp_wait(s_full, t & 1u, abort_flag, lane)) break;
            const bool own = t < own_tiles;
            uint64_t s2[BN / 2];
            tc_fence_after();
            if (own) {
                uint32_t a[2][32], c[2][32];
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    tmem_ld32(quad + T_S + 32 * i, a[i]);
                    tmem_ld32(quad + T_S + BN + 32 * i, c[i]);
                }
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < BN / 2; j++)
                    s2[j] = add2(pair(__uint_as_float(a[j >> 4][2 * (j & 15)]), __uint_as_float(a[j >> 4][2 * (j & 15) + 1])),
                                 pair(__uint_as_float(c[j >> 4][2 * (j & 15)]), __uint_as_float(c[j >> 4][2 * (j & 15) + 1])));
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_cluster(free_bar);
            float alpha = 1.0f;
            uint32_t wh[32], wm[32], wl[32];
            if (own) {
                const uint32_t t0 = t * BN;
                float s[BN];
#pragma unroll
                for (int j = 0; j < BN / 2; j++) unpair(s2[j], s[2 * j], s[2 * j + 1]);
                if (t0 + BN > len) {
#pragma unroll
                    for (int j = 0; j < BN; j++)
                        if (t0 + j >= len) s[j] = -__int_as_float(0x7f800000);
                }
                float mt[4];
#pragma unroll
                for (int j = 0; j < 4; j++) mt[j] = fmaxf(s[j], s[j + 4]);
#pragma unroll
                for (int j = 8; j < BN; j++) mt[j & 3] = fmaxf(mt[j & 3], s[j]);
                const float top = fmaxf(fmaxf(mt[0], mt[1]), fmaxf(mt[2], mt[3]));
                if (top > m + RAISE) {
                    alpha = ex2(m - top);
                    m = top;
                    l *= alpha;
                }
                const uint64_t m2 = pair(-m, -m), scale2 = pair(P_SCALE, P_SCALE);
                uint64_t sum[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
                for (int j = 0; j < BN / 2; j++) {
                    float x, y;
                    unpair(add2(pair(s[2 * j], s[2 * j + 1]), m2), x, y);
                    const uint64_t e = pair(ex2(x), ex2(y));
                    sum[j & 3] = add2(sum[j & 3], e);
                    unpair(mul2(e, scale2), x, y);
                    split3(x, y, wh[j], wm[j], wl[j]);
                }
                float x, y;
                unpair(add2(add2(sum[0], sum[1]), add2(sum[2], sum[3])), x, y);
                x += y;
                l += x;
                if (t0 + BN > len && t0 < len) kept = x * (LOSS_STEP * (float)((t0 + BN - len) / 16u));       // (the row's last keys)
            }
            // the weighted sum before this one has read its weights
            if (t && !warp_wait(o_full, (t - 1u) & 1u, abort_flag, lane)) break;
            tc_fence_after();
            alpha_s[(t & 1u) * BM + row] = alpha;
            if (own) {
                tmem_st32(quad + T_P, wh);
                tmem_st32(quad + T_P + 32, wm);
                tmem_st32(quad + T_P + 64, wl);
                tmem_st_wait();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(alpha_ready + 8u * (t & 1u));
                arrive_cluster(ready_bar);
            }
        }
        stat[row] = l;
        stat[BM + row] = m;
        stat[2 * BM + row] = l == 1.0f ? 0.0f : LOSS - kept / fmaxf(l, 1.0f);      // (a single weight is its value's three parts: nothing is cut off)
        __syncwarp();
        cluster_sync_all();
        regs_dec<REGS>();
    } else {
        // ---- the output: this thread's row ------------------------------------------------------------
        regs_inc<REGS_O>();
        const uint32_t free_bar = in_leader(o_free);
        uint64_t o[D / 2];
#pragma unroll
        for (int j = 0; j < D / 2; j++) o[j] = 0ull;
        for (uint32_t t = 0; t < walk; t++) {
            if (!warp_wait(alpha_ready + 8u * (t & 1u), (t >> 1) & 1u, abort_flag, lane) || !warp_wait(o_full, t & 1u, abort_flag, lane)) break;
            tc_fence_after();
            if (t < own_tiles) {
                const float alpha = alpha_s[(t & 1u) * BM + row];
                if (__any_sync(0xffffffffu, alpha != 1.0f)) {
                    const uint64_t a2 = pair(alpha, alpha);
#pragma unroll
                    for (int j = 0; j < D / 2; j++) o[j] = mul2(o[j], a2);
                }
#pragma unroll
                for (int i = 0; i < 4; i += 2) {
                    uint32_t c[2][32];
                    tmem_ld32(quad + T_O + 32 * i, c[0]);
                    tmem_ld32(quad + T_O + 32 * i + 32, c[1]);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        o[16 * i + j] = add2(o[16 * i + j], pair(__uint_as_float(c[j >> 4][2 * (j & 15)]), __uint_as_float(c[j >> 4][2 * (j & 15) + 1])));
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_cluster(free_bar);
        }
        // every product has been waited for (the last tile's here): the ring and the tensor memory are free once both CTAs are here
        __syncwarp();
        cluster_sync_all();
        if (!*abort_flag) {
#pragma unroll
            for (int j = 0; j < D / 4; j++) {
                float4 v;
                unpair(o[2 * j], v.x, v.y);
                unpair(o[2 * j + 1], v.z, v.w);
                *reinterpret_cast<float4*>(out_s + row * OUT_PITCH + 4 * j) = v;
            }
        }
        if ((*seen & FLAG_TINY) && row < rows && geo.first && geo.last) {
            const float least = stat[row] * (P_SCALE * 0x1p-100f);
#pragma unroll
            for (int j = 0; j < D / 2; j++) {
                float x, y;
                unpair(o[j], x, y);
                low |= fabsf(x) < least || fabsf(y) < least;
            }
        }
        __syncwarp();
        regs_dec<REGS>();
    }
    if (warp == 8) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    bool again = __syncthreads_or(low) || bad;
    if (*abort_flag) {
        // a bounded wait gave up: report it, and give copies in flight time to land.  Nothing has been written.
        if (tid == 0 && p.status) atomicOr(p.status, p.status_wait);
        for (int i = 0; i < 64; i++) __nanosleep(1000);
        __syncthreads();
        return;
    }
    if (!rows) return;
    if (!(geo.first && geo.last)) {               // this pass's part of the rows, with what the earlier ones left
        const uint32_t before = geo.first ? 0u : __ldcg(geo.carry_flags + blockIdx.x);
        const uint32_t so_far = before | (again ? CARRY_BAD : 0u) | (*seen & FLAG_TINY);
        float* mine = geo.carry + (size_t)blockIdx.x * (BM * CARRY_ROW);
        __syncthreads();                          // all have read the flags
        if (tid == 0) __stcg(geo.carry_flags + blockIdx.x, so_far);
        bool small = false;
        if (!(so_far & CARRY_BAD)) {
            for (uint32_t r = warp; r < rows; r += THREADS / 32) {
                float l = stat[r], m = stat[BM + r], cut = stat[2 * BM + r] * l;
                float4 v = *reinterpret_cast<const float4*>(out_s + r * OUT_PITCH + 4 * lane);
                float* there = mine + r * CARRY_ROW;
                if (!geo.first) {
                    const float4 c = __ldcg(reinterpret_cast<const float4*>(there) + lane), s = __ldcg(reinterpret_cast<const float4*>(there + D));
                    const float top = fmaxf(m, s.x), a = ex2(m - top), b = ex2(s.x - top);
                    v = make_float4(fmaf(v.x, a, c.x * b), fmaf(v.y, a, c.y * b), fmaf(v.z, a, c.z * b), fmaf(v.w, a, c.w * b));
                    l = fmaf(l, a, s.y * b);
                    cut = fmaf(cut, a, s.z * b);
                    m = top;
                }
                if (geo.last) {
                    __syncwarp();                 // all lanes have read the row's numbers
                    const float least = l * (P_SCALE * 0x1p-100f);
                    small |= fabsf(v.x) < least || fabsf(v.y) < least || fabsf(v.z) < least || fabsf(v.w) < least;
                    *reinterpret_cast<float4*>(out_s + r * OUT_PITCH + 4 * lane) = v;
                    if (lane == 0) {
                        stat[r] = l;
                        stat[BM + r] = m;
                        stat[2 * BM + r] = l > 0.0f ? cut / l : 0.0f;
                    }
                } else {
                    __stcg(reinterpret_cast<float4*>(there) + lane, v);
                    if (lane == 0) __stcg(reinterpret_cast<float4*>(there + D), make_float4(m, l, cut, 0.0f));
                }
            }
        }
        if (!geo.last) return;
        again = (so_far & CARRY_BAD) || ((so_far & FLAG_TINY) && __syncthreads_or(small));
        __syncthreads();
    }
    if (again) {                                  // values out of range: the block starts over on the f32 pipe
        if (tid < prefill::PF_THREADS) prefill::attend_f32(p, smem, qb, h, b);
        return;
    }
    const size_t orow = ((size_t)b * p.heads + h) * p.seq_q + q0;
    for (uint32_t r = warp; r < rows; r += THREADS / 32) {
        const float l = stat[r], inv = 1.0f / l, loss = stat[2 * BM + r];
        float4 v = *reinterpret_cast<const float4*>(out_s + r * OUT_PITCH + 4 * lane);
        // an estimate of the quotient; then what it leaves of the dividend, and the mean loss, before the one rounding that counts
        auto quotient = [&](float a) {
            const float c = a * inv;
            return fmaf(fmaf(loss, a, fmaf(-c, l, a)), inv, c) * (1.0f / P_SCALE);
        };
        v = l > 0.0f ? make_float4(quotient(v.x), quotient(v.y), quotient(v.z), quotient(v.w)) : make_float4(0.f, 0.f, 0.f, 0.f);   // a row without keys is zero
        *reinterpret_cast<float4*>(p.out + (orow + r) * D + 4 * lane) = v;
    }
    if (p.lse && tid < (int)rows) p.lse[orow + tid] = stat[tid] > 0.0f ? fmaf(stat[BM + tid], LN2, logf(stat[tid])) : -3.402823e+38f;
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

static_assert(THREADS >= prefill::PF_THREADS && BM == prefill::PF_BM && SMEM >= prefill::PF_SMEM + 1024, "a block can start over");
static_assert(BM * OUT_PITCH * 4 <= SLOTS * SLOT && (2 * SLOTS + 7) * 8 <= 256, "layout of the shared memory");

cudaError_t allow_smem(const void* kfn, int which, int bytes, int device) {
    static std::atomic<bool> configured[2][64];
    std::atomic<bool>& done = configured[which][device & 63];
    if (done.load(std::memory_order_relaxed)) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) done.store(true, std::memory_order_relaxed);
    return e;
}

// Allocates and frees wherever the caller is, in a capture too (neither becomes part of it).
struct Uncaptured {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    Uncaptured() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~Uncaptured() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// The context's scratch, from the first call on that needs it; less of it, or none, where memory is short.
void context_scratch(Context* ctx) {
    Uncaptured scope;
    for (size_t n = SCRATCH; !ctx->d_parts && n >= 64 * TILE_SCRATCH; n /= 2) {
        if (cudaMalloc(&ctx->d_parts, n) == cudaSuccess) {
            ctx->d_parts_bytes = n;
        } else {
            ctx->d_parts = nullptr;
            cudaGetLastError();
        }
    }
}

// Scratch of at least `want` bytes for a call that is being captured: the graph's own, shared by what is captured one after the other on
// one stream, and kept until the graph and all that was instantiated from it are gone (a replay in flight included).  Null: there is none.
const GraphParts* graph_scratch(Context* ctx, size_t want) try {
    cudaStreamCaptureStatus st;
    unsigned long long id = 0;
    cudaGraph_t graph = nullptr;
    if (cudaStreamGetCaptureInfo(ctx->stream, &st, &id, &graph) != cudaSuccess || st != cudaStreamCaptureStatusActive) return nullptr;
    GraphParts* best = nullptr;
    for (GraphParts& g : ctx->graph_parts) {
        if (g.bytes < want) continue;
        const bool live = g.live->load(std::memory_order_acquire);
        if (live && g.capture == id && g.stream == ctx->stream) return &g;
        if (!live && (!best || g.bytes < best->bytes)) best = &g;         // a graph that is gone left it
    }
    if (!best) {
        Uncaptured scope;
        GraphParts g{nullptr, want, 0, nullptr, std::make_shared<std::atomic<bool>>(false)};
        ctx->graph_parts.reserve(ctx->graph_parts.size() + 1);
        if (cudaMalloc(&g.p, want) != cudaSuccess) return nullptr;
        ctx->graph_parts.push_back(std::move(g));
        best = &ctx->graph_parts.back();
    }
    auto* held = new std::shared_ptr<std::atomic<bool>>(best->live);
    auto release = [](void* h) {                      // may come from any thread, after the context
        auto* flag = static_cast<std::shared_ptr<std::atomic<bool>>*>(h);
        (*flag)->store(false, std::memory_order_release);
        delete flag;
    };
    cudaUserObject_t object;
    if (cudaUserObjectCreate(&object, held, release, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
        delete held;
        return nullptr;
    }
    best->live->store(true, std::memory_order_release);
    if (cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove) != cudaSuccess) {
        cudaUserObjectRelease(object, 1);
        return nullptr;
    }
    best->capture = id;
    best->stream = ctx->stream;
    return best;
} catch (const std::bad_alloc&) {
    return nullptr;
}

// Gives back what graphs that are gone have left.
void free_idle_graph_scratch(Context* ctx) {
    for (size_t i = 0; i < ctx->graph_parts.size();) {
        if (ctx->graph_parts[i].live->load(std::memory_order_acquire)) {
            i++;
            continue;
        }
        Uncaptured scope;
        cudaFree(ctx->graph_parts[i].p);
        ctx->graph_parts.erase(ctx->graph_parts.begin() + (std::ptrdiff_t)i);
    }
}

}  // namespace pmma
}  // namespace

LuxBackendError launch_attn_prefill(Context* ctx, PrefillArgs p, bool f32_only) {
    using namespace pmma;
    p.q_blocks = (p.seq_q + pmma::BM - 1) / pmma::BM;
    const uint32_t keys = p.causal ? (uint32_t)std::min<uint64_t>((uint64_t)p.causal_base + p.seq_q, p.kv_len) : p.kv_len;
    const uint32_t tiles = (keys + BN - 1) / BN, bks = p.batch * p.kv_heads;
    const size_t per_bk = tiles * TILE_SCRATCH;
    Geometry geo{};
    geo.by_head = p.group % 2 == 0;
    geo.units = geo.by_head ? p.group / 2 : p.group;
    const uint32_t levels = geo.by_head ? p.q_blocks : (p.q_blocks + 1) / 2;
    // The scratch is the context's, or the graph's for a call that is being captured.
    std::lock_guard<std::mutex> lk(ctx->parts_mu);
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(ctx->stream, &capture);
    if (e != cudaSuccess) return map_cuda(e, "lux_attn_prefill_mma_f32");
    const bool direct = capture == cudaStreamCaptureStatusNone;
    void* scratch = nullptr;
    size_t scratch_bytes = 0;
    if (direct) free_idle_graph_scratch(ctx);
    if (!f32_only && per_bk && direct) {
        context_scratch(ctx);
        scratch = ctx->d_parts;
        scratch_bytes = ctx->d_parts_bytes;
    } else if (!f32_only && per_bk) {
        const GraphParts* own = graph_scratch(ctx, per_bk > SCRATCH ? SCRATCH : std::min(bks * per_bk, SCRATCH));
        if (!own) cudaGetLastError();
        scratch = own ? own->p : nullptr;
        scratch_bytes = own ? own->bytes : 0;
    }
    const Passes plan = plan_passes(bks, levels, geo.units, tiles, scratch_bytes, (uint32_t)ctx->sm_count, (uint32_t)std::max(g_tune.attn_pass_tiles, 0));
    if (f32_only || !plan.heads) {                     // (no scratch)
        const char* name = "lux_attn_prefill_f32";
        e = allow_smem((const void*)lux_attn_prefill_f32, 0, prefill::PF_SMEM + 128, ctx->device);
        if (e == cudaSuccess)
            e = launch_pdl(g_tune.pdl != 2, lux_attn_prefill_f32, dim3(p.q_blocks * p.heads * p.batch), dim3(prefill::PF_THREADS),
                           (size_t)prefill::PF_SMEM + 128, ctx->stream, 1, p);
        if (e != cudaSuccess) return map_cuda(e, name);
        count_launch(name);
        return LUX_BACKEND_OK;
    }
    const char* name = "lux_attn_prefill_mma_f32";
    e = allow_smem((const void*)lux_attn_prefill_mma_f32, 1, SMEM, ctx->device);
    // behind the last call that used the context's scratch, on whichever stream that was
    if (e == cudaSuccess && direct && ctx->parts_used && !ctx->parts_ordered) e = cudaStreamWaitEvent(ctx->stream, ctx->parts_event, 0);
    auto pass = [&](uint32_t visible) {                // `visible`: keys of all passes
        unsigned char* parts = (unsigned char*)scratch;
        uint32_t* flags = (uint32_t*)(parts + (size_t)geo.nbk * geo.all_tiles * TILE_BYTES);
        geo.parts = parts;
        geo.flags = flags;
        if (geo.all_tiles) {
            const size_t at = (size_t)geo.key0 * D;
            e = launch_pdl(g_tune.pdl != 2, lux_attn_split_kv, dim3(geo.all_tiles, geo.nbk, 2), dim3(256), (size_t)0, ctx->stream, 1, p.k + at, p.v + at, parts, flags,
                           geo.bk0, std::min(visible - geo.key0, geo.keys), p.kv_stride);
            if (e != cudaSuccess) return;
            count_launch("lux_attn_split_kv");
        }
        e = launch_pdl(g_tune.pdl != 2, lux_attn_prefill_mma_f32, dim3(2u * geo.levels * geo.nbk * geo.units), dim3(THREADS), (size_t)SMEM, ctx->stream, 1, p, geo);
        if (e == cudaSuccess) count_launch(name);
    };
    for (geo.bk0 = 0; e == cudaSuccess && geo.bk0 < bks; geo.bk0 += geo.nbk) {
        geo.nbk = std::min(plan.heads, bks - geo.bk0);
        for (geo.level0 = 0; e == cudaSuccess && geo.level0 < levels; geo.level0 += geo.levels) {
            geo.levels = std::min(plan.levels, levels - geo.level0);
            // the keys that these queries see, in passes of equal numbers of tiles
            const uint64_t end = (uint64_t)(geo.level0 + geo.levels) * (geo.by_head ? 1u : 2u) * pmma::BM;
            const uint32_t visible = p.causal ? (uint32_t)std::min<uint64_t>(keys, (uint64_t)p.causal_base + end) : keys;
            const uint32_t n = (visible + BN - 1) / BN;
            geo.carry = (float*)((unsigned char*)scratch + plan.carry_at);
            geo.carry_flags = (uint32_t*)(geo.carry + (size_t)2u * geo.levels * geo.nbk * geo.units * (pmma::BM * CARRY_ROW));
            for (uint32_t t = 0; e == cudaSuccess && (t < n || t == 0); t += std::max(geo.all_tiles, 1u)) {
                geo.all_tiles = plan.pass_tiles(t, n);
                geo.first = t == 0;
                geo.last = t + geo.all_tiles == n;
                geo.key0 = t * BN;
                geo.keys = geo.all_tiles * BN;
                pass(visible);
            }
        }
    }
    if (e == cudaSuccess && direct) {
        e = cudaEventRecord(ctx->parts_event, ctx->stream);
        ctx->parts_used = ctx->parts_ordered = true;
    }
    return e == cudaSuccess ? LUX_BACKEND_OK : map_cuda(e, name);
}

const void* kernel_addr_attn_prefill_mma_f32() { return (const void*)pmma::lux_attn_prefill_mma_f32; }
const void* kernel_addr_attn_prefill_f32() { return (const void*)pmma::lux_attn_prefill_f32; }
const void* kernel_addr_attn_split_kv() { return (const void*)pmma::lux_attn_split_kv; }

}  // namespace luxcuda
