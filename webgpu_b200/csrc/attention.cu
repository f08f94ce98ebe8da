// attention.cu -- rotary embedding, scaled-dot-product attention, KV-cache append and attention over
// a contiguous or a paged KV cache, all f32 (lux/gpu/attention_ext.h).
//
// What the WGSL does (luxcpp/webgpu kernels/wgsl/gpu/scaled_dot_product_attention.wgsl:81-199, 386-489;
// steel/attention/paged.wgsl:55-405): one 256-thread workgroup per (batch, head, query) walks the
// keys three times, the third time recomputing every score once per output dimension.  Here one
// pass does it, and the pass is shaped by what bounds a decode step on this GPU, the read of the
// KV cache from HBM:
//   * a CTA owns one (sequence, KV head, block of query rows, slice of the keys).  All query heads
//     that share the KV head (and all appended tokens) are rows of the same CTA, so the cache is
//     read from HBM once per KV head, not once per query head;
//   * a producer warp streams 32-key chunks of K and V into a ring in shared memory with bulk
//     copies (cp.async.bulk, one per contiguous run: a whole chunk for a contiguous cache, one per
//     page for a paged one, the page numbers taken from a copy of the block table in shared
//     memory), each chunk signalled through an mbarrier; two CTAs of nine warps share an SM, each
//     with a ring of three chunks (D = 128);
//   * eight consumer warps share a chunk: a key is handled by 8 lanes, each holding 16-byte columns
//     of the row, so a warp takes 4 keys per step; every lane keeps two query rows in registers
//     and runs the running-maximum softmax (the rule of sdpa_flash, :217-362) on its own keys; lanes,
//     warps and, for long contexts, CTAs are merged at the end by the same rule (the partition
//     statistics of paged_attention_v2, paged.wgsl:351-405, are this merge);
//   * only ONE thread per CTA polls an mbarrier (warp 0, for the chunk to land).  Everything else
//     waits on named barriers (bar.sync / bar.arrive), where the hardware parks a warp until the
//     count is reached: the other consumer warps for "chunk ready", the producer for "stage free".
//     With every warp polling its mbarrier the kernel ran at 2.2-5.1 TB/s depending on how many
//     warps happened to be waiting; parked, at 5.0-6.5 TB/s on the same shapes (polls travel the same
//     queue as shared-memory loads and shuffles, and starved the warps that had work);
//   * keys are split over CTAs when there are fewer (sequence, KV head) pairs than SM slots, and
//     each CTA walks its chunks from a different starting point; a small second kernel, resident
//     early through programmatic dependent launch, merges the slices;
//   * a large paged cache whose sequences differ much in length is dealt out in even shares instead
//     (lux_attn_even_f32): one wave of CTAs, each with the same number of chunks of the (sequence,
//     KV head) items laid end to end, so that a CTA may finish one item and begin the next.  The
//     lengths are known on the device only: both kernels are launched and one of them leaves at once.
// The one polling wait is bounded: if it gives up it sets the CTA's abort flag, every warp leaves
// its loop (the consumers first release the stages the producer may be parked on), the device
// status word reports 0x7C050008 and the output of that CTA is not written.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <type_traits>

#include "attention_span.h"
#include "common.cuh"
#include "tc_ptx.cuh"
#include "lux/gpu/attention_ext.h"

namespace luxcuda {

namespace {

using namespace tcptx;

constexpr int ATT_CW = 8;                       // consumer warps
constexpr int ATT_THREADS = (ATT_CW + 1) * 32;  // + the producer warp
constexpr int ATT_CK = 32;                      // keys per staged chunk
constexpr int ATT_MAX_STAGES = 6;
constexpr int ATT_CTAS_PER_SM = 2;
constexpr int ATT_TABLE = 2048;                 // block-table entries a CTA keeps in shared memory
constexpr int ATT_HEADER = 128;                 // barriers, abort flag
constexpr int ATT_EVEN_HEADER = 512;            // lux_attn_even_f32: and, from byte 128 on, each consumer warp's Piece
constexpr int ATT_MAX_PARTS = 512;              // CTAs of lux_attn_even_f32
// floats in which the warps of a CTA of the even form leave their results: [warp][row][head_dim + 2], in whole 128-byte lines
__host__ __device__ constexpr uint32_t att_merge_floats(uint32_t head_dim, uint32_t rt) { return (ATT_CW * rt * (head_dim + 2u) + 31u) / 32u * 32u; }
constexpr size_t ATT_SMEM_BUDGET = 110u << 10;        // per CTA: two CTAs share an SM
constexpr float ATT_NEG = -3.0e38f;             // "no key seen yet" in the base-2 score domain
constexpr float ATT_LOG2E = 1.4426950408889634f;
constexpr float ATT_LN2 = 0.6931471805599453f;
constexpr uint32_t ATT_STATUS_WAIT = 0x7C050008u;     // a bounded wait of the attention kernel gave up
constexpr uint32_t ATT_STATUS_BLOCK = 0x7C050009u;    // a block-table entry outside the cache (read as block 0)
constexpr uint32_t ATT_STATUS_POSITION = 0x7C05000Au; // a rope position outside the cos/sin cache (pair not written)

struct AttnParams {
    const float* q;
    const float* k;
    const float* v;
    float* out;
    float* lse;                  // may be null
    const int32_t* block_tables; // paged only
    const int32_t* context_lens; // paged only
    float* part;                 // partial results: [out row][nsplit][head_dim + 2], or [CTA][2][row][head_dim + 2]
    uint32_t* status;
    uint32_t batch, heads, kv_heads, group, seq_q, head_dim;
    uint32_t kv_len;             // keys a row may see (contiguous caches); paged: context_lens decides
    uint32_t kv_stride;          // rows between the bases of two KV heads of a contiguous cache
    uint32_t causal, causal_base;// causal: query i sees min(causal_base + i + 1, kv_len) keys
    uint32_t block_size, max_blocks_per_seq, num_blocks;   // paged (block_size 0: contiguous)
    uint32_t rgp;                // row groups per CTA (1, 2, 4 or 8): rows per CTA = RT * rgp
    uint32_t rpb;                // rows per CTA
    uint32_t row_blocks, nsplit, split_keys, stages;
    // a paged cache that may be dealt out in even shares
    uint32_t full_chunks;        // 32-key chunks of a full cache, over all KV heads
    uint32_t slack;              // even shares if more of them than this are missing
    uint32_t share, ctas;        // chunks per CTA, at least; CTAs of lux_attn_even_f32
    AttnSpan* spans;             // per (sequence, KV head); ctas 0: slices
    float qscale;                // scale * log2(e)
};

// 2^x for x <= 0 (results below the normal range flush to 0), one MUFU operation
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Named barriers: a warp that waits on one is parked by the hardware and issues nothing, unlike a
// warp polling an mbarrier, whose polls share the queue that shared-memory loads and shuffles go
// through.  With eight warps polling for every chunk the warps that had work ran 2-3 times slower.
constexpr int ATT_BAR_READY = 1;           // consumer warps: the chunk has landed (warp 0 polled for it)
constexpr int ATT_BAR_FREE0 = 2;           // + stage (6 at most): every consumer warp is done with the stage (producer waits)
constexpr int ATT_BAR_MERGE = 8;           // consumer warps: the piece's results are in shared memory; have been read

__device__ __forceinline__ uint32_t row_len(const AttnParams& p, uint32_t qi, uint32_t kv_len) {
    return p.causal ? min(p.causal_base + qi + 1u, kv_len) : kv_len;
}

// Keys that sequence b of a paged cache holds.
__device__ __forceinline__ uint32_t paged_len(const AttnParams& p, uint32_t b) {
    const int32_t cl = p.context_lens[b];
    return cl <= 0 ? 0u : min((uint32_t)cl, p.max_blocks_per_seq * p.block_size);
}
__host__ __device__ __forceinline__ uint32_t chunks_of(uint32_t keys) { return (keys + ATT_CK - 1) / ATT_CK; }

// 32-key chunks of all sequences and KV heads of a paged cache; every warp for itself.
__device__ __forceinline__ uint32_t all_chunks(const AttnParams& p) {
    uint32_t sum = 0u;
    for (uint32_t b = threadIdx.x & 31u; b < p.batch; b += 32) sum += chunks_of(paged_len(p, b));
    for (int off = 16; off; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    return sum * p.kv_heads;
}
// Whether so many chunks are dealt out in even shares, not in slices.
__device__ __forceinline__ bool ragged(const AttnParams& p, uint32_t all) { return p.full_chunks - all > p.slack; }

// The rows of a consumer warp of lux_attn_even_f32: a lane's columns of RT query rows, their running maxima, denominators and
// outputs.  (lux_attn_stream_f32 has the same arithmetic written out in its loop: through this struct its registers were
// allotted otherwise and contiguous caches took 1 to 2 % longer, 32 x 2048 keys 93.5 -> 95.5 us a step.)
template <int VPL, int RT, bool FULL>
struct Rows {
    float4 q[RT][VPL], o[RT][VPL];
    float m[RT], l[RT];
    uint32_t len[RT], min_len;
    bool col_ok[VPL];

    __device__ __forceinline__ void columns(uint32_t D, int sub) {
#pragma unroll
        for (int j = 0; j < VPL; j++) col_ok[j] = (uint32_t)(j * 8 + sub) * 4u < D;
    }
    // rows row0 .. row0 + RT of KV head g of sequence b, which see kv_len keys
    __device__ __forceinline__ void begin(const AttnParams& p, uint32_t b, uint32_t g, uint32_t row0, uint32_t kv_len, int sub) {
        min_len = 0xffffffffu;
#pragma unroll
        for (int i = 0; i < RT; i++) {
            const uint32_t r = row0 + i;
            const bool valid = r < p.group * p.seq_q;
            const uint32_t qi = valid ? r / p.group : 0u, head = g * p.group + (valid ? r % p.group : 0u);
            len[i] = valid ? row_len(p, qi, kv_len) : 0xffffffffu;       // a padding row: q = 0, never written, never masks a chunk
            min_len = min(min_len, len[i]);
            const float* qr = p.q + (((size_t)b * p.heads + head) * p.seq_q + qi) * p.head_dim;
            m[i] = ATT_NEG;
            l[i] = 0.0f;
#pragma unroll
            for (int j = 0; j < VPL; j++) {
                float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
                if (valid && col_ok[j]) t = __ldg(reinterpret_cast<const float4*>(qr) + j * 8 + sub);
                q[i][j] = make_float4(t.x * p.qscale, t.y * p.qscale, t.z * p.qscale, t.w * p.qscale);
                o[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    }
    static __device__ __forceinline__ float4 lds4(uint32_t addr) {
        float4 r;
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "r"(addr));
        return r;
    }
    // One step: the warp's four keys (one per group of 8 lanes) against its RT rows.  The
    // running maximum of a lane is only raised when a score passes it by more than 8 (in the
    // base-2 domain), so weights stay below 2^8 and the common step has no rescaling in it:
    // scores, one exp2 per row, the weighted sum.  MASKED steps (the last chunk of a slice, a
    // causal edge) check each key against the chunk and each row's length.
    template <bool MASKED>
    __device__ __forceinline__ void step(uint32_t kaddr, uint32_t vaddr, bool inb, uint32_t t) {
        float sc[RT];
#pragma unroll
        for (int i = 0; i < RT; i++) sc[i] = 0.0f;
#pragma unroll
        for (int j = 0; j < VPL; j++) {
            float4 kk = make_float4(0.f, 0.f, 0.f, 0.f);
            if ((FULL || col_ok[j]) && (!MASKED || inb)) kk = lds4(kaddr + (uint32_t)j * 128u);
#pragma unroll
            for (int i = 0; i < RT; i++)
                sc[i] = fmaf(q[i][j].x, kk.x, fmaf(q[i][j].y, kk.y, fmaf(q[i][j].z, kk.z, fmaf(q[i][j].w, kk.w, sc[i]))));
        }
#pragma unroll
        for (int i = 0; i < RT; i++) {
            sc[i] += __shfl_xor_sync(0xffffffffu, sc[i], 1);
            sc[i] += __shfl_xor_sync(0xffffffffu, sc[i], 2);
            sc[i] += __shfl_xor_sync(0xffffffffu, sc[i], 4);
        }
        bool vis[RT], up = false, any = false;
#pragma unroll
        for (int i = 0; i < RT; i++) {
            vis[i] = !MASKED || (inb && t < len[i]);
            up |= vis[i] && sc[i] > m[i] + 8.0f;
            any |= vis[i];
        }
        if (__any_sync(0xffffffffu, up)) {
#pragma unroll
            for (int i = 0; i < RT; i++) {
                const float mn = vis[i] ? fmaxf(m[i], sc[i]) : m[i];
                const float alpha = ex2(m[i] - mn);
                l[i] *= alpha;
#pragma unroll
                for (int j = 0; j < VPL; j++) {
                    o[i][j].x *= alpha; o[i][j].y *= alpha; o[i][j].z *= alpha; o[i][j].w *= alpha;
                }
                m[i] = mn;
            }
        }
        float pw[RT];
#pragma unroll
        for (int i = 0; i < RT; i++) {
            pw[i] = ex2(sc[i] - m[i]);
            if (MASKED && !vis[i]) pw[i] = 0.0f;
            l[i] += pw[i];
        }
        if (!MASKED || any) {
#pragma unroll
            for (int j = 0; j < VPL; j++) {
                float4 vv = make_float4(0.f, 0.f, 0.f, 0.f);
                if (FULL || col_ok[j]) vv = lds4(vaddr + (uint32_t)j * 128u);
#pragma unroll
                for (int i = 0; i < RT; i++) {
                    o[i][j].x = fmaf(pw[i], vv.x, o[i][j].x);
                    o[i][j].y = fmaf(pw[i], vv.y, o[i][j].y);
                    o[i][j].z = fmaf(pw[i], vv.z, o[i][j].z);
                    o[i][j].w = fmaf(pw[i], vv.w, o[i][j].w);
                }
            }
        }
    }
    // a warp's part of a chunk of nk keys from key t0 on, at kchunk in shared memory (V: v_off further)
    __device__ __forceinline__ void chunk(uint32_t kchunk, uint32_t v_off, uint32_t row_bytes, uint32_t t0, uint32_t nk, uint32_t kslot, uint32_t wpg, int kg) {
        if (nk == ATT_CK && t0 + ATT_CK <= min_len) {
            for (uint32_t kb = kslot * 4u; kb < ATT_CK; kb += wpg * 4u) {
                const uint32_t ka = kchunk + (kb + (uint32_t)kg) * row_bytes;
                step<false>(ka, ka + v_off, true, 0u);
            }
        } else {
            for (uint32_t kb = kslot * 4u; kb < nk; kb += wpg * 4u) {
                const uint32_t key = kb + (uint32_t)kg, ka = kchunk + key * row_bytes;
                step<true>(ka, ka + v_off, key < nk, t0 + key);
            }
        }
    }
    // the four key slots of the warp, merged by the running-maximum rule
    __device__ __forceinline__ void fold(int i) {
        float mm = fmaxf(m[i], __shfl_xor_sync(0xffffffffu, m[i], 8));
        mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, 16));
        const float alpha = ex2(m[i] - mm);
        m[i] = mm;
        l[i] *= alpha;
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 8);
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 16);
#pragma unroll
        for (int j = 0; j < VPL; j++) {
            float* e = reinterpret_cast<float*>(&o[i][j]);
#pragma unroll
            for (int x = 0; x < 4; x++) {
                float val = e[x] * alpha;
                val += __shfl_xor_sync(0xffffffffu, val, 8);
                val += __shfl_xor_sync(0xffffffffu, val, 16);
                e[x] = val;
            }
        }
    }
    // row i to shared memory: outputs by column, its maximum and denominator at [D] and [D + 1] (rows are 8-byte aligned, not 16)
    __device__ __forceinline__ void store(int i, float* dst, uint32_t D, int lane) const {
        if (lane >= 8) return;
#pragma unroll
        for (int j = 0; j < VPL; j++)
            if (col_ok[j]) {
                float* d4 = dst + (j * 8 + lane) * 4;
                d4[0] = o[i][j].x; d4[1] = o[i][j].y; d4[2] = o[i][j].z; d4[3] = o[i][j].w;
            }
        if (lane == 0) {
            dst[D] = m[i];
            dst[D + 1] = l[i];
        }
    }
};

// One output element of row ir of the CTA's block: column d of what the wpg warps of its row group left in mrg.
template <int RT>
__device__ __forceinline__ void merge_warps(const float* mrg, uint32_t ir, uint32_t d, uint32_t D, uint32_t rgp, uint32_t wpg, float& M, float& L, float& acc) {
    const uint32_t rgi = ir / RT, ii = ir % RT, MS = D + 2u;
    M = ATT_NEG;
    for (uint32_t w = 0; w < wpg; w++) M = fmaxf(M, mrg[((size_t)(w * rgp + rgi) * RT + ii) * MS + D]);
    L = 0.0f;
    acc = 0.0f;
    for (uint32_t w = 0; w < wpg; w++) {
        const float* src = mrg + ((size_t)(w * rgp + rgi) * RT + ii) * MS;
        const float wgt = ex2(src[D] - M);
        L = fmaf(src[D + 1], wgt, L);
        acc = fmaf(src[d], wgt, acc);
    }
}

// The producer's page numbers: lane i holds the table's entries of pages base + i and base + 32 + i of a sequence, and of page i of
// the piece that comes next, so that no entry is waited for (read one chunk ahead, with the memory busy, they came later than the
// ring had room: 16 sequences of 4096 keys, 16-token pages, 113 us a step against 101).
struct Pages {
    uint32_t b, base;
    int32_t cur, ahead, next;
    __device__ __forceinline__ int32_t ask(const AttnParams& p, uint32_t seq, uint32_t page, uint32_t keys) const {
        if (page >= p.max_blocks_per_seq || page * p.block_size >= keys) return 0;
        return p.block_tables[(size_t)seq * p.max_blocks_per_seq + page];
    }
    // pages from `page` on of a sequence of so many keys, asked for earlier
    __device__ __forceinline__ void begin(const AttnParams& p, uint32_t seq, uint32_t page, uint32_t keys, int lane) {
        b = seq;
        base = page;
        cur = next;
        ahead = ask(p, b, base + 32u + lane, keys);
    }
    // keys [t0, t0 + nk): one copy per page the chunk touches; lane i takes the i-th page
    __device__ __forceinline__ void copy(const AttnParams& p, uint32_t g, uint32_t t0, uint32_t nk, uint32_t keys, float* ks, float* vs, uint32_t bar, int lane) {
        const uint32_t first = t0 / p.block_size;
        if (first >= base + 32u) {
            base += 32u;
            cur = ahead;
            ahead = ask(p, b, base + 32u + lane, keys);
        }
        const uint32_t blk = first + (uint32_t)lane, i = blk - base;
        const int32_t lo = __shfl_sync(0xffffffffu, cur, i & 31u), hi = __shfl_sync(0xffffffffu, ahead, i & 31u);
        int32_t entry = i < 32u ? lo : hi;
        if (blk <= (t0 + nk - 1u) / p.block_size) {
            const uint32_t ta = max(t0, blk * p.block_size), tb = min(t0 + nk, (blk + 1u) * p.block_size);
            if ((uint32_t)entry >= p.num_blocks) {
                entry = 0;
                if (p.status) atomicOr(p.status, ATT_STATUS_BLOCK);
            }
            const size_t off = (((size_t)entry * p.kv_heads + g) * p.block_size + (ta - blk * p.block_size)) * p.head_dim;
            bulk_g2s(smem_u32(ks + (size_t)(ta - t0) * p.head_dim), p.k + off, (tb - ta) * p.head_dim * 4u, bar);
            bulk_g2s(smem_u32(vs + (size_t)(ta - t0) * p.head_dim), p.v + off, (tb - ta) * p.head_dim * 4u, bar);
        }
    }
};

// A bounded wait gave up: report it and give copies still in flight time to land in this CTA's shared memory before it
// is released.
__device__ __forceinline__ void report_abort(const AttnParams& p) {
    if (threadIdx.x == 0 && p.status) atomicOr(p.status, ATT_STATUS_WAIT);
    for (int i = 0; i < 64; i++) __nanosleep(1000);
    __syncthreads();
}

// One CTA per slice of the keys of (sequence, KV head, block of rows).
// GATED: unless the cache is ragged; then lux_attn_even_f32, launched beside it, does all.
template <int VPL, int RT, bool FULL, bool GATED>
__global__ void __launch_bounds__(ATT_THREADS, ATT_CTAS_PER_SM) lux_attn_stream_f32(const AttnParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    const uint32_t bar_full = smem_u32(smem);
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + 16 * ATT_MAX_STAGES);
    int32_t* table = reinterpret_cast<int32_t*>(smem + ATT_HEADER);
    float* stages = reinterpret_cast<float*>(smem + ATT_HEADER + (p.block_size ? ATT_TABLE * 4 : 0));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t D = p.head_dim, NS = p.stages;
    const size_t stage_floats = (size_t)2 * ATT_CK * D;

    pdl_launch_dependents();                   // the merge kernel may take its place; it waits for this grid
    pdl_wait();                                // q, the cache and the tables may come from the kernels just before

    if (GATED && ragged(p, all_chunks(p))) return;
    uint32_t idx = blockIdx.x;
    const uint32_t split = idx % p.nsplit; idx /= p.nsplit;
    if (GATED && split == 0u && tid == 0) p.spans[idx] = AttnSpan{0, p.nsplit == 1 ? 1 : 0};
    const uint32_t rb = idx % p.row_blocks; idx /= p.row_blocks;
    const uint32_t g = idx % p.kv_heads, b = idx / p.kv_heads;

    uint32_t kv_len = p.kv_len;
    if (p.block_size) {
        const int32_t cl = p.context_lens[b];
        if (cl <= 0) return;                   // paged.wgsl:66-67: the rows stay as they are
        kv_len = min((uint32_t)cl, p.max_blocks_per_seq * p.block_size);
    }
    // rows of this CTA: row r of the KV head is (query qi = r / group, head g * group + r % group),
    // so a block of rows holds neighbouring queries and a causal block stops at its last row's keys
    const uint32_t R = p.group * p.seq_q, rpb = RT * p.rgp, row0 = rb * rpb;
    const uint32_t last_row = min(R, row0 + rpb) - 1u;
    const uint32_t lmax = row_len(p, last_row / p.group, kv_len);
    const uint32_t k_begin = split * p.split_keys;
    const uint32_t k_end = min(lmax, k_begin + p.split_keys);
    const uint32_t nchunks = k_end > k_begin ? (k_end - k_begin + ATT_CK - 1) / ATT_CK : 0u;
    const uint32_t tbl0 = p.block_size ? k_begin / p.block_size : 0u;
    // Every CTA walks its chunks from a different starting point (and wraps around), so that the CTAs
    // of a wave, which start together and advance at the same pace, are not all at the same offset
    // of equally spaced slices.
    const uint32_t rot = nchunks ? (blockIdx.x * 2654435761u >> 8) % nchunks : 0u;
    auto chunk_at = [&](uint32_t c) { const uint32_t cc = c + rot; return cc >= nchunks ? cc - nchunks : cc; };

    if (tid == 0) {
        *abort_flag = 0u;
        for (uint32_t s = 0; s < NS; s++) {
            mbar_init(bar_full + 8u * s, 1u);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (p.block_size && nchunks) {
        const uint32_t nblk = (k_end - 1u) / p.block_size - tbl0 + 1u;      // <= ATT_TABLE by the launcher's split
        const int32_t* src = p.block_tables + (size_t)b * p.max_blocks_per_seq + tbl0;
        for (uint32_t i = tid; i < nblk; i += ATT_THREADS) {
            int32_t e = src[i];
            if ((uint32_t)e >= p.num_blocks) {
                e = 0;
                if (p.status) atomicOr(p.status, ATT_STATUS_BLOCK);
            }
            table[i] = e;
        }
    }
    __syncthreads();

    // per-lane state of the consumer warps (the producer warp carries it unused)
    const int sub = lane & 7, kg = lane >> 3;
    float4 q[RT][VPL], o[RT][VPL];
    float m[RT], l[RT];
    uint32_t len[RT];
    bool col_ok[VPL];
#pragma unroll
    for (int j = 0; j < VPL; j++) col_ok[j] = (uint32_t)(j * 8 + sub) * 4u < D;

    if (warp == ATT_CW) {
        // ---- producer: one chunk = keys [t0, t0 + nk) of K and of V ------------------------------
        for (uint32_t c = 0; c < nchunks; c++) {
            const uint32_t s = c % NS;
            if (c >= NS) {
                named_bar_sync<ATT_BAR_FREE0>(s, ATT_THREADS);          // all consumer warps have left the stage
                if (*abort_flag) break;
            }
            const uint32_t t0 = k_begin + chunk_at(c) * ATT_CK, nk = min((uint32_t)ATT_CK, k_end - t0);
            const uint32_t bar = bar_full + 8u * s;
            float* ks = stages + s * stage_floats;
            float* vs = ks + (size_t)ATT_CK * D;
            if (lane == 0) mbar_expect_tx(bar, 2u * nk * D * 4u);
            __syncwarp();
            if (!p.block_size) {
                if (lane == 0) {
                    const size_t off = (((size_t)b * p.kv_heads + g) * p.kv_stride + t0) * D;
                    bulk_g2s(smem_u32(ks), p.k + off, nk * D * 4u, bar);
                    bulk_g2s(smem_u32(vs), p.v + off, nk * D * 4u, bar);
                }
            } else {
                // one copy per page the chunk touches; lane i takes the i-th page
                const uint32_t blk = t0 / p.block_size + (uint32_t)lane;
                const uint32_t ta = max(t0, blk * p.block_size), tb = min(t0 + nk, (blk + 1u) * p.block_size);
                if (ta < tb) {
                    const size_t off = (((size_t)table[blk - tbl0] * p.kv_heads + g) * p.block_size + (ta - blk * p.block_size)) * D;
                    bulk_g2s(smem_u32(ks + (size_t)(ta - t0) * D), p.k + off, (tb - ta) * D * 4u, bar);
                    bulk_g2s(smem_u32(vs + (size_t)(ta - t0) * D), p.v + off, (tb - ta) * D * 4u, bar);
                }
            }
        }
    } else {
        // ---- consumers -------------------------------------------------------------------------
        const uint32_t rg = (uint32_t)warp % p.rgp, kslot = (uint32_t)warp / p.rgp, wpg = ATT_CW / p.rgp;
#pragma unroll
        for (int i = 0; i < RT; i++) {
            const uint32_t r = row0 + rg * RT + i;
            const bool valid = r < R;
            const uint32_t qi = valid ? r / p.group : 0u, head = g * p.group + (valid ? r % p.group : 0u);
            len[i] = valid ? row_len(p, qi, kv_len) : 0xffffffffu;       // a padding row: q = 0, never written, never masks a chunk
            const float* qr = p.q + (((size_t)b * p.heads + head) * p.seq_q + qi) * D;
            m[i] = ATT_NEG;
            l[i] = 0.0f;
#pragma unroll
            for (int j = 0; j < VPL; j++) {
                float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
                if (valid && col_ok[j]) t = __ldg(reinterpret_cast<const float4*>(qr) + j * 8 + sub);
                q[i][j] = make_float4(t.x * p.qscale, t.y * p.qscale, t.z * p.qscale, t.w * p.qscale);
                o[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        // One step: the warp's four keys (one per group of 8 lanes) against its RT rows.  The
        // running maximum of a lane is only raised when a score passes it by more than 8 (in the
        // base-2 domain), so weights stay below 2^8 and the common step has no rescaling in it:
        // scores, one exp2 per row, the weighted sum.  MASKED steps (the last chunk of a slice, a
        // causal edge) check each key against the chunk and each row's length.
        const uint32_t row_bytes = D * 4u, lane_off = (uint32_t)sub * 16u;
        auto lds4 = [](uint32_t addr) {
            float4 r;
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "r"(addr));
            return r;
        };
        auto step = [&](auto masked, uint32_t kaddr, uint32_t vaddr, bool inb, uint32_t t) {
            constexpr bool MASKED = decltype(masked)::value;
            float sc[RT];
#pragma unroll
            for (int i = 0; i < RT; i++) sc[i] = 0.0f;
#pragma unroll
            for (int j = 0; j < VPL; j++) {
                float4 kk = make_float4(0.f, 0.f, 0.f, 0.f);
                if ((FULL || col_ok[j]) && (!MASKED || inb)) kk = lds4(kaddr + (uint32_t)j * 128u);
#pragma unroll
                for (int i = 0; i < RT; i++)
                    sc[i] = fmaf(q[i][j].x, kk.x, fmaf(q[i][j].y, kk.y, fmaf(q[i][j].z, kk.z, fmaf(q[i][j].w, kk.w, sc[i]))));
            }
#pragma unroll
            for (int i = 0; i < RT; i++) {
                sc[i] += __shfl_xor_sync(0xffffffffu, sc[i], 1);
                sc[i] += __shfl_xor_sync(0xffffffffu, sc[i], 2);
                sc[i] += __shfl_xor_sync(0xffffffffu, sc[i], 4);
            }
            bool vis[RT], up = false, any = false;
#pragma unroll
            for (int i = 0; i < RT; i++) {
                vis[i] = !MASKED || (inb && t < len[i]);
                up |= vis[i] && sc[i] > m[i] + 8.0f;
                any |= vis[i];
            }
            if (__any_sync(0xffffffffu, up)) {
#pragma unroll
                for (int i = 0; i < RT; i++) {
                    const float mn = vis[i] ? fmaxf(m[i], sc[i]) : m[i];
                    const float alpha = ex2(m[i] - mn);
                    l[i] *= alpha;
#pragma unroll
                    for (int j = 0; j < VPL; j++) {
                        o[i][j].x *= alpha; o[i][j].y *= alpha; o[i][j].z *= alpha; o[i][j].w *= alpha;
                    }
                    m[i] = mn;
                }
            }
            float pw[RT];
#pragma unroll
            for (int i = 0; i < RT; i++) {
                pw[i] = ex2(sc[i] - m[i]);
                if (MASKED && !vis[i]) pw[i] = 0.0f;
                l[i] += pw[i];
            }
            if (!MASKED || any) {
#pragma unroll
                for (int j = 0; j < VPL; j++) {
                    float4 vv = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (FULL || col_ok[j]) vv = lds4(vaddr + (uint32_t)j * 128u);
#pragma unroll
                    for (int i = 0; i < RT; i++) {
                        o[i][j].x = fmaf(pw[i], vv.x, o[i][j].x);
                        o[i][j].y = fmaf(pw[i], vv.y, o[i][j].y);
                        o[i][j].z = fmaf(pw[i], vv.z, o[i][j].z);
                        o[i][j].w = fmaf(pw[i], vv.w, o[i][j].w);
                    }
                }
            }
        };
        uint32_t min_len = 0xffffffffu;
#pragma unroll
        for (int i = 0; i < RT; i++) min_len = min(min_len, len[i]);
        const uint32_t stage0 = smem_u32(stages), stage_bytes = 2u * ATT_CK * row_bytes, v_off = ATT_CK * row_bytes;
        for (uint32_t c = 0; c < nchunks; c++) {
            const uint32_t s = c % NS;
            // one poller per CTA: warp 0 waits for the copies, the named barrier releases the other seven
            if (warp == 0) warp_wait(bar_full + 8u * s, (c / NS) & 1u, abort_flag, lane);
            named_bar_sync_c<ATT_BAR_READY>(ATT_CW * 32);
            if (*abort_flag) {
                // the producer may be parked on the stages this warp would still have released
                for (uint32_t cc = c; cc < c + NS && cc + NS < nchunks; cc++) named_bar_arrive<ATT_BAR_FREE0>(cc % NS, ATT_THREADS);
                break;
            }
            const uint32_t t0 = k_begin + chunk_at(c) * ATT_CK, nk = min((uint32_t)ATT_CK, k_end - t0);
            const uint32_t kchunk = stage0 + s * stage_bytes + lane_off;
            if (nk == ATT_CK && t0 + ATT_CK <= min_len) {
                for (uint32_t kb = kslot * 4u; kb < ATT_CK; kb += wpg * 4u) {
                    const uint32_t ka = kchunk + (kb + (uint32_t)kg) * row_bytes;
                    step(std::false_type{}, ka, ka + v_off, true, 0u);
                }
            } else {
                for (uint32_t kb = kslot * 4u; kb < nk; kb += wpg * 4u) {
                    const uint32_t key = kb + (uint32_t)kg, ka = kchunk + key * row_bytes;
                    step(std::true_type{}, ka, ka + v_off, key < nk, t0 + key);
                }
            }
            // done with the stage (not needed for the last NS chunks: nobody refills them)
            if (c + NS < nchunks) named_bar_arrive<ATT_BAR_FREE0>(s, ATT_THREADS);
        }
        // the four key slots of the warp, merged by the running-maximum rule
#pragma unroll
        for (int i = 0; i < RT; i++) {
            float mm = fmaxf(m[i], __shfl_xor_sync(0xffffffffu, m[i], 8));
            mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, 16));
            const float alpha = ex2(m[i] - mm);
            m[i] = mm;
            l[i] *= alpha;
            l[i] += __shfl_xor_sync(0xffffffffu, l[i], 8);
            l[i] += __shfl_xor_sync(0xffffffffu, l[i], 16);
#pragma unroll
            for (int j = 0; j < VPL; j++) {
                float* e = reinterpret_cast<float*>(&o[i][j]);
#pragma unroll
                for (int x = 0; x < 4; x++) {
                    float val = e[x] * alpha;
                    val += __shfl_xor_sync(0xffffffffu, val, 8);
                    val += __shfl_xor_sync(0xffffffffu, val, 16);
                    e[x] = val;
                }
            }
        }
    }

    __syncthreads();               // every chunk has landed and been read: the ring is free
    if (*abort_flag) {
        // A bounded wait gave up: report it and give copies still in flight time to land in this
        // CTA's shared memory before it is released.  Nothing is written.
        if (tid == 0 && p.status) atomicOr(p.status, ATT_STATUS_WAIT);
        for (int i = 0; i < 64; i++) __nanosleep(1000);
        __syncthreads();
        return;
    }
    // warps of one row group -> shared memory (over the ring), then one thread per output element
    float* mrg = stages;                                   // [warp][RT][D + 2]
    const uint32_t MS = D + 2u;
    if (warp < ATT_CW && kg == 0) {
#pragma unroll
        for (int i = 0; i < RT; i++) {
            float* dst = mrg + ((size_t)warp * RT + i) * MS;
#pragma unroll
            for (int j = 0; j < VPL; j++)
                if (col_ok[j]) {
                    // D + 2 floats per row: rows are 8-byte aligned, not 16
                    float* d4 = dst + (j * 8 + sub) * 4;
                    d4[0] = o[i][j].x; d4[1] = o[i][j].y; d4[2] = o[i][j].z; d4[3] = o[i][j].w;
                }
            if (sub == 0) {
                dst[D] = m[i];
                dst[D + 1] = l[i];
            }
        }
    }
    __syncthreads();
    const uint32_t wpg = ATT_CW / p.rgp;
    for (uint32_t e = tid; e < rpb * D; e += ATT_THREADS) {
        const uint32_t ir = e / D, d = e - ir * D, r = row0 + ir;
        if (r >= R) continue;
        const uint32_t rgi = ir / RT, ii = ir % RT;
        float M = ATT_NEG;
        for (uint32_t w = 0; w < wpg; w++) M = fmaxf(M, mrg[((size_t)(w * p.rgp + rgi) * RT + ii) * MS + D]);
        float L = 0.0f, acc = 0.0f;
        for (uint32_t w = 0; w < wpg; w++) {
            const float* src = mrg + ((size_t)(w * p.rgp + rgi) * RT + ii) * MS;
            const float wgt = ex2(src[D] - M);
            L = fmaf(src[D + 1], wgt, L);
            acc = fmaf(src[d], wgt, acc);
        }
        const uint32_t qi = r / p.group, head = g * p.group + r % p.group;
        const size_t orow = ((size_t)b * p.heads + head) * p.seq_q + qi;
        if (p.nsplit == 1) {
            p.out[orow * D + d] = L > 0.0f ? acc / L : 0.0f;
            if (d == 0 && p.lse) p.lse[orow] = L > 0.0f ? fmaf(M, ATT_LN2, logf(L)) : -3.402823e+38f;
        } else {
            float* dst = p.part + (orow * p.nsplit + split) * MS;
            dst[d] = acc;
            if (d == 0) {
                dst[D] = M;
                dst[D + 1] = L;
            }
        }
    }
}

// What a CTA of the even form does next: chunks [lo, hi) of the n of (sequence b, KV head g).
struct Piece {
    uint32_t b, g, keys, lo, hi, n;
    uint32_t ahead;              // keys of the next sequence, asked for early
    __device__ __forceinline__ void load(const volatile Piece* s) {
        b = s->b; g = s->g; keys = s->keys; lo = s->lo; hi = s->hi; n = s->n; ahead = s->ahead;
    }
};

// A decode step over a paged cache, dealt out evenly: all 32-key chunks of all (sequence, KV head) items, one after the other,
// each CTA taking the next so many of them.
template <int VPL, int RT, bool FULL>
__global__ void __launch_bounds__(ATT_THREADS, ATT_CTAS_PER_SM) lux_attn_even_f32(const AttnParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    const uint32_t bar_full = smem_u32(smem);
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + 16 * ATT_MAX_STAGES);
    float* mrg = reinterpret_cast<float*>(smem + ATT_EVEN_HEADER);         // [warp][RT][D + 2]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t D = p.head_dim, NS = p.stages, MS = D + 2u;
    float* stages = mrg + att_merge_floats(D, RT);
    const size_t stage_floats = (size_t)2 * ATT_CK * D;

    pdl_launch_dependents();                   // the merge kernel may take its place; it waits for this grid
    pdl_wait();                                // q, the cache and the tables may come from the kernels just before

    const uint32_t R = p.group, rpb = RT * p.rgp;        // rows: the heads of a KV head
    const uint32_t all = all_chunks(p);
    if (!ragged(p, all)) return;
    // every warp for itself, 32 sequences at a time: the sequence in which this CTA starts
    const uint32_t share = max(p.share, (all + gridDim.x - 1u) / gridDim.x), at = blockIdx.x * share;
    if (at >= all) return;
    Piece first;
    uint32_t before = 0u;
    for (uint32_t b0 = 0;; b0 += 32) {
        const uint32_t n = b0 + lane < p.batch ? chunks_of(paged_len(p, b0 + lane)) : 0u;
        uint32_t upto = n;                     // inclusive
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, upto, off);
            if (lane >= off) upto += v;
        }
        const uint32_t hit = __ballot_sync(0xffffffffu, (before + upto) * p.kv_heads > at);
        if (hit) {
            const int src = __ffs(hit) - 1;
            first.b = b0 + src;
            before += __shfl_sync(0xffffffffu, upto - n, src);
            break;
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
    }
    first.keys = paged_len(p, first.b);
    first.n = chunks_of(first.keys);
    first.ahead = first.b + 1u < p.batch ? paged_len(p, first.b + 1u) : 0u;
    const uint32_t in = at - before * p.kv_heads;
    first.g = in / first.n;
    first.lo = in - first.g * first.n;
    const uint32_t total = min(share, all - at);         // chunks of this CTA
    first.hi = min(first.lo + total, first.n);
    auto next = [&](Piece& w, uint32_t left) { // the piece after w, `left` chunks still to do
        if (++w.g == p.kv_heads) {
            w.g = 0u;
            w.keys = w.ahead;
            for (w.b++; w.keys == 0u && w.b + 1u < p.batch;) w.keys = paged_len(p, ++w.b);     // (left > 0: there is one)
            w.n = chunks_of(w.keys);
            w.ahead = w.b + 1u < p.batch ? paged_len(p, w.b + 1u) : 0u;
        }
        w.lo = 0u;
        w.hi = min(left, w.n);
    };

    if (tid == 0) {
        *abort_flag = 0u;
        for (uint32_t s = 0; s < NS; s++) {
            mbar_init(bar_full + 8u * s, 1u);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp == ATT_CW) {
        // ---- producer: one chunk = keys [t0, t0 + nk) of K and of V ------------------------------
        Pages pages;
        Piece w = first, then = first;         // the piece at hand, the one after it
        uint32_t c = 0;
        pages.next = pages.ask(p, w.b, w.lo * ATT_CK / p.block_size + lane, w.keys);
        for (;;) {
            const uint32_t end = c + (w.hi - w.lo);
            pages.begin(p, w.b, w.lo * ATT_CK / p.block_size, w.keys, lane);
            if (end < total) {
                next(then, total - end);
                pages.next = pages.ask(p, then.b, lane, then.keys);
            }
            for (uint32_t t0 = w.lo * ATT_CK; c < end; c++, t0 += ATT_CK) {
                const uint32_t s = c % NS, nk = min((uint32_t)ATT_CK, w.keys - t0), bar = bar_full + 8u * s;
                if (c >= NS) {
                    named_bar_sync<ATT_BAR_FREE0>(s, ATT_THREADS);      // all consumer warps have left the stage
                    if (*abort_flag) break;
                }
                float* ks = stages + s * stage_floats;
                if (lane == 0) mbar_expect_tx(bar, 2u * nk * D * 4u);
                __syncwarp();
                pages.copy(p, w.g, t0, nk, w.keys, ks, ks + (size_t)ATT_CK * D, bar, lane);
            }
            if (c < end || c == total) break;
            w = then;
        }
    } else {
        // ---- consumers -------------------------------------------------------------------------
        const uint32_t rg = (uint32_t)warp % p.rgp, kslot = (uint32_t)warp / p.rgp, wpg = ATT_CW / p.rgp;
        Rows<VPL, RT, FULL> rows;
        rows.columns(D, lane & 7);
        const uint32_t row_bytes = D * 4u, lane_off = (uint32_t)(lane & 7) * 16u;
        const uint32_t stage0 = smem_u32(stages), stage_bytes = 2u * ATT_CK * row_bytes, v_off = ATT_CK * row_bytes;
        uint32_t c = 0;
        auto walk = [&](const Piece& w) {                                // the chunks of a piece; false: a wait gave up
            const uint32_t t_end = min(w.hi * ATT_CK, w.keys);
            uint32_t t0 = w.lo * ATT_CK;
            for (const uint32_t c_end = c + (w.hi - w.lo); c < c_end; c++) {
                const uint32_t s = c % NS;
                // one poller per CTA: warp 0 waits for the copies, the named barrier releases the other seven
                if (warp == 0) warp_wait(bar_full + 8u * s, (c / NS) & 1u, abort_flag, lane);
                named_bar_sync_c<ATT_BAR_READY>(ATT_CW * 32);
                if (*abort_flag) {
                    // the producer may be parked on the stages this warp would still have released
                    for (uint32_t cc = c; cc < c + NS && cc + NS < total; cc++) named_bar_arrive<ATT_BAR_FREE0>(cc % NS, ATT_THREADS);
                    return false;
                }
                rows.chunk(stage0 + s * stage_bytes + lane_off, v_off, row_bytes, t0, min((uint32_t)ATT_CK, t_end - t0), kslot, wpg, lane >> 3);
                // done with the stage (not needed for the last NS chunks: nobody refills them)
                if (c + NS < total) named_bar_arrive<ATT_BAR_FREE0>(s, ATT_THREADS);
                t0 += ATT_CK;
            }
            return true;
        };
        // the end of a piece: the warps of each row group are merged and the rows written: the outputs of a whole item, else
        // partial results
        auto finish = [&](const Piece& w) {
#pragma unroll
            for (int i = 0; i < RT; i++) {
                rows.fold(i);
                rows.store(i, mrg + ((size_t)warp * RT + i) * MS, D, lane);
            }
            named_bar_sync_c<ATT_BAR_MERGE>(ATT_CW * 32);
            const bool whole = w.lo == 0u && w.hi == w.n;
            if (w.lo == 0u && tid == 0)                                  // the item may go on in the CTAs after this one
                p.spans[w.b * p.kv_heads + w.g] = AttnSpan{(int32_t)blockIdx.x, (int32_t)(1u + (w.n - w.hi + share - 1u) / share)};
            for (uint32_t e = tid; e < rpb * D; e += ATT_CW * 32) {
                const uint32_t ir = e / D, d = e - ir * D;
                if (ir >= R) continue;
                float M, L, acc;
                merge_warps<RT>(mrg, ir, d, D, p.rgp, wpg, M, L, acc);
                const size_t orow = (size_t)w.b * p.heads + w.g * p.group + ir;
                if (whole) {
                    p.out[orow * D + d] = L > 0.0f ? acc / L : 0.0f;
                } else {
                    float* dst = p.part + ((size_t)(blockIdx.x * 2u + (w.lo == 0u ? 1u : 0u)) * rpb + ir) * MS;
                    dst[d] = acc;
                    if (d == 0) {
                        dst[D] = M;
                        dst[D + 1] = L;
                    }
                }
            }
            named_bar_sync_c<ATT_BAR_MERGE>(ATT_CW * 32);                // before the next piece is merged
        };
        // the piece lies in shared memory while its chunks are worked on: the loop has no registers left for it
        Piece* const kept = reinterpret_cast<Piece*>(smem + ATT_HEADER) + warp;
        Piece w = first;
        for (;;) {
            rows.begin(p, w.b, w.g, rg * RT, w.keys, lane & 7);
            if (lane == 0) *kept = w;
            __syncwarp();
            if (!walk(w)) break;
            w.load(kept);
            finish(w);
            if (c == total) break;
            next(w, total - c);
            __syncwarp();
        }
    }

    __syncthreads();               // every chunk has landed and been read
    if (*abort_flag) report_abort(p);          // the piece it was in is not written, nor what comes after it
}

// Merge of the key slices of one output row (paged_attention_v2_reduce, paged.wgsl:351-405, with
// the statistics in the base-2 domain).  One CTA per row; resident early, it waits for the slices.
__global__ void __launch_bounds__(128) lux_attn_merge_f32(const float* __restrict__ part, float* __restrict__ out, float* __restrict__ lse,
                                                          const int32_t* __restrict__ context_lens, uint32_t rows_per_seq,
                                                          uint32_t nsplit, uint32_t D) {
    __shared__ float wgt[256];
    __shared__ float stat[2];
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t row = blockIdx.x, MS = D + 2u;
    if (context_lens && context_lens[row / rows_per_seq] <= 0) return;
    const float* base = part + (size_t)row * nsplit * MS;
    if (threadIdx.x < 32) {
        float M = ATT_NEG;
        for (uint32_t s = threadIdx.x; s < nsplit; s += 32) M = fmaxf(M, base[(size_t)s * MS + D]);
        for (int off = 16; off; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
        float L = 0.0f;
        for (uint32_t s = threadIdx.x; s < nsplit; s += 32) {
            const float w = exp2f(base[(size_t)s * MS + D] - M);
            wgt[s] = w;
            L = fmaf(base[(size_t)s * MS + D + 1], w, L);
        }
        for (int off = 16; off; off >>= 1) L += __shfl_xor_sync(0xffffffffu, L, off);
        if (threadIdx.x == 0) {
            stat[0] = M;
            stat[1] = L;
        }
    }
    __syncthreads();
    const float L = stat[1], inv = L > 0.0f ? 1.0f / L : 0.0f;
    for (uint32_t d = threadIdx.x; d < D; d += blockDim.x) {
        float acc = 0.0f;
        for (uint32_t s = 0; s < nsplit; s++) acc = fmaf(base[(size_t)s * MS + d], wgt[s], acc);
        out[(size_t)row * D + d] = acc * inv;
    }
    if (threadIdx.x == 0 && lse) lse[row] = L > 0.0f ? fmaf(stat[0], ATT_LN2, logf(L)) : -3.402823e+38f;
}

// The same for a paged cache that may have been dealt out in even shares: slices, what several CTAs did of a row, or nothing to do.
__global__ void __launch_bounds__(128) lux_attn_merge_even_f32(const AttnParams p) {
    __shared__ float wgt[ATT_MAX_PARTS];
    __shared__ float denominator;
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t row = blockIdx.x, D = p.head_dim, MS = D + 2u, b = row / p.heads, head = row - b * p.heads;
    if (p.context_lens[b] <= 0) return;
    const AttnSpan span = p.spans[b * p.kv_heads + head / p.group];
    if (span.ctas == 1) return;                        // one CTA saw all of it and wrote the row
    // partial result 0, partial result 1 and the step from it to each of the others
    const float *base0 = p.part + (size_t)row * p.nsplit * MS, *base1 = base0 + MS;
    size_t step = MS;
    uint32_t parts = p.nsplit;
    if (span.ctas != 0) {
        if (!span_fits(span, p.ctas)) {                // never written: a wait gave up in the CTA in which the item begins
            if (threadIdx.x == 0 && p.status) atomicOr(p.status, ATT_STATUS_WAIT);
            return;
        }
        const uint32_t ir = head % p.group;
        base0 = p.part + ((size_t)span_place(span, 0) * p.rpb + ir) * MS;
        base1 = p.part + ((size_t)span_place(span, 1) * p.rpb + ir) * MS;
        step = (size_t)2 * p.rpb * MS;
        parts = (uint32_t)span.ctas;
    }
    auto part = [&](uint32_t s) { return s == 0 ? base0 : base1 + (size_t)(s - 1u) * step; };
    if (threadIdx.x < 32) {
        float M = ATT_NEG;
        for (uint32_t s = threadIdx.x; s < parts; s += 32) M = fmaxf(M, part(s)[D]);
        for (int off = 16; off; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
        float L = 0.0f;
        for (uint32_t s = threadIdx.x; s < parts; s += 32) {
            const float w = exp2f(part(s)[D] - M);
            wgt[s] = w;
            L = fmaf(part(s)[D + 1], w, L);
        }
        for (int off = 16; off; off >>= 1) L += __shfl_xor_sync(0xffffffffu, L, off);
        if (threadIdx.x == 0) denominator = L;
    }
    __syncthreads();
    const float L = denominator, inv = L > 0.0f ? 1.0f / L : 0.0f;
    for (uint32_t d = threadIdx.x; d < D; d += blockDim.x) {
        float acc = 0.0f;
        for (uint32_t s = 0; s < parts; s++) acc = fmaf(part(s)[d], wgt[s], acc);
        p.out[(size_t)row * D + d] = acc * inv;
    }
}

// Any head_dim, any alignment: one CTA per output row, 256 keys per step (a thread per key for the
// scores, a thread per output dimension for the weighted sum), the same running-maximum rule.
__device__ __forceinline__ const float* plain_row(const AttnParams& p, const float* base, uint32_t b, uint32_t g, uint32_t t,
                                                  const int32_t* table) {
    if (!p.block_size) return base + (((size_t)b * p.kv_heads + g) * p.kv_stride + t) * p.head_dim;
    int32_t e = table[t / p.block_size];
    if ((uint32_t)e >= p.num_blocks) e = 0;
    return base + (((size_t)e * p.kv_heads + g) * p.block_size + t % p.block_size) * p.head_dim;
}

__global__ void __launch_bounds__(256) lux_attn_plain_f32(const AttnParams p) {
    extern __shared__ float sm[];
    float* o = sm;                       // [head_dim]
    float* pw = sm + p.head_dim;         // [256]
    __shared__ float red[8];
    const uint32_t D = p.head_dim, tid = threadIdx.x;
    uint32_t idx = blockIdx.x;
    const uint32_t qi = idx % p.seq_q; idx /= p.seq_q;
    const uint32_t head = idx % p.heads, b = idx / p.heads, g = head / p.group;
    uint32_t kv_len = p.kv_len;
    const int32_t* table = nullptr;
    if (p.block_size) {
        const int32_t cl = p.context_lens[b];
        if (cl <= 0) return;
        kv_len = min((uint32_t)cl, p.max_blocks_per_seq * p.block_size);
        table = p.block_tables + (size_t)b * p.max_blocks_per_seq;
    }
    const uint32_t len = row_len(p, qi, kv_len);
    const size_t orow = ((size_t)b * p.heads + head) * p.seq_q + qi;
    const float* qr = p.q + orow * D;
    for (uint32_t d = tid; d < D; d += 256) o[d] = 0.0f;
    float m = ATT_NEG, l = 0.0f;
    for (uint32_t t0 = 0; t0 < len; t0 += 256) {
        const uint32_t t = t0 + tid;
        float s = ATT_NEG;
        if (t < len) {
            const float* kr = plain_row(p, p.k, b, g, t, table);
            float dot = 0.0f;
            for (uint32_t d = 0; d < D; d++) dot = fmaf(qr[d], kr[d], dot);
            s = dot * p.qscale;
        }
        float tm = s;
        for (int off = 16; off; off >>= 1) tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, off));
        if ((tid & 31) == 0) red[tid >> 5] = tm;
        __syncthreads();
        tm = red[0];
        for (int w = 1; w < 8; w++) tm = fmaxf(tm, red[w]);
        const float mn = fmaxf(m, tm), alpha = exp2f(m - mn);
        const float e = t < len ? exp2f(s - mn) : 0.0f;
        pw[tid] = e;
        float ts = e;
        for (int off = 16; off; off >>= 1) ts += __shfl_xor_sync(0xffffffffu, ts, off);
        __syncthreads();                                   // red[] read by everyone, pw[] written
        if ((tid & 31) == 0) red[tid >> 5] = ts;
        __syncthreads();
        ts = 0.0f;
        for (int w = 0; w < 8; w++) ts += red[w];
        l = fmaf(l, alpha, ts);
        m = mn;
        const uint32_t n = min(256u, len - t0);
        for (uint32_t d = tid; d < D; d += 256) {
            float acc = o[d] * alpha;
            for (uint32_t j = 0; j < n; j++) acc = fmaf(pw[j], plain_row(p, p.v, b, g, t0 + j, table)[d], acc);
            o[d] = acc;
        }
        __syncthreads();
    }
    for (uint32_t d = tid; d < D; d += 256) p.out[orow * D + d] = l > 0.0f ? o[d] / l : 0.0f;
    if (tid == 0 && p.lse) p.lse[orow] = l > 0.0f ? fmaf(m, ATT_LN2, logf(l)) : -3.402823e+38f;
}

// ---- rotary embedding ------------------------------------------------------------------------------

struct RopeParams {
    const float* x;
    float* out;
    const float* x2;               // second tensor of the fused q/k call (null otherwise), rotated in place
    float* out2;
    const float* cos_cache;
    const float* sin_cache;
    const uint32_t* position_ids;
    uint32_t* status;
    uint32_t batch, seq, heads, heads2, half;
    uint32_t position_offset, cache_positions, ntk, backward;
    float theta, head_dim_f;
};

// correctly rounded theta^(-2 i / head_dim) for all but a vanishing share of arguments: the f32
// exponent of the shader (rope.wgsl:56-60), the power in double, one rounding
__device__ __forceinline__ float rope_freq(uint32_t i, float head_dim_f, float theta) {
    const float exponent = __fdiv_rn(__fmul_rn(-2.0f, (float)i), head_dim_f);
    return (float)pow((double)theta, (double)exponent);
}

// I: the index type (32 bits wherever the call has fewer than 2^31 items: a 64-bit division is a subroutine,
// and three of them per pair took longer than the pair's 16 bytes).  V: pairs per thread; two where rows
// and views allow 16-byte accesses.  512 tokens x 32 heads x 128: 9.7 -> 6.9 us (17 MB).
template <typename I, int V>
__global__ void __launch_bounds__(256) lux_rope_f32(const RopeParams p) {
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t half = p.half / V;                      // items per head
    const I per_tok = (I)(p.heads + p.heads2) * half;
    const I total = (I)p.batch * p.seq * per_tok;
    for (I e = (I)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (I)gridDim.x * blockDim.x) {
        const I tok = e / per_tok;
        uint32_t rem = (uint32_t)(e - tok * per_tok);
        const uint32_t s = (uint32_t)(tok % p.seq);
        uint32_t position = p.position_ids ? p.position_ids[tok] : p.position_offset + s;
        if (p.ntk) position = s;                          // rope_ntk_scaled uses the index alone (rope.wgsl:337-339)
        const float* src = p.x;
        float* dst = p.out;
        uint32_t heads = p.heads;
        if (rem >= p.heads * half) {
            rem -= p.heads * half;
            src = p.x2;
            dst = p.out2;
            heads = p.heads2;
        }
        const uint32_t i = rem % half * V;                 // first pair of the head
        float c[V], sn[V];
        if (p.cos_cache) {
            if (position >= p.cache_positions) {
                if (p.status) atomicOr(p.status, ATT_STATUS_POSITION);
                continue;
            }
#pragma unroll
            for (int j = 0; j < V; j++) {
                c[j] = __ldg(p.cos_cache + (size_t)position * p.half + i + j);
                sn[j] = __ldg(p.sin_cache + (size_t)position * p.half + i + j);
            }
        } else {
#pragma unroll
            for (int j = 0; j < V; j++) {
                const float angle = __fmul_rn((float)position, rope_freq(i + j, p.head_dim_f, p.theta));
                c[j] = cosf(angle);
                sn[j] = sinf(angle);
            }
        }
        const size_t i0 = ((size_t)tok * heads) * (2 * (size_t)p.half) + (size_t)(2 * V) * rem;
        alignas(16) float x[2 * V], y[2 * V];
        if (V == 2) *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(src + i0);
        else *reinterpret_cast<float2*>(x) = *reinterpret_cast<const float2*>(src + i0);
#pragma unroll
        for (int j = 0; j < V; j++) {
            const float xx = x[2 * j], xy = x[2 * j + 1];
            if (!p.backward) {
                y[2 * j] = __fsub_rn(__fmul_rn(xx, c[j]), __fmul_rn(xy, sn[j]));
                y[2 * j + 1] = __fadd_rn(__fmul_rn(xx, sn[j]), __fmul_rn(xy, c[j]));
            } else {
                y[2 * j] = __fadd_rn(__fmul_rn(xx, c[j]), __fmul_rn(xy, sn[j]));
                y[2 * j + 1] = __fadd_rn(__fmul_rn(-xx, sn[j]), __fmul_rn(xy, c[j]));
            }
        }
        if (V == 2) *reinterpret_cast<float4*>(dst + i0) = *reinterpret_cast<const float4*>(y);
        else *reinterpret_cast<float2*>(dst + i0) = *reinterpret_cast<const float2*>(y);
    }
}

__global__ void __launch_bounds__(256) lux_rope_cache_f32(float* __restrict__ cos_out, float* __restrict__ sin_out, uint32_t max_seq_len,
                                                          uint32_t half, float head_dim_f, float theta) {
    const size_t total = (size_t)max_seq_len * half;
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const uint32_t pos = (uint32_t)(e / half), i = (uint32_t)(e % half);
        const float angle = __fmul_rn((float)pos, rope_freq(i, head_dim_f, theta));
        cos_out[e] = cosf(angle);
        sin_out[e] = sinf(angle);
    }
}

// update_kv_cache: one thread per V consecutive elements of a row (pairs of caches, same index arithmetic);
// V = 4 where rows and views allow 16-byte accesses, and the index type as in the rotation above
template <typename I, int V>
__global__ void __launch_bounds__(256) lux_kv_append_f32(const float* __restrict__ k, const float* __restrict__ v, float* __restrict__ k_cache,
                                                         float* __restrict__ v_cache, uint32_t bh, uint32_t seq_q, uint32_t cache_len,
                                                         uint32_t max_cache_len, uint32_t D) {
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t items = D / V;                          // per row
    const I total = (I)bh * seq_q * items;
    for (I e = (I)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (I)gridDim.x * blockDim.x) {
        const I t = e / items;
        const uint32_t d = (uint32_t)(e - t * items) * V;
        const I h = t / seq_q;
        const uint32_t s = (uint32_t)(t - h * seq_q);
        const uint64_t pos = (uint64_t)cache_len + s;
        if (pos >= max_cache_len) continue;                // cache overflow is dropped (:523-525)
        const size_t dst = ((size_t)h * max_cache_len + pos) * D + d, src = (size_t)e * V;
        if (V == 4) {
            *reinterpret_cast<float4*>(k_cache + dst) = *reinterpret_cast<const float4*>(k + src);
            *reinterpret_cast<float4*>(v_cache + dst) = *reinterpret_cast<const float4*>(v + src);
        } else {
            k_cache[dst] = k[src];
            v_cache[dst] = v[src];
        }
    }
}

// ---- host side -------------------------------------------------------------------------------------

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
uint32_t pow2ceil(uint32_t v) {
    uint32_t r = 1;
    while (r < v) r <<= 1;
    return r;
}

using AttnKernel = void (*)(const AttnParams);
enum Form { SLICES, SLICES_GATED, EVEN };
template <int VPL, int RT, bool FULL> AttnKernel decode_kernel(Form f) {
    return f == EVEN ? lux_attn_even_f32<VPL, RT, FULL> : f == SLICES_GATED ? lux_attn_stream_f32<VPL, RT, FULL, true> : lux_attn_stream_f32<VPL, RT, FULL, false>;
}
template <int VPL, int RT> AttnKernel decode_kernel(bool full, Form f) {
    return full ? decode_kernel<VPL, RT, true>(f) : decode_kernel<VPL, RT, false>(f);
}
// full: head_dim is exactly VPL * 32, so no lane has a column to skip
AttnKernel pick_kernel(int vpl, int rt, bool full, Form f) {
    switch (vpl * 10 + rt) {
        case 11: return decode_kernel<1, 1>(full, f); case 12: return decode_kernel<1, 2>(full, f);
        case 21: return decode_kernel<2, 1>(full, f); case 22: return decode_kernel<2, 2>(full, f);
        case 31: return decode_kernel<3, 1>(full, f); case 32: return decode_kernel<3, 2>(full, f);
        case 41: return decode_kernel<4, 1>(full, f); case 42: return decode_kernel<4, 2>(full, f);
        case 81: return decode_kernel<8, 1>(full, f);
    }
    return nullptr;
}

// What lux_attn_prefill_mma_f32 takes (q, k and v have been found aligned).
bool prefill_fits(const AttnParams& p) {
    return !p.block_size && p.head_dim == 128 && aligned16(p.out) && (uint64_t)p.batch * p.heads * ((p.seq_q + 127ull) / 128u) <= 0x7fffffffu;
}
// Which of the two kernels answers a call: by what the streaming kernel takes in us on 148 SMs and what the prompt kernel
// took when its products were mma.sync ones.  Over 178 shapes (64 .. 2049 queries, 64 .. 16384 keys, 4 .. 64 heads,
// batch 1 .. 8) that choice was nowhere slower than the streaming kernel by more than 3 %.  The prompt kernel has become two to
// five times faster since (attention_prefill_mma.cu), so it is the faster one wherever it is chosen (by this line / the streaming kernel,
// 32 heads, 8 KV heads, us: 256 queries over 4096 keys 156 / 858, over 131072 4294 / 26015) and also where it is not: 65 over 4096 151 / 236, 128
// over 131072 4249 / 13435.  The line has stayed, and with it which kernel, and so which order of sums, a call gets.
// The mma.sync form: a CTA per SM owned 128 queries of a head and walked all their keys, 5.5 us a tile of 32, 4.6 where half
// of its warps had no rows.
double prefill_us(const AttnParams& p, int sms) {
    double total = 0.0, longest = 0.0;
    uint64_t blocks = 0;
    for (uint64_t q0 = 0; q0 < p.seq_q; q0 += 128, blocks++) {
        const uint64_t rows = std::min<uint64_t>(128u, p.seq_q - q0);
        const uint64_t keys = p.causal ? std::min<uint64_t>(p.causal_base + q0 + rows, p.kv_len) : p.kv_len;
        const double us = (double)((keys + 31) / 32) * (rows > 64 ? 5.5 : 4.6);
        total += us;
        longest = std::max(longest, us);
    }
    const double bh = (double)p.batch * p.heads;
    return 6.0 + (blocks * bh <= sms ? longest : std::max(longest, total * bh / sms + longest / 4));
}
// The streaming kernel: two CTAs per SM, each 16 rows of a KV head against a slice of the keys, 0.115 us a key (0.6 of
// it where a CTA has its SM to itself) and a start-up of 32.
double stream_us(const AttnParams& p, uint32_t slices, uint32_t slice_keys, int sms) {
    // causal rows see one key more each until they see all
    const double climb = p.causal ? std::min<double>(p.seq_q, std::max(0.0, (double)p.kv_len - p.causal_base)) : 0.0;
    const double keys = (climb * (p.causal_base + (climb + 1) / 2) + (p.seq_q - climb) * p.kv_len) / p.seq_q;
    const double items = (double)p.batch * p.kv_heads * p.row_blocks, ctas = items * slices;
    const double longest = std::min<double>(slice_keys, p.kv_len) + 32.0, slots = 2.0 * sms;
    const double span = ctas <= slots ? longest * (0.6 + 0.4 * std::max(0.0, ctas - sms) / sms)
                                      : std::max(longest, items * (keys + slices * 32.0) / slots + longest / 2);
    return (slices > 1 ? 12.0 : 9.0) + 0.115 * span;      // launches (and the merge of slices)
}

// Fills the launch geometry of p and launches.  max_keys: the longest context any row can have.
LuxBackendError attn_launch(Context* ctx, AttnParams& p, uint32_t max_keys, uint32_t flags, const char* what) {
    cudaSetDevice(ctx->device);
    p.status = ctx->d_status;
    const uint32_t D = p.head_dim;
    const size_t out_rows = (size_t)p.batch * p.heads * p.seq_q;
    if (out_rows == 0) return LUX_BACKEND_OK;
    const bool stream_ok = D % 4 == 0 && D <= 256 && aligned16(p.q) && aligned16(p.k) && aligned16(p.v) && out_rows <= 0x7fffffffu;
    if (!stream_ok) {
        if (out_rows > 0x7fffffffu) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
        const size_t smem = ((size_t)D + 256) * 4;
        if (smem > 200u << 10) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
        if (smem > 48u << 10) cudaFuncSetAttribute(lux_attn_plain_f32, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        p.nsplit = 1;
        lux_attn_plain_f32<<<(unsigned)out_rows, 256, smem, ctx->stream>>>(p);
        count_launch("lux_attn_plain_f32");
        return finish_op(ctx, (flags & LUX_QMATMUL_FLAG_NO_SYNC) != 0, what);
    }
    int vpl = (int)((D + 31) / 32);
    if (vpl > 4) vpl = 8;
    const uint32_t R = p.group * p.seq_q;
    // two query rows per lane: more would halve the shared-memory reads per row, but the registers
    // of four rows leave one CTA of nine warps per SM, too few to hide the latency of each step
    // (measured: causal prefill of 2048 tokens, Llama-3-8B heads, 15.2 TFLOP/s against 20.4)
    const int rt = R >= 2 && vpl <= 4 ? 2 : 1;
    p.rgp = pow2ceil(std::min<uint32_t>((R + rt - 1) / rt, ATT_CW));
    const uint32_t rpb = rt * p.rgp;
    p.rpb = rpb;
    p.row_blocks = (R + rpb - 1) / rpb;
    const size_t items = (size_t)p.batch * p.kv_heads * p.row_blocks;
    // Slices of the keys.  CTAs run two per SM, so the grid should fill whole waves of 2 x SMs; a slice
    // costs a CTA start-up and a row in the merge, about as much as streaming 64 keys, and is at
    // least 128 keys long.  The block-table copy caps the pages a slice may span.
    auto geometry = [&](uint32_t want) {
        p.split_keys = std::max<uint32_t>(((max_keys + want - 1) / want + ATT_CK - 1) / ATT_CK * ATT_CK, ATT_CK);
        p.nsplit = std::max<uint32_t>((max_keys + p.split_keys - 1) / p.split_keys, 1u);
    };
    uint32_t min_split = 1;
    if (p.block_size) {
        // a slice (a multiple of the chunk) spans at most split_keys / block_size + 2 pages
        const uint64_t cap = (uint64_t)(ATT_TABLE - 2) * p.block_size / ATT_CK * ATT_CK;
        min_split = (uint32_t)std::max<uint64_t>((max_keys + cap - 1) / cap, 1);
    }
    uint32_t best = min_split;
    double best_score = -1.0;
    const uint32_t sm = (uint32_t)ctx->sm_count * ATT_CTAS_PER_SM;
    for (uint32_t n = min_split; n <= 256; n++) {
        geometry(n);
        if (p.nsplit != n) continue;                                   // rounding to chunks merged this count into a smaller one
        // (a decode step over up to 512 keys goes down to 64: a slice is then two chunks of the ring, and what counts
        // is how soon it ends: one sequence, Llama-3-8B heads, 300 keys, 10.4 -> 9.3 us a call; at 2000 keys slices
        // of 64 are 12.6 us against 11.5, and a prompt of 150 tokens, which fills the chip with its rows, 43 against 29)
        if (n > min_split && p.split_keys < (max_keys <= 512 && p.row_blocks == 1 ? 64u : 128u)) break;
        const double ctas = (double)items * n, waves = std::ceil(ctas / sm);
        const double score = ctas / (waves * sm) * p.split_keys / (p.split_keys + 64.0);
        if (score > best_score * 1.02) {                               // a larger count has to earn its merge
            best_score = score;
            best = n;
        }
        if (ctas > 8.0 * sm) break;
    }
    geometry(best);
    if (prefill_fits(p) && g_tune.attn_prefill != 2 && (g_tune.attn_prefill || (p.seq_q >= 64 && p.kv_len &&
        prefill_us(p, ctx->sm_count) < 0.97 * stream_us(p, p.nsplit, p.split_keys, ctx->sm_count)))) {
        PrefillArgs f{};
        f.q = p.q; f.k = p.k; f.v = p.v; f.out = p.out; f.lse = p.lse;
        f.status = p.status; f.status_wait = ATT_STATUS_WAIT;
        f.batch = p.batch; f.heads = p.heads; f.kv_heads = p.kv_heads; f.group = p.group; f.seq_q = p.seq_q;
        f.kv_len = p.kv_len; f.kv_stride = p.kv_stride; f.causal = p.causal; f.causal_base = p.causal_base;
        f.qscale = p.qscale;
        const LuxBackendError e = launch_attn_prefill(ctx, f, g_tune.attn_prefill == 3);
        return e != LUX_BACKEND_OK ? e : finish_op(ctx, (flags & LUX_QMATMUL_FLAG_NO_SYNC) != 0, what);
    }
    geometry(g_tune.attn_splits > 0 ? std::max<uint32_t>((uint32_t)g_tune.attn_splits, min_split) : best);
    if (p.nsplit > 256) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;     // a context beyond 256 x 2046 pages
    // A paged cache whose sequences may differ in length by enough has both kernels launched (gated): even shares if more than
    // `slack` of a full cache's chunks are missing, else slices.  A share costs a CTA some microseconds where it ends one item and
    // begins the next, about what 7 chunks take (9 where a few items are cut into many parts: 2 x 16000 with 9 missing a CTA 50.9 us by slices, 50.6 by
    // shares, 4 x 8000 with 8 48.8 / 49.5), or 14 chunks an item where CTAs take many items each; the kernel that leaves at once 1 to 3 us.
    // So this is for caches large enough that sequences of evenly spread lengths leave more than that missing (0.42 of a full one).
    // Llama-3-8B heads, 16-token pages, us a step by slices / by shares / gated.  Lengths 1, .2, .5, .9, ... of the longest: 8 x 2500 37.3 / 34.3 / 37.1,
    // 8 x 8000 83.8 / 64.6 / 66.7, 16 x 4000 90.0 / 68.4 / 71.4, 32 x 2000 85.7 / 71.2 / 73.3, 64 x 1500 107 / 97.8 / 102.8; not gated:
    // 8 x 2000 32.3 / 31.3, 20 x 1000 39.4 / 37.0, 32 x 1000 48.5 / 48.8, 48 x 1000 64.6 / 66.2, 64 x 1000 76.2 / 79.9.  All as long as the longest: 1 x 32768
    // 57.0 / 63.4 / 58.3, 8 x 8192 97.8 / 100.1 / 100.9, 32 x 2048 89.4 / 101.5 / 94.8.
    const uint32_t slots = (uint32_t)ctx->sm_count * (D > 128 ? 1 : ATT_CTAS_PER_SM);
    const uint64_t full_chunks = (uint64_t)items * chunks_of(max_keys);
    const size_t even_part = std::max((size_t)slots * 2 * rpb, out_rows * p.nsplit) * (D + 2) * 4 / 16 * 16 + 16;
    const uint64_t slack = g_tune.attn_even == 1 ? 0u : std::max<uint64_t>((items < 64 ? 9u : 7u) * slots, 14u * items);
    const bool gated = p.block_size && p.row_blocks == 1 && full_chunks < (1u << 31) && full_chunks * 5u >= slack * 12u && g_tune.attn_even != 2 &&
                       !g_tune.attn_splits && slots <= ATT_MAX_PARTS && even_part + items * sizeof(AttnSpan) <= ctx->d_attn_bytes;
    if (gated) {
        p.full_chunks = (uint32_t)full_chunks;
        p.slack = (uint32_t)slack;
        p.share = 4;                           // a share is no shorter than the shortest slice above
        p.ctas = (uint32_t)std::min<uint64_t>((full_chunks + p.share - 1) / p.share, slots);
        p.part = (float*)ctx->d_attn;
        p.spans = (AttnSpan*)((unsigned char*)ctx->d_attn + even_part);
    } else if (p.nsplit > 1) {
        if (out_rows * p.nsplit * (D + 2) * 4 > ctx->d_attn_bytes) {
            // fewer slices than wanted rather than an allocation inside a call
            const uint32_t fit = (uint32_t)(ctx->d_attn_bytes / (out_rows * (D + 2) * 4));
            if (std::max(fit, 1u) < min_split) return LUX_BACKEND_ERROR_OUT_OF_MEMORY;
            geometry(std::max(fit, 1u));
        }
        p.part = (float*)ctx->d_attn;
    }
    const size_t ctas = items * p.nsplit;
    if (ctas > 0x7fffffffu) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    const bool full = D == (uint32_t)vpl * 32u;
    auto launch = [&](Form form, size_t grid) {
        const size_t stage_bytes = (size_t)2 * ATT_CK * D * 4;
        const size_t fixed = form == EVEN ? ATT_EVEN_HEADER + att_merge_floats(D, rt) * 4 : ATT_HEADER + (p.block_size ? ATT_TABLE * 4 : 0);
        // heads wider than 128 take the whole SM's shared memory (one CTA per SM)
        const size_t budget = D > 128 ? 2 * ATT_SMEM_BUDGET : ATT_SMEM_BUDGET;
        p.stages = (uint32_t)std::min<size_t>(ATT_MAX_STAGES, (budget - fixed) / stage_bytes);
        AttnKernel kfn = pick_kernel(vpl, rt, full, form);
        if (!kfn || p.stages < 2) return LUX_BACKEND_ERROR_INTERNAL;
        static std::mutex mu;
        static bool attr_set[16][9][3][2][3];
        {
            std::lock_guard<std::mutex> lk(mu);
            bool& done = attr_set[ctx->device & 15][vpl][rt][full ? 1 : 0][form];
            if (!done) {
                if (cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(2 * ATT_SMEM_BUDGET)) != cudaSuccess)
                    return map_cuda(cudaGetLastError(), what);
                done = true;
            }
        }
        const cudaError_t e = launch_pdl(g_tune.pdl != 2, kfn, dim3((unsigned)grid), dim3(ATT_THREADS), fixed + p.stages * stage_bytes, ctx->stream, 1, p);
        if (e != cudaSuccess) return map_cuda(e, what);
        count_launch(form == EVEN ? "lux_attn_even_f32" : "lux_attn_stream_f32");
        return LUX_BACKEND_OK;
    };
    // The kernel that leaves at once costs less behind the other.  Lengths spread between 1/8 and all of the longest one, which fills the
    // table, leave 0.44 of the other sequences' chunks missing: one sequence, or two of 16 k keys, are more likely to
    // get slices (1 x 32768 keys 58.3 us with these first, 60.0 with shares first; 8 x 2500 ragged ones 39.7 / 37.1).
    const bool shares_first = gated && full_chunks * 44u * (p.batch - 1u) >= slack * 100u * p.batch;
    LuxBackendError le = shares_first ? launch(EVEN, p.ctas) : LUX_BACKEND_OK;
    if (le == LUX_BACKEND_OK) le = launch(gated ? SLICES_GATED : SLICES, ctas);
    if (le == LUX_BACKEND_OK && gated && !shares_first) le = launch(EVEN, p.ctas);
    if (le != LUX_BACKEND_OK) return le;
    if (gated || p.nsplit > 1) {
        const dim3 grid((unsigned)out_rows), block(128);
        const cudaError_t e = gated ? launch_pdl(g_tune.pdl != 2, lux_attn_merge_even_f32, grid, block, 0, ctx->stream, 1, p)
                                    : launch_pdl(g_tune.pdl != 2, lux_attn_merge_f32, grid, block, 0, ctx->stream, 1, (const float*)p.part, p.out, p.lse,
                                                 p.context_lens, p.heads * p.seq_q, p.nsplit, D);
        if (e != cudaSuccess) return map_cuda(e, what);
        count_launch("lux_attn_merge_f32");
    }
    return finish_op(ctx, (flags & LUX_QMATMUL_FLAG_NO_SYNC) != 0, what);
}

bool holds(const Buffer* b, size_t elems, size_t elem_bytes = 4) { return b && b->ptr && b->size / elem_bytes >= elems; }
// products of u32 arguments as a size, saturating
size_t mul(std::initializer_list<uint64_t> v) {
    unsigned __int128 r = 1;
    for (uint64_t x : v) {
        r *= x;
        if (r > (unsigned __int128)0x3fffffffffffffffull) return (size_t)0x3fffffffffffffffull;
    }
    return (size_t)r;
}

}  // namespace

// entries of the kernel table (kernel_table.cu): the Llama-shaped instance of the streaming kernel
const void* kernel_addr_attn_stream_f32() { return (const void*)lux_attn_stream_f32<4, 2, true, false>; }
const void* kernel_addr_attn_merge_f32() { return (const void*)lux_attn_merge_f32; }
const void* kernel_addr_attn_plain_f32() { return (const void*)lux_attn_plain_f32; }
const void* kernel_addr_rope_f32() { return (const void*)lux_rope_f32<uint32_t, 2>; }
const void* kernel_addr_kv_append_f32() { return (const void*)lux_kv_append_f32<uint32_t, 4>; }

}  // namespace luxcuda

using namespace luxcuda;

extern "C" LuxBackendError lux_cuda_rope_precompute_cache_f32(LuxBackendContext* context, LuxBackendBuffer* cos_out, LuxBackendBuffer* sin_out,
                                                              uint32_t max_seq_len, uint32_t head_dim, float theta_base, uint32_t flags) {
    Context* ctx = as_ctx(context);
    Buffer *bc = as_buf(cos_out), *bs = as_buf(sin_out);
    if (!ctx || !bc || !bs || head_dim == 0 || head_dim % 2 || !(theta_base > 0.0f)) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    const size_t total = mul({max_seq_len, head_dim / 2});
    if (!holds(bc, total) || !holds(bs, total)) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    if (total == 0) return LUX_BACKEND_OK;
    cudaSetDevice(ctx->device);
    const size_t blocks = std::min<size_t>((total + 255) / 256, (size_t)ctx->sm_count * 8);
    lux_rope_cache_f32<<<(unsigned)blocks, 256, 0, ctx->stream>>>((float*)bc->ptr, (float*)bs->ptr, max_seq_len, head_dim / 2, (float)head_dim,
                                                                 theta_base);
    count_launch("lux_rope_cache_f32");
    return finish_op(ctx, (flags & LUX_QMATMUL_FLAG_NO_SYNC) != 0, "rope_precompute_cache_f32");
}

namespace {
LuxBackendError rope_common(Context* ctx, RopeParams& p, Buffer* bc, Buffer* bs, uint32_t head_dim, uint32_t flags, const char* what) {
    if ((bc != nullptr) != (bs != nullptr)) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    p.half = head_dim / 2;
    p.head_dim_f = (float)head_dim;
    p.cos_cache = bc ? (const float*)bc->ptr : nullptr;
    p.sin_cache = bs ? (const float*)bs->ptr : nullptr;
    p.cache_positions = 0;
    if (bc) {
        if (!bc->ptr || !bs->ptr) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
        p.cache_positions = (uint32_t)std::min<size_t>(std::min(bc->size, bs->size) / 4 / p.half, 0xffffffffu);
        if (!p.position_ids && (uint64_t)p.position_offset + p.seq > p.cache_positions) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    }
    p.backward = (flags & LUX_ROPE_FLAG_BACKWARD) ? 1u : 0u;
    p.status = ctx->d_status;
    const size_t total = mul({p.batch, p.seq, (uint64_t)p.heads + p.heads2, p.half});
    if (total == 0) return LUX_BACKEND_OK;
    cudaSetDevice(ctx->device);
    const bool vec = p.half % 2 == 0 && aligned16(p.x) && aligned16(p.out) && aligned16(p.x2) && aligned16(p.out2);
    const size_t items = vec ? total / 2 : total, blocks = std::min<size_t>((items + 255) / 256, (size_t)ctx->sm_count * 16);
    const bool small = total < ((size_t)1 << 31);
    auto kfn = small ? (vec ? lux_rope_f32<uint32_t, 2> : lux_rope_f32<uint32_t, 1>) : (vec ? lux_rope_f32<size_t, 2> : lux_rope_f32<size_t, 1>);
    cudaError_t e = launch_pdl(g_tune.pdl != 2, kfn, dim3((unsigned)blocks), dim3(256), 0, ctx->stream, 1, p);
    if (e != cudaSuccess) return map_cuda(e, what);
    count_launch("lux_rope_f32");
    return finish_op(ctx, (flags & LUX_QMATMUL_FLAG_NO_SYNC) != 0, what);
}
}  // namespace

extern "C" LuxBackendError lux_cuda_rope_f32(LuxBackendContext* context, LuxBackendBuffer* x, LuxBackendBuffer* out, LuxBackendBuffer* cos_cache,
                                             LuxBackendBuffer* sin_cache, LuxBackendBuffer* position_ids, uint32_t batch_size,
                                             uint32_t seq_len, uint32_t num_heads, uint32_t head_dim, float theta_base,
                                             uint32_t position_offset, float ntk_scale, uint32_t flags) {
    Context* ctx = as_ctx(context);
    Buffer *bx = as_buf(x), *bo = as_buf(out), *bp = as_buf(position_ids);
    if (!ctx || !bx || !bo || head_dim == 0 || head_dim % 2) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    const size_t total = mul({batch_size, seq_len, num_heads, head_dim});
    if (!holds(bx, total) || !holds(bo, total)) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    if (bp && !holds(bp, mul({batch_size, seq_len}))) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    if ((reinterpret_cast<uintptr_t>(bx->ptr) | reinterpret_cast<uintptr_t>(bo->ptr)) & 7u) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    const bool cached = cos_cache || sin_cache;
    if (!cached && !(theta_base > 0.0f)) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    if (ntk_scale > 0.0f && (cached || head_dim <= 2)) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    RopeParams p{};
    p.x = (const float*)bx->ptr;
    p.out = (float*)bo->ptr;
    p.position_ids = bp ? (const uint32_t*)bp->ptr : nullptr;
    p.batch = batch_size;
    p.seq = seq_len;
    p.heads = num_heads;
    p.heads2 = 0;
    p.position_offset = position_offset;
    p.theta = theta_base;
    if (ntk_scale > 0.0f) {
        // scaled base, rope.wgsl:335, formed once on the host
        p.theta = theta_base * powf(ntk_scale, (float)head_dim / ((float)head_dim - 2.0f));
        p.ntk = 1;
    }
    return rope_common(ctx, p, as_buf(cos_cache), as_buf(sin_cache), head_dim, flags, "rope_f32");
}

extern "C" LuxBackendError lux_cuda_rope_qk_f32(LuxBackendContext* context, LuxBackendBuffer* q, LuxBackendBuffer* k, LuxBackendBuffer* cos_cache,
                                                LuxBackendBuffer* sin_cache, uint32_t batch_size, uint32_t seq_len, uint32_t num_heads,
                                                uint32_t num_kv_heads, uint32_t head_dim, uint32_t position_offset, uint32_t flags) {
    Context* ctx = as_ctx(context);
    Buffer *bq = as_buf(q), *bk = as_buf(k);
    if (!ctx || !bq || !bk || !cos_cache || !sin_cache || head_dim == 0 || head_dim % 2) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    if (!holds(bq, mul({batch_size, seq_len, num_heads, head_dim})) || !holds(bk, mul({batch_size, seq_len, num_kv_heads, head_dim})))
        return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    if ((reinterpret_cast<uintptr_t>(bq->ptr) | reinterpret_cast<uintptr_t>(bk->ptr)) & 7u) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    RopeParams p{};
    p.x = (const float*)bq->ptr;
    p.out = (float*)bq->ptr;
    p.x2 = (const float*)bk->ptr;
    p.out2 = (float*)bk->ptr;
    p.batch = batch_size;
    p.seq = seq_len;
    p.heads = num_heads;
    p.heads2 = num_kv_heads;
    p.position_offset = position_offset;
    p.theta = 1.0f;
    return rope_common(ctx, p, as_buf(cos_cache), as_buf(sin_cache), head_dim, flags, "rope_qk_f32");
}

extern "C" LuxBackendError lux_cuda_sdpa_f32(LuxBackendContext* context, LuxBackendBuffer* q, LuxBackendBuffer* k, LuxBackendBuffer* v,
                                             LuxBackendBuffer* out, LuxBackendBuffer* lse, uint32_t batch_size, uint32_t num_heads,
                                             uint32_t num_kv_heads, uint32_t seq_len_q, uint32_t seq_len_kv, uint32_t head_dim, float scale,
                                             uint32_t flags) {
    Context* ctx = as_ctx(context);
    Buffer *bq = as_buf(q), *bk = as_buf(k), *bv = as_buf(v), *bo = as_buf(out), *bl = as_buf(lse);
    if (!ctx || !bq || !bk || !bv || !bo || head_dim == 0 || num_kv_heads == 0 || num_heads % num_kv_heads) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    const size_t qn = mul({batch_size, num_heads, seq_len_q, head_dim}), kn = mul({batch_size, num_kv_heads, seq_len_kv, head_dim});
    if (!holds(bq, qn) || !holds(bo, qn)) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    if (kn && (!holds(bk, kn) || !holds(bv, kn))) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    if (bl && !holds(bl, mul({batch_size, num_heads, seq_len_q}))) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    AttnParams p{};
    p.q = (const float*)bq->ptr;
    p.k = (const float*)bk->ptr;
    p.v = (const float*)bv->ptr;
    p.out = (float*)bo->ptr;
    p.lse = bl ? (float*)bl->ptr : nullptr;
    p.batch = batch_size;
    p.heads = num_heads;
    p.kv_heads = num_kv_heads;
    p.group = num_heads / num_kv_heads;
    p.seq_q = seq_len_q;
    p.head_dim = head_dim;
    p.kv_len = seq_len_kv;
    p.kv_stride = seq_len_kv;
    p.causal = (flags & LUX_ATTN_FLAG_CAUSAL) ? 1u : 0u;
    p.causal_base = 0;
    p.qscale = scale * ATT_LOG2E;
    return attn_launch(ctx, p, seq_len_kv, flags, "sdpa_f32");
}

extern "C" LuxBackendError lux_cuda_update_kv_cache_f32(LuxBackendContext* context, LuxBackendBuffer* k, LuxBackendBuffer* v,
                                                        LuxBackendBuffer* k_cache, LuxBackendBuffer* v_cache, uint32_t batch_size,
                                                        uint32_t num_kv_heads, uint32_t seq_len_q, uint32_t cache_len, uint32_t max_cache_len,
                                                        uint32_t head_dim, uint32_t flags) {
    Context* ctx = as_ctx(context);
    Buffer *bk = as_buf(k), *bv = as_buf(v), *bkc = as_buf(k_cache), *bvc = as_buf(v_cache);
    if (!ctx || !bk || !bv || !bkc || !bvc || head_dim == 0) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    const size_t n = mul({batch_size, num_kv_heads, seq_len_q, head_dim}), cn = mul({batch_size, num_kv_heads, max_cache_len, head_dim});
    if (!holds(bk, n) || !holds(bv, n) || !holds(bkc, cn) || !holds(bvc, cn)) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    if (n == 0) return LUX_BACKEND_OK;
    cudaSetDevice(ctx->device);
    const bool vec = head_dim % 4 == 0 && aligned16(bk->ptr) && aligned16(bv->ptr) && aligned16(bkc->ptr) && aligned16(bvc->ptr);
    const size_t items = vec ? n / 4 : n, blocks = std::min<size_t>((items + 255) / 256, (size_t)ctx->sm_count * 16);
    const bool small = n < ((size_t)1 << 31);
    auto kfn = small ? (vec ? lux_kv_append_f32<uint32_t, 4> : lux_kv_append_f32<uint32_t, 1>)
                     : (vec ? lux_kv_append_f32<size_t, 4> : lux_kv_append_f32<size_t, 1>);
    cudaError_t e = launch_pdl(g_tune.pdl != 2, kfn, dim3((unsigned)blocks), dim3(256), 0, ctx->stream, 1, (const float*)bk->ptr,
                               (const float*)bv->ptr, (float*)bkc->ptr, (float*)bvc->ptr, batch_size * num_kv_heads, seq_len_q, cache_len,
                               max_cache_len, head_dim);
    if (e != cudaSuccess) return map_cuda(e, "update_kv_cache_f32");
    count_launch("lux_kv_append_f32");
    return finish_op(ctx, (flags & LUX_QMATMUL_FLAG_NO_SYNC) != 0, "update_kv_cache_f32");
}

extern "C" LuxBackendError lux_cuda_sdpa_kv_cache_f32(LuxBackendContext* context, LuxBackendBuffer* q, LuxBackendBuffer* k_cache,
                                                      LuxBackendBuffer* v_cache, LuxBackendBuffer* out, uint32_t batch_size, uint32_t num_heads,
                                                      uint32_t num_kv_heads, uint32_t seq_len_q, uint32_t cache_len, uint32_t max_cache_len,
                                                      uint32_t head_dim, float scale, uint32_t flags) {
    Context* ctx = as_ctx(context);
    Buffer *bq = as_buf(q), *bk = as_buf(k_cache), *bv = as_buf(v_cache), *bo = as_buf(out);
    if (!ctx || !bq || !bk || !bv || !bo || head_dim == 0 || num_kv_heads == 0 || num_heads % num_kv_heads || seq_len_q == 0)
        return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    if ((uint64_t)cache_len + seq_len_q > max_cache_len) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    const size_t qn = mul({batch_size, num_heads, seq_len_q, head_dim}), cn = mul({batch_size, num_kv_heads, max_cache_len, head_dim});
    if (!holds(bq, qn) || !holds(bo, qn) || !holds(bk, cn) || !holds(bv, cn)) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    AttnParams p{};
    p.q = (const float*)bq->ptr;
    p.k = (const float*)bk->ptr;
    p.v = (const float*)bv->ptr;
    p.out = (float*)bo->ptr;
    p.batch = batch_size;
    p.heads = num_heads;
    p.kv_heads = num_kv_heads;
    p.group = num_heads / num_kv_heads;
    p.seq_q = seq_len_q;
    p.head_dim = head_dim;
    p.kv_len = cache_len + seq_len_q;
    p.kv_stride = max_cache_len;
    p.causal = (flags & LUX_ATTN_FLAG_CAUSAL) ? 1u : 0u;
    p.causal_base = cache_len;
    p.qscale = scale * ATT_LOG2E;
    return attn_launch(ctx, p, p.kv_len, flags, "sdpa_kv_cache_f32");
}

extern "C" LuxBackendError lux_cuda_paged_attention_f32(LuxBackendContext* context, LuxBackendBuffer* q, LuxBackendBuffer* k_cache,
                                                        LuxBackendBuffer* v_cache, LuxBackendBuffer* block_tables,
                                                        LuxBackendBuffer* context_lens, LuxBackendBuffer* out, uint32_t num_seqs,
                                                        uint32_t num_heads, uint32_t num_kv_heads, uint32_t head_dim, uint32_t block_size,
                                                        uint32_t max_blocks_per_seq, float scale, uint32_t flags) {
    Context* ctx = as_ctx(context);
    Buffer *bq = as_buf(q), *bk = as_buf(k_cache), *bv = as_buf(v_cache), *bt = as_buf(block_tables), *bc = as_buf(context_lens),
           *bo = as_buf(out);
    if (!ctx || !bq || !bk || !bv || !bt || !bc || !bo || head_dim == 0 || num_kv_heads == 0 || num_heads % num_kv_heads || block_size == 0 ||
        max_blocks_per_seq == 0)
        return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    const size_t qn = mul({num_seqs, num_heads, head_dim});
    if (!holds(bq, qn) || !holds(bo, qn) || !holds(bt, mul({num_seqs, max_blocks_per_seq})) || !holds(bc, num_seqs))
        return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    const size_t block_elems = mul({num_kv_heads, block_size, head_dim});
    const size_t num_blocks = std::min(bk->size, bv->size) / 4 / block_elems;
    const uint64_t max_keys = (uint64_t)max_blocks_per_seq * block_size;
    if (num_blocks == 0 || !bk->ptr || !bv->ptr || max_keys > 0x7fffffffu) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    AttnParams p{};
    p.q = (const float*)bq->ptr;
    p.k = (const float*)bk->ptr;
    p.v = (const float*)bv->ptr;
    p.out = (float*)bo->ptr;
    p.block_tables = (const int32_t*)bt->ptr;
    p.context_lens = (const int32_t*)bc->ptr;
    p.batch = num_seqs;
    p.heads = num_heads;
    p.kv_heads = num_kv_heads;
    p.group = num_heads / num_kv_heads;
    p.seq_q = 1;
    p.head_dim = head_dim;
    p.kv_len = (uint32_t)max_keys;
    p.block_size = block_size;
    p.max_blocks_per_seq = max_blocks_per_seq;
    p.num_blocks = (uint32_t)std::min<size_t>(num_blocks, 0x7fffffffu);
    p.qscale = scale * ATT_LOG2E;
    return attn_launch(ctx, p, (uint32_t)max_keys, flags, "paged_attention_f32");
}
