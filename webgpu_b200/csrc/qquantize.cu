// lux_qquantize -- the quantize side of the group-quantized format: an f32 (or 16-bit) matrix
// [N, K] becomes the packed integers, the scale table and the zero-point table that the matmul
// kernels read.  One pass over the input, HBM-bound (4 bytes read and 0.5-1 byte written per
// element); the reference does it in two dispatches,
//
//   compute_group_scales       luxcpp/webgpu kernels/wgsl/gpu/quantized_nax.wgsl:157-232
//   quantize_nax_int4_sym      :236-259
//   quantize_nax_int4_asym     :288-310 (with pack_nax_int4_asym_x8, :115-122)
//   quantize_nax_int8_group    :336-362 (symmetric branch; pack_nax_int8_x4, :135-140)
//
// whose arithmetic is reproduced operation by operation (IEEE division, round-half-to-even,
// saturating float -> int conversion, min / max seeded with +-1e30, the zero-point computed before
// the "scale == 0 -> 1" guard), so that packed bytes, scales and zero-points come out bit-identical.
// That includes the asymmetric int4 shader's own behaviour: it stores clamp(round(v / scale), 0, 15),
// the zero-point is subtracted and added back around a second clamp and never shifts the value, so
// negative inputs are stored as 0.  LUX_QQUANT_FLAG_SHIFTED selects the usual
// clamp(round(v / scale) + zp, 0, 15) instead (an extension, not the reference's arithmetic).
//
// A warp works on 256 consecutive elements of a row at a time, 8 per lane: two int4 groups of 128 (16 lanes
// each) or eight int8 groups of 32 (4 lanes each).  Group minimum and maximum by shuffles inside the
// group's lanes; one 4-byte (int4) or 8-byte (int8) store per lane, coalesced over the warp; the two
// int4 zero-points of a warp share one byte of the zero-point table (low nibble first).
//
// This kernel WRITES buffers that a later matmul binds as weights.  It is a plain launch (no
// programmatic-launch trigger), and the entry point marks the context so that the next matmul is
// launched fully ordered behind it.
#include "common.cuh"
#include "round_div.cuh"

#include <type_traits>

namespace luxcuda {

namespace {

struct QuantParams {
    const void* x;          // [N, K] f32 / f16 / bf16
    uint8_t* w;             // int4: [N, K/2]; int8: [N, K]
    void* scales;           // [N, G] f32 or f16
    uint8_t* zeros;         // int4 asymmetric: [N, ZS]; else null
    int N, K, G, ZS;
    int scale_dtype;
    int shifted;            // LUX_QQUANT_FLAG_SHIFTED
    int chunks_per_row;     // ceil(K / 256)
};

// Where a lane's eight elements come from: f32 by one 32-byte load where the matrix is 32-byte aligned (by two 16-byte ones each of a
// warp's requests takes half of every sector it touches), f16, bf16.
enum Source { SRC_F32, SRC_F32_WIDE, SRC_F16, SRC_BF16 };
template <int SRC>
__device__ __forceinline__ void request8(const QuantParams& p, size_t idx, float4 (&r)[SRC <= SRC_F32_WIDE ? 2 : 1]) {
    if constexpr (SRC == SRC_F32_WIDE) {
        load32(reinterpret_cast<const float*>(p.x) + idx, r[0], r[1]);
    } else if constexpr (SRC == SRC_F32) {
        r[0] = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.x) + idx));
        r[1] = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.x) + idx) + 1);
    } else {
        r[0] = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const uint16_t*>(p.x) + idx));
    }
}
template <int SRC>
__device__ __forceinline__ void widen8(const float4 (&r)[SRC <= SRC_F32_WIDE ? 2 : 1], float (&v)[8]) {
    if constexpr (SRC <= SRC_F32_WIDE) {
        v[0] = r[0].x; v[1] = r[0].y; v[2] = r[0].z; v[3] = r[0].w; v[4] = r[1].x; v[5] = r[1].y; v[6] = r[1].z; v[7] = r[1].w;
    } else {
        const uint32_t u[4] = {__float_as_uint(r[0].x), __float_as_uint(r[0].y), __float_as_uint(r[0].z), __float_as_uint(r[0].w)};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (SRC == SRC_F16) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&u[i]));
                v[2 * i] = f.x; v[2 * i + 1] = f.y;
            } else {
                v[2 * i] = __uint_as_float(u[i] << 16);
                v[2 * i + 1] = __uint_as_float(u[i] & 0xFFFF0000u);
            }
        }
    }
}

// BITS = 4: groups of 128 (16 lanes); BITS = 8: groups of 32 (4 lanes), symmetric only.
// With a division per element, and the group's three per eight elements, the arithmetic took longer than the
// memory: 14336 x 4096 f32 to int4 with zero-points 72 us (266 MB, 3.7 TB/s).  round_div.cuh divides only
// next to half-integers and the group's divisions are spread over its lanes: 57 to 59 us (4.5 to 4.7 TB/s); with 32-byte loads
// 49.6 (5.4; timed alone, where 16-byte ones took 54.9).
// A warp takes QCH consecutive 256-element chunks of a row and requests all of them before it
// reduces the first: 4 KB in flight per warp, so that a streaming kernel with this little
// arithmetic keeps HBM busy.
constexpr int QCH = 4;

template <int BITS, bool SYM, int SRC>
__global__ void __launch_bounds__(256, 4) lux_qquantize(const QuantParams p) {
    constexpr int GL = BITS == 4 ? 16 : 4;                  // lanes per group
    const int lane = threadIdx.x & 31;
    const uint32_t wid = blockIdx.x * 8u + (threadIdx.x >> 5);
    const uint32_t wpr = (uint32_t)(p.chunks_per_row + QCH - 1) / QCH;     // warps per row
    const uint32_t row = wid / wpr;
    if (row >= (uint32_t)p.N) return;
    const size_t n = row;
    const int c0 = (int)(wid - row * wpr) * QCH;
    // all requests before the first value is used (16-bit values widened one chunk at a time, each as it arrived, had one
    // chunk of a warp in flight: 14336 x 4096 bf16 to int4 70 us, more than f32)
    float4 raw[QCH][SRC <= SRC_F32_WIDE ? 2 : 1];
    bool live[QCH];
#pragma unroll
    for (int ch = 0; ch < QCH; ch++) {
        const int k0 = (c0 + ch) * 256 + lane * 8;
        live[ch] = k0 < p.K;                                 // K is a multiple of the group size, so of 8
        if (live[ch]) request8<SRC>(p, n * (size_t)p.K + k0, raw[ch]);
    }
    float v[QCH][8];
#pragma unroll
    for (int ch = 0; ch < QCH; ch++)
        if (live[ch]) widen8<SRC>(raw[ch], v[ch]);
    // group statistics of all chunks
    float mx[QCH], mn[QCH];
#pragma unroll
    for (int ch = 0; ch < QCH; ch++) {
        mx[ch] = -1e30f;                                     // the shader's seeds (:169-170)
        mn[ch] = 1e30f;
        if (live[ch]) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                mx[ch] = fmaxf(mx[ch], v[ch][i]);
                mn[ch] = fminf(mn[ch], v[ch][i]);
            }
        }
#pragma unroll
        for (int o = GL / 2; o > 0; o >>= 1) {
            mx[ch] = fmaxf(mx[ch], __shfl_xor_sync(0xffffffffu, mx[ch], o));
            mn[ch] = fminf(mn[ch], __shfl_xor_sync(0xffffffffu, mn[ch], o));
        }
    }
    // Scale, zero-point and reciprocal: each lane works them out for ONE of its group's positions in the QCH
    // chunks (lane % QCH), so that a warp goes through those divisions once, not once per chunk.
    static_assert(QCH == 4 && GL >= QCH, "one lane of a group per chunk");
    const bool h1 = lane & 1, h2 = lane & 2;
    const float amx = h2 ? (h1 ? mx[3] : mx[2]) : (h1 ? mx[1] : mx[0]), amn = h2 ? (h1 ? mn[3] : mn[2]) : (h1 ? mn[1] : mn[0]);
    float scale;
    int zp = 0;
    if (SYM) {
        scale = __fdiv_rn(fmaxf(fabsf(amx), fabsf(amn)), BITS == 4 ? 7.0f : 127.0f);
    } else {
        scale = __fdiv_rn(amx - amn, 15.0f);
        zp = min(max(__float2int_rz(rintf(__fdiv_rn(-amn, scale))), 0), 15);   // before the guard, as in the shader
    }
    if (scale == 0.0f) scale = 1.0f;
    // compact table: an f16 table stores the rounded scale, and the values are quantized with the
    // number the table holds (what dequantize will multiply by)
    const __half s16 = __float2half_rn(scale);
    if (p.scale_dtype == LUX_QDTYPE_F16) scale = __half2float(s16);
    const float ri = __frcp_rn(scale);
    {
        const int k0 = (c0 + (lane & 3)) * 256 + (lane & ~(GL - 1)) * 8;       // first element of this lane's group
        if ((lane & (GL - 1)) < QCH && k0 < p.K) {
            const size_t at = n * (size_t)p.G + k0 / (BITS == 4 ? 128 : 32);
            if (p.scale_dtype == LUX_QDTYPE_F16) reinterpret_cast<__half*>(p.scales)[at] = s16;
            else reinterpret_cast<float*>(p.scales)[at] = scale;
        }
        if (BITS == 4 && !SYM) {
            // the two groups of a chunk share a byte (the second is absent in the last chunk of an odd row)
            const int zp_hi = __shfl_down_sync(0xffffffffu, zp, 16);
            if (lane < QCH && k0 < p.K) p.zeros[n * (size_t)p.ZS + c0 + lane] = (uint8_t)(zp | (k0 + 128 < p.K ? zp_hi << 4 : 0));
        }
    }
    const bool ok = round_div_ok(scale);
#pragma unroll
    for (int ch = 0; ch < QCH; ch++) {
        const int c = c0 + ch;
        const int k0 = c * 256 + lane * 8;
        if (c >= p.chunks_per_row) break;                    // warp-uniform
        const int src = (lane & ~(GL - 1)) | ch;             // the lane that worked out this chunk's group
        const float sc = __shfl_sync(0xffffffffu, scale, src), rc = __shfl_sync(0xffffffffu, ri, src);
        const int zc = __shfl_sync(0xffffffffu, zp | (ok ? 256 : 0), src);
        if (!live[ch]) continue;
        // stored value = clamp(rint(v / scale), lo, hi) + off:
        //   int8 and symmetric int4: the signed range; asymmetric int4: clamp(.., 0, 15) (the shader takes
        //   the zero-point out and back in around a second clamp); shifted: clamp(rint + zp, 0, 15)
        const int off = BITS == 8 ? 0 : SYM ? 8 : p.shifted ? zc & 15 : 0;
        uint32_t t[8];
        round_div<BITS>(v[ch], sc, rc, zc >= 256, BITS == 8 ? -128 : -off, BITS == 8 ? 127 : 15 - off, off, t);
        if (BITS == 4)
            reinterpret_cast<uint32_t*>(p.w)[(n * (size_t)p.K + k0) >> 3] = round_div_pack4(t);
        else
            reinterpret_cast<uint2*>(p.w)[(n * (size_t)p.K + k0) >> 3] =
                make_uint2(round_div_pack8(t[0], t[1], t[2], t[3]), round_div_pack8(t[4], t[5], t[6], t[7]));
    }
}

}  // namespace

const void* kernel_addr_qquantize_i4() { return (const void*)lux_qquantize<4, false, SRC_F32_WIDE>; }
const void* kernel_addr_qquantize_i8() { return (const void*)lux_qquantize<8, true, SRC_F32_WIDE>; }

}  // namespace luxcuda

using namespace luxcuda;

extern "C" LuxBackendError lux_cuda_qquantize(LuxBackendContext* context, const LuxQMatmulDesc* d, LuxBackendBuffer* x,
                                              LuxBackendBuffer* w_out, LuxBackendBuffer* scales_out,
                                              LuxBackendBuffer* zeros_out) {
    Context* ctx = as_ctx(context);
    Buffer *bx = as_buf(x), *bw = as_buf(w_out), *bs = as_buf(scales_out), *bz = as_buf(zeros_out);
    if (!ctx || !d || d->struct_size < sizeof(LuxQMatmulDesc) || !bx || !bw || !bs) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    if (d->N == 0 || d->K == 0 || (d->bits != 4 && d->bits != 8)) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    if (d->x_dtype > LUX_QDTYPE_BF16 || d->scale_dtype > LUX_QDTYPE_BF16) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    // the layouts the matmul kernels read: int4 in groups of 128 (f16 or f32 scales, with or without
    // zero-points), int8 in groups of 32 with f32 scales and no zero-points
    if (d->bits == 4 && (d->group_size != 128 || d->scale_dtype == LUX_QDTYPE_BF16)) return LUX_BACKEND_ERROR_NOT_SUPPORTED;
    if (d->bits == 8 && (d->group_size != 32 || d->scale_dtype != LUX_QDTYPE_F32 || bz)) return LUX_BACKEND_ERROR_NOT_SUPPORTED;
    if (d->K % d->group_size) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    const size_t N = d->N, K = d->K, G = K / d->group_size, ZS = (G + 1) / 2;
    const size_t xs = d->x_dtype == LUX_QDTYPE_F32 ? 4 : 2, ss = d->scale_dtype == LUX_QDTYPE_F32 ? 4 : 2;
    if (bx->size < N * K * xs || bw->size < N * K * d->bits / 8 || bs->size < N * G * ss) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    if (bz && bz->size < N * ZS) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    auto aligned16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    if (!aligned16(bx->ptr) || !aligned16(bw->ptr) || !aligned16(bs->ptr)) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;
    if (N * ((K + 255) / 256) > ((size_t)1 << 33)) return LUX_BACKEND_ERROR_INVALID_ARGUMENT;

    QuantParams p{};
    p.x = bx->ptr;
    p.w = (uint8_t*)bw->ptr;
    p.scales = bs->ptr;
    p.zeros = bz ? (uint8_t*)bz->ptr : nullptr;
    p.N = (int)N; p.K = (int)K; p.G = (int)G; p.ZS = (int)ZS;
    p.scale_dtype = (int)d->scale_dtype;
    p.shifted = (d->flags & LUX_QQUANT_FLAG_SHIFTED) ? 1 : 0;
    p.chunks_per_row = (int)((K + 255) / 256);
    const int src = d->x_dtype == LUX_QDTYPE_F16 ? SRC_F16 : d->x_dtype == LUX_QDTYPE_BF16 ? SRC_BF16
                    : (reinterpret_cast<uintptr_t>(bx->ptr) & 31u) ? SRC_F32 : SRC_F32_WIDE;
    const size_t warps = N * (size_t)((p.chunks_per_row + QCH - 1) / QCH);
    const unsigned grid = (unsigned)((warps + 7) / 8);
    cudaSetDevice(ctx->device);
    auto pick = [&](auto of) {
        constexpr int SRC = decltype(of)::value;
        return d->bits == 8 ? lux_qquantize<8, true, SRC> : bz ? lux_qquantize<4, false, SRC> : lux_qquantize<4, true, SRC>;
    };
    auto kfn = src == SRC_F16 ? pick(std::integral_constant<int, SRC_F16>{}) : src == SRC_BF16 ? pick(std::integral_constant<int, SRC_BF16>{})
               : src == SRC_F32 ? pick(std::integral_constant<int, SRC_F32>{}) : pick(std::integral_constant<int, SRC_F32_WIDE>{});
    kfn<<<grid, 256, 0, ctx->stream>>>(p);
    count_launch("lux_qquantize");
    ctx->writer_pending = true;          // cleared by the wait in finish_op unless NO_SYNC
    return finish_op(ctx, (d->flags & LUX_QMATMUL_FLAG_NO_SYNC) != 0, "lux_cuda_qquantize");
}
