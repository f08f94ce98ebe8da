"""The work a user of the backend has it do, as cases that can be timed and compared.

Every case goes through the public entry points (``webgpu_b200.backend``: the vtable slots and the
``lux_cuda_*`` symbols) the way a PyTorch host drives them: one context per process on torch's
current stream, tensors owned by torch and wrapped as backend buffers once, weights resident.
Calls that take the NO_SYNC flag carry it, as in a decode loop; the f32 vtable slots and the integer
path have no such flag and wait for the stream themselves.

Families (``kind``):
  linear     one quantized linear layer: int4 g128 with f16 / bf16 activations, int8 g32 with f32
  host       the same layer with the activations in host memory (copied in and out by the call)
  layer      the linear layers of one decoder layer: qkv, o, then the FFN (gate_up + SwiGLU, down)
  ffn        the FFN alone, at the sizes of the large model
  decode     decode attention: rotary embedding of the new token, KV append, attention over the cache
  prefill    attention of a whole prompt
  w8a8       activation-quantized integer layer: dynamic quantize, int8 matmul, requantize
  rows       the f32 slots around the linear layers of a prompt or a batch
  quantize   packing a weight matrix on the device
"""
import math

import torch

from webgpu_b200 import backend as B

_DT = {"f32": (torch.float32, B.F32), "f16": (torch.float16, B.F16), "bf16": (torch.bfloat16, B.BF16)}
_HEADS, _KV_HEADS, _HEAD_DIM = 32, 8, 128       # attention heads of the 8B-class decoder layer

_ctx = None


def _context():
    """One context per process, on the stream torch works on."""
    global _ctx
    if _ctx is None:
        _ctx = B.load().create_context(torch.cuda.current_device())
    _ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    return _ctx


# -- the cases --------------------------------------------------------------------------------------

def listed():
    return [
        # the smallest call: one int8 layer, one token, f32 activations (configuration 1)
        dict(name="int8_token", kind="linear", bits=8, dtype="f32", M=1, N=4096, K=4096, zeros=False),
        # one token whose activations live in host memory: latency of the whole call (configuration 2)
        dict(name="int4_token_host", kind="host", dtype="f16", M=1, N=14336, K=4096, zeros=True),
        # a decode step's linear layers, one user (configuration 4)
        dict(name="layer_batch1", kind="layer", dtype="f16", M=1, D=4096, QKV=6144, I=14336, zeros=True),
        # the same with sixteen users decoding together (configuration 4)
        dict(name="layer_batch16", kind="layer", dtype="f16", M=16, D=4096, QKV=6144, I=14336, zeros=True),
        # a ragged call: odd batch, outputs that fill no tile (the least that this route takes is a
        # multiple of 8), symmetric weights, bf16
        dict(name="ragged_bf16", kind="linear", bits=4, dtype="bf16", M=77, N=11016, K=4096, zeros=False),
        # prefill of a 512-token prompt (configuration 3)
        dict(name="prefill_linear", kind="linear", bits=4, dtype="bf16", M=512, N=4096, K=4096, zeros=True),
        # the FFN of the 70B-class model at its largest batch: the most arithmetic (configuration 5)
        dict(name="ffn_large_batch256", kind="ffn", dtype="f16", M=256, D=8192, I=28672, zeros=True),
        # serving: decode attention of 32 sequences of different lengths over a paged KV cache
        dict(name="paged_batch32", kind="decode", batch=32, context=4096, page=16),
        # prefill attention: causal, 2048 tokens
        dict(name="prefill_attention", kind="prefill", batch=1, seq=2048, causal=True, lse=False),
        # an activation-quantized layer over a 512-token prompt
        dict(name="w8a8_prompt", kind="w8a8", M=512, N=4096, K=4096),
        # norm, rotary embedding, gate product, residual and softmax of a 512-token prompt
        dict(name="rows_prompt", kind="rows", rows=512, dim=4096),
        # packing an 8B-class MLP matrix at load time
        dict(name="quantize_weights", kind="quantize", bits=4, dtype="f32", N=14336, K=4096, zeros=True),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mult(rng, lo, hi, m):
    """A multiple of m between lo and hi, spread over the logarithm."""
    return max(lo, min(hi, _log(rng, lo, hi) // m * m))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "host", "layer", "layer", "ffn", "decode", "decode", "prefill",
                       "w8a8", "rows", "quantize"])
    zeros = rng.random() < 0.7
    dtype = rng.choice(["f16", "bf16"])
    if kind == "linear" and rng.random() < 0.2:
        return dict(kind=kind, bits=8, dtype="f32", M=_log(rng, 1, 4), N=_log(rng, 1024, 16384), K=_mult(rng, 1024, 8192, 64), zeros=False)
    if kind == "linear":
        # layers whose outputs come in whole tiles of 128, and others: any number of outputs at up to
        # 32 f16 rows, a multiple of 8 elsewhere
        m = _log(rng, 1, 1024)
        n = _mult(rng, 1024, 28672, 128) if rng.random() < 0.6 else _log(rng, 1000, 28672)
        if m > 32 or dtype == "bf16":
            n = n // 8 * 8
        return dict(kind=kind, bits=4, dtype=dtype, M=m, N=n, K=_mult(rng, 1024, 14336, 128), zeros=zeros)
    if kind == "host":
        return dict(kind=kind, dtype=dtype, M=_log(rng, 1, 64), N=_mult(rng, 1024, 28672, 16), K=_mult(rng, 1024, 14336, 128), zeros=zeros)
    if kind == "layer":
        d = _mult(rng, 2048, 8192, 256)
        return dict(kind=kind, dtype=dtype, M=_log(rng, 1, 192), D=d, QKV=d + d // 2, I=_mult(rng, 2 * d, 7 * d // 2, 128), zeros=zeros)
    if kind == "ffn":
        return dict(kind=kind, dtype=dtype, M=_log(rng, 1, 256), D=8192, I=28672, zeros=zeros)
    if kind == "decode":
        batch = _log(rng, 1, 32)
        return dict(kind=kind, batch=batch, context=_log(rng, 200, min(32768, 65536 // batch)), page=rng.choice([0, 0, 16, 32]))
    if kind == "prefill":
        batch = rng.choice([1, 1, 2, 3])
        causal = rng.random() < 0.8
        # the pairs of positions stay below those of the listed 2048-token prompt
        seq = _log(rng, 150, int(2048 / math.sqrt(batch * (1 if causal else 2))))
        return dict(kind=kind, batch=batch, seq=seq, causal=causal, lse=rng.random() < 0.5)
    if kind == "w8a8":
        return dict(kind=kind, M=_log(rng, 16, 2048), N=_mult(rng, 1024, 8192, 16), K=_mult(rng, 1024, 8192, 16))
    if kind == "rows":
        dim = _mult(rng, 1024, 8192, 128)
        return dict(kind=kind, rows=_log(rng, 1, 8 * 1024 * 1024 // dim), dim=dim)
    bits = rng.choice([4, 4, 8])
    return dict(kind=kind, bits=bits, dtype=rng.choice(["f32", "bf16"]), N=_log(rng, 1000, 14336), K=_mult(rng, 1024, 4096, 128),
                zeros=bits == 4 and zeros)


# -- inputs -----------------------------------------------------------------------------------------

class _State:
    pass


def _normal(g, shape, dtype):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).to(dtype)


def _wrap(ctx, t):
    return ctx.wrap(t.data_ptr(), t.numel() * t.element_size())


def _layer(ctx, g, bits, N, K, zeros, keep):
    """Random packed weights with the distributions of the benchmark configurations."""
    if bits == 8:
        w = torch.randint(-127, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
        s = _normal(g, (N, K // 32), torch.float32).abs() * (0.02 / 127.0)
        keep += [w, s]
        return B.DeviceQLayer(8, 32, N, K, _wrap(ctx, w), _wrap(ctx, s), None, B.F32)
    w = torch.randint(0, 256, (N, K // 2), generator=g, device="cuda", dtype=torch.uint8)
    G = K // 128
    s = (_normal(g, (N, G), torch.float32).abs() * (0.02 / 7.0)).to(torch.float16)
    z = None
    if zeros:
        z = torch.randint(0, 256, (N, (G + 1) // 2), generator=g, device="cuda", dtype=torch.uint8)
        if G % 2:
            z[:, -1] &= 15
        keep.append(z)
    keep += [w, s]
    return B.DeviceQLayer(4, 128, N, K, _wrap(ctx, w), _wrap(ctx, s), _wrap(ctx, z) if zeros else None, B.F16)


def prepare(case, seed):
    ctx = _context()
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    s = _State()
    s.case, s.ctx, s.keep = case, ctx, []
    kind = case["kind"]

    def new(shape, dtype):
        t = torch.zeros(shape, device="cuda", dtype=dtype)
        return t, _wrap(ctx, t)

    def rand(shape, dtype=torch.float32):
        t = _normal(g, shape, dtype)
        s.keep.append(t)
        return _wrap(ctx, t)

    if kind in ("linear", "layer", "ffn"):
        td, s.code = _DT[case["dtype"]]
        M = case["M"]
        if kind == "linear":
            s.x = rand((M, case["K"]), td)
            s.w = _layer(ctx, g, case["bits"], case["N"], case["K"], case["zeros"], s.keep)
            s.y, s.by = new((M, case["N"]), td)
        else:
            D, I = case["D"], case["I"]
            s.x = rand((M, D), td)
            s.gate_up = _layer(ctx, g, 4, 2 * I, D, case["zeros"], s.keep)
            s.down = _layer(ctx, g, 4, D, I, case["zeros"], s.keep)
            s.h, s.bh = new((M, I), td)
            s.y, s.by = new((M, D), td)
            if kind == "layer":
                s.wqkv = _layer(ctx, g, 4, case["QKV"], D, case["zeros"], s.keep)
                s.wo = _layer(ctx, g, 4, D, D, case["zeros"], s.keep)
                s.attn = rand((M, D), td)               # what attention hands to the o projection
                s.qkv, s.bqkv = new((M, case["QKV"]), td)
                s.o, s.bo = new((M, D), td)
    elif kind == "host":
        td, _ = _DT[case["dtype"]]
        x = _normal(g, (case["M"], case["K"]), td).cpu()
        s.x = x.view(torch.int16).numpy().view("uint16") if td == torch.bfloat16 else x.numpy()
        s.w = _layer(ctx, g, 4, case["N"], case["K"], case["zeros"], s.keep)
    elif kind == "decode":
        b, n, page = case["batch"], case["context"], case["page"]
        H, KV, D = _HEADS, _KV_HEADS, _HEAD_DIM
        s.q, s.k, s.v = rand((b, 1, H, D)), rand((b, 1, KV, D)), rand((b, 1, KV, D))
        s.q_rot, s.bq_rot = new((b, 1, H, D), torch.float32)
        s.k_rot, s.bk_rot = new((b, 1, KV, D), torch.float32)
        s.out, s.bout = new((b, H, D), torch.float32)
        s.cos, s.bcos = new((n + 1, D // 2), torch.float32)
        s.sin, s.bsin = new((n + 1, D // 2), torch.float32)
        ctx.rope_precompute_cache(s.bcos, s.bsin, n + 1, D, 500000.0, B.FLAG_NO_SYNC)
        if page:
            # sequences of different lengths, the longest `context`; pages handed out in no order
            lens = torch.randint(max(1, n // 8), n + 1, (b,), generator=g, device="cuda", dtype=torch.int32)
            lens[0] = n
            blocks = (n + page - 1) // page
            table = torch.randperm(b * blocks, generator=g, device="cuda").to(torch.int32).reshape(b, blocks).contiguous()
            pos = (lens - 1).contiguous()
            s.kc, s.vc = rand((b * blocks, KV, page, D)), rand((b * blocks, KV, page, D))
            s.keep += [lens, table, pos]
            s.lens, s.table, s.pos = _wrap(ctx, lens), _wrap(ctx, table), _wrap(ctx, pos)
            s.blocks = blocks
        else:
            s.kc, s.vc = rand((b, KV, n, D)), rand((b, KV, n, D))
    elif kind == "prefill":
        b, n = case["batch"], case["seq"]
        s.q = rand((b, _HEADS, n, _HEAD_DIM))
        s.k, s.v = rand((b, _KV_HEADS, n, _HEAD_DIM)), rand((b, _KV_HEADS, n, _HEAD_DIM))
        s.out, s.bout = new((b, _HEADS, n, _HEAD_DIM), torch.float32)
        s.lse, s.blse = new((b, _HEADS, n), torch.float32) if case["lse"] else (None, None)
    elif kind == "w8a8":
        M, N, K = case["M"], case["N"], case["K"]
        s.x = rand((M, K))
        w = torch.randint(-127, 128, (K, N), generator=g, device="cuda", dtype=torch.int8)
        s.keep.append(w)
        s.w = _wrap(ctx, w)
        s.xq, s.bxq = new((M, K), torch.int8)
        s.scale, s.bscale = new((1,), torch.float32)
        s.acc, s.bacc = new((M, N), torch.int32)
        s.yq, s.byq = new((M, N), torch.int32)
    elif kind == "rows":
        r, d = case["rows"], case["dim"]
        s.x, s.res, s.up = rand((r, d)), rand((r, d)), rand((r, d))
        s.gamma = rand((d,))
        heads = d // _HEAD_DIM
        s.heads = heads
        s.cos, s.bcos = new((r, _HEAD_DIM // 2), torch.float32)
        s.sin, s.bsin = new((r, _HEAD_DIM // 2), torch.float32)
        ctx.rope_precompute_cache(s.bcos, s.bsin, r, _HEAD_DIM, 500000.0, B.FLAG_NO_SYNC)
        s.outs = [new((r, d), torch.float32) for _ in range(6)]
    elif kind == "quantize":
        N, K, bits = case["N"], case["K"], case["bits"]
        td, code = _DT[case["dtype"]]
        x = _normal(g, (N, K), td) * 0.02
        s.keep.append(x)
        s.x = _wrap(ctx, x)
        group, sd = (128, torch.float16) if bits == 4 else (32, torch.float32)
        G = K // group
        s.w, s.bw = new((N, K * bits // 8), torch.uint8)
        s.scales, s.bscales = new((N, G), sd)
        s.zeros, s.bzeros = new((N, (G + 1) // 2), torch.uint8) if case["zeros"] else (None, None)
        s.desc = B.make_desc(0, N, K, bits, group, code, B.F16 if bits == 4 else B.F32, B.F32, B.FLAG_NO_SYNC)
    else:
        raise ValueError(kind)
    return s


# -- one pass ---------------------------------------------------------------------------------------

def run(s):
    case, ctx, NS = s.case, s.ctx, B.FLAG_NO_SYNC
    kind = case["kind"]
    if kind == "linear":
        ctx.qmatmul(s.x, s.w, s.by, case["M"], s.code, flags=NS)
        return s.y
    if kind == "host":
        return ctx.qmatmul_host(s.x, s.w)
    if kind == "layer":
        M = case["M"]
        ctx.qmatmul(s.x, s.wqkv, s.bqkv, M, s.code, flags=NS)
        ctx.qmatmul(s.attn, s.wo, s.bo, M, s.code, flags=NS)
        ctx.qmlp(s.bo, s.gate_up, s.down, s.bh, s.by, M, s.code, flags=NS)
        return {"qkv": s.qkv, "o": s.o, "y": s.y}
    if kind == "ffn":
        ctx.qmlp(s.x, s.gate_up, s.down, s.bh, s.by, case["M"], s.code, flags=NS)
        return s.y
    if kind == "decode":
        b, n, page = case["batch"], case["context"], case["page"]
        H, KV, D = _HEADS, _KV_HEADS, _HEAD_DIM
        scale = 1.0 / math.sqrt(D)
        if page:
            ctx.rope(s.q, s.bq_rot, b, 1, H, D, cos=s.bcos, sin=s.bsin, position_ids=s.pos, flags=NS)
            ctx.paged_attention(s.bq_rot, s.kc, s.vc, s.table, s.lens, s.bout, b, H, KV, D, page, s.blocks, scale, flags=NS)
            return s.out
        ctx.rope(s.q, s.bq_rot, b, 1, H, D, cos=s.bcos, sin=s.bsin, position_offset=n - 1, flags=NS)
        ctx.rope(s.k, s.bk_rot, b, 1, KV, D, cos=s.bcos, sin=s.bsin, position_offset=n - 1, flags=NS)
        ctx.update_kv_cache(s.bk_rot, s.v, s.kc, s.vc, b, KV, 1, n - 1, n, D, flags=NS)
        ctx.sdpa_kv_cache(s.bq_rot, s.kc, s.vc, s.bout, b, H, KV, 1, n - 1, n, D, scale, flags=NS)
        return {"out": s.out, "k": s.k_rot}
    if kind == "prefill":
        b, n = case["batch"], case["seq"]
        ctx.sdpa(s.q, s.k, s.v, s.bout, b, _HEADS, _KV_HEADS, n, n, _HEAD_DIM, 1.0 / math.sqrt(_HEAD_DIM), lse=s.blse,
                 flags=NS | (B.FLAG_ATTN_CAUSAL if case["causal"] else 0))
        return [s.out] if s.lse is None else [s.out, s.lse]
    if kind == "w8a8":
        M, N, K = case["M"], case["N"], case["K"]
        ctx.dynamic_quantize(s.x, s.bxq, s.bscale, M * K)
        ctx.matmul_int8(s.bxq, s.w, s.bacc, M, N, K)
        # calibrated scales of the layer: sums of K products of about 30 by 70, mapped to the int8 range
        ctx.requantize(s.bacc, s.byq, M * N, 1.0, 70.0 * math.sqrt(K), 3)
        return {"xq": s.xq, "scale": s.scale, "acc": s.acc, "yq": s.yq}
    if kind == "rows":
        r, d = case["rows"], case["dim"]
        (h, bh), (n, bn), (ro, bro), (a, ba), (p, bp), (sm, bsm) = s.outs
        ctx.binary_f32("add", s.x, s.res, bh, r * d)                     # residual
        ctx.rms_norm_f32(bh, s.gamma, bn, r, d, 1e-5)
        ctx.rope(bn, bro, 1, r, s.heads, _HEAD_DIM, cos=s.bcos, sin=s.bsin, flags=NS)
        ctx.unary_f32("silu", bn, ba, r * d)
        ctx.binary_f32("mul", ba, s.up, bp, r * d)                       # gate product
        ctx.softmax_f32(bh, bsm, r, d)
        return [h, n, ro, a, p, sm]
    code = ctx.backend.lib.lux_cuda_qquantize(ctx.handle, s.desc, s.x.handle, s.bw.handle, s.bscales.handle,
                                              s.bzeros.handle if s.bzeros else None)
    if code != B.OK:
        raise B.BackendError(code, "lux_cuda_qquantize")
    return [s.w, s.scales] + ([s.zeros] if s.zeros is not None else [])


# -- what a pass cannot do without ------------------------------------------------------------------

def _weights(bits, N, K, zeros):
    if bits == 8:
        return N * K + N * (K // 32) * 4
    G = K // 128
    return N * K // 2 + N * G * 2 + (N * ((G + 1) // 2) if zeros else 0)


def work(case):
    kind = case["kind"]
    if kind in ("linear", "host"):
        bits = case.get("bits", 4)
        e = 4 if case["dtype"] == "f32" else 2
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": _weights(bits, N, K, case["zeros"]) + M * (N + K) * e, "flops": 2 * M * N * K}
    if kind in ("layer", "ffn"):
        M, D, I, z = case["M"], case["D"], case["I"], case["zeros"]
        b = _weights(4, 2 * I, D, z) + _weights(4, D, I, z) + 2 * M * D
        f = 6 * M * I * D
        if kind == "layer":
            q = case["QKV"]
            b += _weights(4, q, D, z) + _weights(4, D, D, z) + 2 * M * (3 * D + q)
            f += 2 * M * D * (q + D)
        else:
            b += 2 * M * D
        return {"bytes": b, "flops": f}
    if kind == "decode":
        b, n = case["batch"], case["context"]
        keys = n if not case["page"] else n * (1 + 9 / 16 * (b - 1)) / b     # mean of the lengths drawn
        kv = b * keys * _KV_HEADS * _HEAD_DIM
        return {"bytes": 2 * kv * 4 + b * (4 * _HEADS + 4 * _KV_HEADS) * _HEAD_DIM * 4, "flops": 4 * b * keys * _HEADS * _HEAD_DIM}
    if kind == "prefill":
        b, n = case["batch"], case["seq"]
        pairs = n * (n + 1) / 2 if case["causal"] else n * n
        return {"bytes": b * n * _HEAD_DIM * 4 * (2 * _HEADS + 2 * _KV_HEADS), "flops": 4 * b * _HEADS * pairs * _HEAD_DIM}
    if kind == "w8a8":
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": 5 * M * K + K * N + 8 * M * N, "flops": 2 * M * N * K}
    if kind == "rows":
        return {"bytes": case["rows"] * case["dim"] * 4 * 9, "flops": 20 * case["rows"] * case["dim"]}
    N, K = case["N"], case["K"]
    e = 4 if case["dtype"] == "f32" else 2
    return {"bytes": N * K * e + _weights(case["bits"], N, K, case["zeros"]), "flops": 4 * N * K}


def tolerance(case):
    kind = case["kind"]
    if kind in ("w8a8", "quantize"):
        return "exact"
    # about four times what the path shows against the same computation in 64 bits: 2.5e-7 (largest
    # single difference 3e-6 of the rms) in f32, and at 16 bits the rounding of weights and outputs,
    # once for a layer (f16 3.0e-4, bf16 2.4e-3) and again for a layer that feeds another
    if kind in ("decode", "prefill", "rows") or case["dtype"] == "f32":
        return {"rel": 2e-6, "max": 2e-5}
    chained = kind in ("layer", "ffn")
    if case["dtype"] == "f16":
        return {"rel": 2.6e-3, "max": 1.2e-2} if chained else {"rel": 1.2e-3, "max": 5e-3}
    return {"rel": 2e-2, "max": 0.1} if chained else {"rel": 1e-2, "max": 5e-2}
