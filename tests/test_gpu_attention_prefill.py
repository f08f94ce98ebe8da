"""lux_attn_prefill_mma_f32 and the f32 arithmetic it falls back to (many queries per head, head size 128) at the sizes where
their tiling can go wrong: queries and keys one off a tile of 64 or a block of 128, one tile, several,
masked and not, appended to a cache, heads that share a KV head, operands of very different magnitudes, NaN
and infinities; against the oracle, and against the streaming kernel.  Tolerance as in test_gpu_attention.py:
relative L2 <= 2e-6 (f32 sums in another order; the three bf16 parts of a factor keep all of its 24 bits)."""
import numpy as np
import pytest

from oracle import oracle as orc
from webgpu_b200 import backend as B

pytestmark = pytest.mark.gpu
TOL = 2e-6
KERNELS = {1: "lux_attn_prefill_mma_f32", 3: "lux_attn_prefill_f32"}      # by the tunable attn_prefill


class _Tuned:
    def __init__(self, backend, **kw):
        self.backend, self.kw = backend, kw

    def __enter__(self):
        for k, v in self.kw.items():
            self.backend.tune(k, v)

    def __exit__(self, *exc):
        for k in self.kw:
            self.backend.tune(k, 0)


def _qkv(seed, B_, H, Hkv, Sq, Skv, D=128):
    rng = np.random.default_rng(seed)
    return [rng.standard_normal(s, np.float32) for s in ((B_, H, Sq, D), (B_, Hkv, Skv, D), (B_, Hkv, Skv, D))]


def _sdpa(ctx, q, k, v, causal, scale=None):
    B_, H, Sq, D = q.shape
    qb, kb, vb, ob, lb = ctx.upload(q), ctx.upload(k), ctx.upload(v), ctx.alloc(q.nbytes), ctx.alloc(B_ * H * Sq * 4)
    ctx.sdpa(qb, kb, vb, ob, B_, H, k.shape[1], Sq, k.shape[2], D, 1 / np.sqrt(D) if scale is None else scale, lse=lb,
             flags=B.FLAG_ATTN_CAUSAL if causal else 0)
    return ob.to_host(np.float32, q.shape), lb.to_host(np.float32, (B_, H, Sq))


@pytest.mark.parametrize("mode", [1, 3])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("B_,H,Hkv,Sq,Skv", [(1, 2, 2, 127, 128), (1, 1, 1, 129, 191), (1, 2, 1, 260, 300), (1, 2, 2, 1, 1), (1, 2, 1, 63, 63), (1, 2, 2, 64, 64), (2, 4, 2, 65, 65), (1, 4, 1, 17, 129),
                                             (1, 3, 3, 130, 40), (2, 4, 4, 200, 257)])
def test_tile_edges(ctx, backend, B_, H, Hkv, Sq, Skv, causal, mode):
    q, k, v = _qkv(Sq * 1000 + Skv, B_, H, Hkv, Sq, Skv)
    with _Tuned(backend, attn_prefill=mode):
        got, lse = _sdpa(ctx, q, k, v, causal)
        assert backend.last_kernel_name() == KERNELS[mode]
    want, want_lse = orc.sdpa(q, k, v, 1 / np.sqrt(128), causal, want_lse=True)
    assert orc.rel_l2(got, want) < TOL
    np.testing.assert_allclose(got, want, rtol=1e-4, atol=1e-5)
    np.testing.assert_allclose(lse, want_lse, rtol=1e-5, atol=1e-5)
    assert ctx.last_device_status() == 0


@pytest.mark.parametrize("Sq,cache_len,max_len", [(64, 0, 64), (65, 63, 200), (100, 301, 512)])
def test_chunk_appended_to_a_cache(ctx, backend, Sq, cache_len, max_len):
    """Causal rows start at cache_len, and two KV heads lie max_len rows apart: the streaming kernel's answer
    to the same call is the reference (both sum in f32; 2e-6 as against the oracle)."""
    q, k, v = _qkv(cache_len, 2, 8, 2, Sq, max_len)
    qb, kb, vb, ob = ctx.upload(q), ctx.upload(k), ctx.upload(v), ctx.alloc(q.nbytes)
    outs = []
    for mode in (1, 3, 2):
        with _Tuned(backend, attn_prefill=mode):
            ctx.sdpa_kv_cache(qb, kb, vb, ob, 2, 8, 2, Sq, cache_len, max_len, 128, 1 / np.sqrt(128), flags=B.FLAG_ATTN_CAUSAL)
            assert mode == 2 or backend.last_kernel_name() == KERNELS[mode]
        outs.append(ob.to_host(np.float32, q.shape).copy())
    assert orc.rel_l2(outs[0], outs[2]) < TOL and orc.rel_l2(outs[1], outs[2]) < TOL


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_values_a_row_must_not_see_do_not_reach_it(ctx, backend, bad):
    """A causal row ignores later positions altogether: a NaN or infinity in V (or NaN in K) there leaves every
    earlier row bit for bit as it was, and reaches every row that sees it."""
    q, k, v = _qkv(5, 1, 2, 1, 150, 150)
    v2, k2 = v.copy(), k.copy()
    v2[0, 0, 70, 3] = bad
    k2[0, 0, 100, 5] = np.nan
    with _Tuned(backend, attn_prefill=3):
        clean, _ = _sdpa(ctx, q, k, v, True)
        got, lse = _sdpa(ctx, q, k2, v2, True)
    assert np.array_equal(got[:, :, :70].view(np.uint32), clean[:, :, :70].view(np.uint32))
    assert not np.isfinite(got[:, :, 70:100, 3]).any() and np.array_equal(got[:, :, 70:100, 4], clean[:, :, 70:100, 4])
    # the tensor-core kernel leaves such a call to the f32 kernel: the same bits; the next call is its own again
    with _Tuned(backend, attn_prefill=1):
        got1, lse1 = _sdpa(ctx, q, k2, v2, True)
        after, _ = _sdpa(ctx, q, k, v, True)
    assert np.array_equal(got1.view(np.uint32), got.view(np.uint32)) and np.array_equal(lse1.view(np.uint32), lse.view(np.uint32))
    assert orc.rel_l2(after, clean) < TOL


@pytest.mark.parametrize("bad", [np.nan, -np.inf])
@pytest.mark.parametrize("row", [0, 15, 16, 77, 127, 128, 149])
def test_a_non_finite_query_is_noticed_by_every_warp(ctx, backend, row, bad):
    """One value of Q, in the first or last row of a warp, a block and the call: the f32 kernel's bits, whichever
    warp meets it and however early."""
    q, k, v = _qkv(11, 1, 1, 1, 150, 150)
    q[0, 0, row, row % 128] = bad
    outs = []
    for mode in (3, 1):
        with _Tuned(backend, attn_prefill=mode):
            outs.append(_sdpa(ctx, q, k, v, True))
    for a, b in zip(*outs):
        assert np.array_equal(a[:, :, row // 128 * 128:][:, :, :128].view(np.uint32), b[:, :, row // 128 * 128:][:, :, :128].view(np.uint32))


@pytest.mark.parametrize("mode", [1, 3])
def test_no_keys_and_large_scores(ctx, backend, mode):
    q, k, v = _qkv(6, 1, 2, 2, 70, 70)
    with _Tuned(backend, attn_prefill=mode):
        got, lse = _sdpa(ctx, q * 100, k, v, False)
        empty, _ = _sdpa(ctx, q, k[:, :, :0], v[:, :, :0], False)
    want, want_lse = orc.sdpa(q * 100, k, v, 1 / np.sqrt(128), False, want_lse=True)
    # scores reach 450, where a rounding of the score is worth 450 x 2^-24 = 3e-5 of a weight; a few such add up
    assert orc.rel_l2(got, want) < 1e-4
    np.testing.assert_allclose(lse, want_lse, rtol=1e-5, atol=1e-4)
    assert not empty.any()


def test_magnitudes_far_apart(ctx, backend):
    """Rows of K, columns of V and the whole of Q at scales from 1e-12 to 1e12 of each other: every output column keeps
    its own relative precision (the parts have f32's exponents)."""
    q, k, v = _qkv(8, 1, 2, 1, 140, 200)
    rng = np.random.default_rng(8)
    ks = 10.0 ** rng.uniform(-12, 0, (1, 1, 200, 1))
    vs = 10.0 ** rng.uniform(-12, 12, (1, 1, 1, 128))
    k, v = (k * ks).astype(np.float32), (v * vs).astype(np.float32)
    with _Tuned(backend, attn_prefill=1):
        got, _ = _sdpa(ctx, q, k, v, False)
    want = orc.sdpa(q, k, v, 1 / np.sqrt(128), False)
    err = np.sqrt((((got - want) / vs) ** 2).sum(axis=(0, 1, 2)) / ((want / vs) ** 2).sum(axis=(0, 1, 2)))
    assert err.max() < 2 * TOL, err.max()                 # the worst of 128 columns, each with 280 values


def _sdpa64(q, k, v, causal, scale=None):
    """Attention in 64 bits (weights exp(s - max), as they are)."""
    q, k, v = (x.astype(np.float64) for x in (q, k, v))
    g = q.shape[1] // k.shape[1]
    k, v = np.repeat(k, g, axis=1), np.repeat(v, g, axis=1)
    s = q @ k.transpose(0, 1, 3, 2) * (1 / np.sqrt(q.shape[-1]) if scale is None else scale)
    if causal:
        s = np.where(np.tril(np.ones(s.shape[-2:], bool)), s, -np.inf)
    w = np.exp(s - s.max(axis=-1, keepdims=True))
    return w @ v / w.sum(axis=-1, keepdims=True)


@pytest.mark.parametrize("factor", [1e5, 1e8, 1e12, 1e30])
@pytest.mark.parametrize("key", [63, 149])
def test_large_finite_values_behind_the_mask_do_not_reach_earlier_rows(ctx, backend, key, factor):
    """V of a later key, in the same tile, times up to 1e30: the rows that must not see it keep their precision."""
    q, k, v = _qkv(12, 1, 2, 1, 150, 150)
    want = _sdpa64(q, k, v, True)[:, :, :key]
    v[0, 0, key] *= np.float32(factor)
    with _Tuned(backend, attn_prefill=1):
        got, _ = _sdpa(ctx, q, k, v, True)
    assert orc.rel_l2(got[:, :, :key], want) < TOL


@pytest.mark.parametrize("lo,hi", [(-6, 6), (-6, 12), (-30, 0)])
def test_keys_of_very_different_magnitude(ctx, backend, lo, hi):
    """V growing from key to key: a causal row's result is as precise as the largest value that it SEES allows."""
    q, k, v = _qkv(13, 1, 2, 1, 150, 150)
    v = (v * 10.0 ** np.linspace(lo, hi, 150).reshape(1, 1, 150, 1)).astype(np.float32)
    with _Tuned(backend, attn_prefill=1):
        got, _ = _sdpa(ctx, q, k, v, True)
    want = _sdpa64(q, k, v, True)
    err = np.linalg.norm(got - want, axis=-1) / np.linalg.norm(want, axis=-1)
    # one row of 128 values at a time: the largest of 300 such errors, against TOL over a whole call
    assert err.max() < 2 * TOL, err.max()


@pytest.mark.parametrize("drop", [14, 18, 21, 30, 60, 80])
def test_small_weights_under_a_dominant_key_without_a_value(ctx, backend, drop):
    """One key takes the row's weight and its V is zero: the output is made of weights of e^-drop, down to 2^-115, alone."""
    rng = np.random.default_rng(14)
    q, k, v = _qkv(14, 1, 2, 1, 140, 140)
    k *= np.float32(0.1)
    k[0, 0, 0] = 0.0
    q[..., 0], k[..., 0] = np.float32(np.sqrt(128)), np.float32(0)
    k[0, 0, 0, 0] = drop                                   # its score is `drop`, the others' about 0
    v[0, 0, 0] = 0.0
    with _Tuned(backend, attn_prefill=1):
        got, _ = _sdpa(ctx, q, k, v, False)
    # the maximum and the exponent's argument, drop log2(e) in size, are each rounded to half an ulp, and an absolute error
    # there is a relative one of the weight: up to 2 ln(2) 2^-25 2^ceil(log2(drop log2(e))), 2.6e-6 at 30 and 5.3e-6 at 80
    bound = 2 * np.log(2) * 2.0 ** -25 * 2 ** np.ceil(np.log2(drop / np.log(2)))
    assert orc.rel_l2(got, _sdpa64(q, k, v, False)) < bound + 1e-6


@pytest.mark.parametrize("columns", [slice(None), slice(5, 6)])
@pytest.mark.parametrize("scale", [1e-28, 1e-31, 1e-34, 1e-37])
def test_values_close_to_the_smallest_normal_number(ctx, backend, scale, columns):
    """V (or one column of it) down to 1e-37: f32 keeps 24 bits there, and so does every column of the output."""
    q, k, v = _qkv(21, 1, 2, 1, 140, 140)
    v[..., columns] *= np.float32(scale)
    with _Tuned(backend, attn_prefill=1):
        got, _ = _sdpa(ctx, q, k, v, True)
    want = _sdpa64(q, k, v, True)
    err = np.sqrt(((got - want) ** 2).sum(axis=(0, 1, 2)) / (want ** 2).sum(axis=(0, 1, 2)))
    assert err.max() < 2 * TOL, err.max()                 # the worst of 128 columns, each with 280 values


@pytest.mark.parametrize("qs,ks", [(1e15, 1e-15), (1e30, 1e-30), (1e37, 1e-37), (1e-30, 1e30), (1e-37, 1e37)])
def test_scores_of_ordinary_size_from_extreme_operands(ctx, backend, qs, ks):
    """Q and K far from 1 with ordinary products: no scale of the kernel's own overflows or takes bits away."""
    q, k, v = _qkv(15, 1, 2, 1, 140, 140)
    q, k = q * np.float32(qs), k * np.float32(ks)
    with _Tuned(backend, attn_prefill=1):
        got, _ = _sdpa(ctx, q, k, v, True)
    assert orc.rel_l2(got, _sdpa64(q, k, v, True)) < TOL


@pytest.mark.parametrize("value", [np.float32(2) - np.float32(2) ** -23, np.float32(1), np.float32(3e-30)])
def test_a_constant_v_comes_back(ctx, backend, value):
    """Weights sum to one: with one value in all of V every output is that value to a few roundings, and not
    all of them on one side of it."""
    q, k, v = _qkv(16, 1, 4, 4, 300, 300)
    v[:] = value
    with _Tuned(backend, attn_prefill=1):
        got, _ = _sdpa(ctx, q, k, v, True)
    r = got.astype(np.float64) / np.float64(value) - 1
    assert np.abs(r).max() < 8 * 2.0 ** -24 and abs(r.mean()) < 2.0 ** -24


@pytest.mark.parametrize("where,bad", [("q", np.nan), ("k", np.inf), ("v", np.nan), ("v", 1e30)])
def test_a_block_out_of_range_leaves_the_others_alone(ctx, backend, where, bad):
    """What the tensor-core parts cannot carry is met in one sequence: its blocks that see it take the f32 kernel's bits, every
    block that does not see it keeps its own."""
    q, k, v = _qkv(17, 2, 2, 1, 300, 300)
    dirty = {"q": q.copy(), "k": k.copy(), "v": v.copy()}
    dirty[where][1, 0, 200, 5] = bad
    with _Tuned(backend, attn_prefill=1):
        clean, clean_lse = _sdpa(ctx, q, k, v, True)
        got, lse = _sdpa(ctx, **dirty, causal=True)
    with _Tuned(backend, attn_prefill=3):
        want, want_lse = _sdpa(ctx, **dirty, causal=True)
    seen = np.zeros((2, 2, 300), bool)                     # rows of blocks (128 queries) that meet it
    seen[1, :1 if where == "q" else 2, 128:256 if where == "q" else 300] = True
    for g, c, w in ((got, clean, want), (lse, clean_lse, want_lse)):
        assert np.array_equal(g[seen].view(np.uint32), w[seen].view(np.uint32))
        assert np.array_equal(g[~seen].view(np.uint32), c[~seen].view(np.uint32))


def test_output_over_the_queries(ctx, backend):
    """out == q, with and without a value out of range: a block reads its queries before it writes."""
    q, k, v = _qkv(18, 1, 2, 1, 260, 260)
    bad = v.copy()
    bad[0, 0, 250, 7] = np.inf
    for vv in (v, bad):
        with _Tuned(backend, attn_prefill=1):
            want, _ = _sdpa(ctx, q, k, vv, True)
            qb = ctx.upload(q)
            ctx.sdpa(qb, ctx.upload(k), ctx.upload(vv), qb, 1, 2, 1, 260, 260, 128, 1 / np.sqrt(128), flags=B.FLAG_ATTN_CAUSAL)
        assert np.array_equal(qb.to_host(np.float32, q.shape).view(np.uint32), want.view(np.uint32))


def test_replays_of_a_captured_call_do_not_remember(backend):
    """Captured once, replayed with finite, non-finite and finite inputs: the last replay gives the first one's bits."""
    import torch
    c = backend.create_context(0)
    try:
        st = torch.cuda.Stream()
        c.set_stream(st.cuda_stream)
        q, k, v = (torch.from_numpy(x).cuda() for x in _qkv(19, 1, 2, 1, 150, 150))
        o = torch.zeros_like(q)
        bufs = [c.wrap(t.data_ptr(), t.numel() * 4) for t in (q, k, v, o)]
        call = lambda: c.sdpa(*bufs, 1, 2, 1, 150, 150, 128, 1 / np.sqrt(128), flags=B.FLAG_NO_SYNC | B.FLAG_ATTN_CAUSAL)
        with _Tuned(backend, attn_prefill=1):
            torch.cuda.synchronize()
            with torch.cuda.stream(st):
                call()
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=st, capture_error_mode="relaxed"):
                    call()
            outs = []
            for val in (None, float("nan"), None):
                keep = v[0, 0, 100, 3].clone()
                if val is not None:
                    v[0, 0, 100, 3] = val
                torch.cuda.synchronize()
                g.replay()
                torch.cuda.synchronize()
                outs.append(o.cpu().numpy().copy())
                v[0, 0, 100, 3] = keep
        torch.cuda.synchronize()
        del g
        assert np.isnan(outs[1][0, :, 100:, 3]).all() and np.isfinite(outs[2]).all()
        assert np.array_equal(outs[0].view(np.uint32), outs[2].view(np.uint32))
    finally:
        c.destroy()


@pytest.mark.parametrize("H,S,kernels", [(32, 256, ("lux_attn_prefill_mma_f32",)), (8, 128, ("lux_attn_stream_f32", "lux_attn_merge_f32"))])
def test_default_choice(ctx, backend, H, S, kernels):
    """Prompts with enough (head, 64 queries) blocks to fill the chip take it, small ones the key-splitting kernel."""
    q, k, v = _qkv(7, 1, H, H, S, S)
    got, _ = _sdpa(ctx, q, k, v, True)
    assert backend.last_kernel_name() in kernels
    assert orc.rel_l2(got[:, :2], orc.sdpa(q[:, :2], k[:, :2], v[:, :2], 1 / np.sqrt(128), True)) < TOL


@pytest.mark.parametrize("Sq,keys,takes", [(65, 4096, False), (128, 4096, False), (512, 4096, True), (65, 300, False), (256, 300, True)])
def test_default_choice_over_a_cache(ctx, backend, Sq, keys, takes):
    """A chunk of a prompt over a longer cache: its blocks of 128 queries walk all keys alone, so few of them go to the
    kernel that also splits the keys; either way the answer is that kernel's to rounding."""
    q, k, v = _qkv(20, 1, 32, 8, Sq, keys)
    qb, kb, vb, ob = ctx.upload(q), ctx.upload(k), ctx.upload(v), ctx.alloc(q.nbytes)
    outs = []
    for mode in (0, 2):
        with _Tuned(backend, attn_prefill=mode):
            ctx.sdpa_kv_cache(qb, kb, vb, ob, 1, 32, 8, Sq, keys - Sq, keys, 128, 1 / np.sqrt(128), flags=B.FLAG_ATTN_CAUSAL)
            assert mode or (backend.last_kernel_name() == "lux_attn_prefill_mma_f32") == takes
        outs.append(ob.to_host(np.float32, q.shape).copy())
    assert orc.rel_l2(outs[0], outs[1]) < TOL


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("B_,H,Hkv,Sq,Skv", [(1, 1, 1, 65, 65), (1, 5, 1, 129, 640), (1, 3, 3, 257, 449), (1, 6, 2, 128, 512), (1, 4, 2, 385, 385), (2, 8, 2, 250, 1000)])
def test_pairs_of_blocks(ctx, backend, B_, H, Hkv, Sq, Skv, causal):
    """Two heads of a KV head, or two blocks of queries of one head (the last one alone, or seeing fewer tiles than its
    partner), over as many tiles as the ring has slots and more; against 64 bits."""
    q, k, v = _qkv(Sq + Skv, B_, H, Hkv, Sq, Skv)
    with _Tuned(backend, attn_prefill=1):
        got, _ = _sdpa(ctx, q, k, v, causal)
    assert orc.rel_l2(got, _sdpa64(q, k, v, causal)) < TOL and ctx.last_device_status() == 0


@pytest.mark.parametrize("where", ["q", "k", "v"])
def test_an_odd_pair_with_one_block_out_of_range(ctx, backend, where):
    """Two blocks of queries of one head make a pair: what only the later one meets leaves the earlier one its own bits."""
    q, k, v = _qkv(22, 1, 1, 1, 250, 250)
    dirty = {"q": q.copy(), "k": k.copy(), "v": v.copy()}
    dirty[where][0, 0, 200, 5] = np.inf
    with _Tuned(backend, attn_prefill=1):
        clean, _ = _sdpa(ctx, q, k, v, True)
        got, _ = _sdpa(ctx, **dirty, causal=True)
    with _Tuned(backend, attn_prefill=3):
        want, _ = _sdpa(ctx, **dirty, causal=True)
    assert np.array_equal(got[:, :, :128].view(np.uint32), clean[:, :, :128].view(np.uint32))
    assert np.array_equal(got[:, :, 128:].view(np.uint32), want[:, :, 128:].view(np.uint32))


@pytest.mark.parametrize("B_,Hkv,Skv,kernel", [(3, 50, 1000, "lux_attn_prefill_mma_f32"), (1, 1, 131073, "lux_attn_prefill_mma_f32"), (1, 2, 90001, "lux_attn_prefill_mma_f32")])
def test_more_keys_than_the_scratch_holds(ctx, backend, B_, Hkv, Skv, kernel):
    """128 k keys of all KV heads have their parts in the scratch at a time: more heads, or longer ones, go in several passes;
    either way the streaming kernel's answer to rounding."""
    q, k, v = _qkv(23, B_, Hkv, Hkv, 66, Skv)
    outs = []
    for mode in (1, 2):
        with _Tuned(backend, attn_prefill=mode):
            outs.append(_sdpa(ctx, q, k, v, False)[0])
            assert mode == 2 or backend.last_kernel_name() == kernel
    # an output is the mean of Skv values: its rounding errors grow with the square root of the chain of sums
    assert orc.rel_l2(outs[0], outs[1]) < TOL * max(1.0, (Skv / 4096) ** 0.5)


def test_no_less_precise_than_the_streaming_kernel(ctx, backend):
    """Error against 64 bits over lengths of one tile to many, masked and not: the tensor core's chains are short, so it
    stays below that of ordinary f32 sums."""
    for Sq, causal in ((64, True), (150, True), (512, True), (700, False)):
        q, k, v = _qkv(Sq, 1, 4, 1, Sq, Sq)
        want = _sdpa64(q, k, v, causal)
        errs = []
        for mode in (1, 2):
            with _Tuned(backend, attn_prefill=mode):
                errs.append(orc.rel_l2(_sdpa(ctx, q, k, v, causal)[0], want))
        assert errs[0] < errs[1], (Sq, causal, errs)


def test_keys_and_values_at_a_16_byte_offset(ctx, backend):
    """K and V that are 16- but not 32-byte aligned are read by 16-byte loads: the same bits."""
    q, k, v = _qkv(24, 1, 4, 2, 130, 200)
    with _Tuned(backend, attn_prefill=1):
        want, _ = _sdpa(ctx, q, k, v, False)
        bufs = []
        for a in (k, v):
            big = ctx.upload(np.concatenate([np.zeros(4, np.float32), a.ravel()]))
            bufs += [big, ctx.wrap(big.device_ptr + 16, a.nbytes)]
        ob = ctx.alloc(q.nbytes)
        ctx.sdpa(ctx.upload(q), bufs[1], bufs[3], ob, 1, 4, 2, 130, 200, 128, 1 / np.sqrt(128))
        assert backend.last_kernel_name() == "lux_attn_prefill_mma_f32"
    assert np.array_equal(ob.to_host(np.uint32, q.shape), want.view(np.uint32))


def test_calls_on_two_streams_share_the_scratch_in_order(backend):
    """Calls enqueued on one stream, then on another, without a wait: each keeps the bits that it has alone, though both
    split their K and V into the same scratch."""
    import torch
    c = backend.create_context(0)
    try:
        streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        data, want = [], []
        for i, S in enumerate((1500, 700)):
            t = [torch.from_numpy(x).cuda() for x in _qkv(60 + i, 1, 8, 2, S, S)]
            t.append(torch.zeros_like(t[0]))
            data.append((S, t, [c.wrap(x.data_ptr(), x.numel() * 4) for x in t]))
        call = lambda S, b, fl: c.sdpa(*b, 1, 8, 2, S, S, 128, 1 / np.sqrt(128), flags=fl | B.FLAG_ATTN_CAUSAL)
        with _Tuned(backend, attn_prefill=1):
            torch.cuda.synchronize()
            for S, t, b in data:
                call(S, b, 0)
                want.append(t[3].cpu().numpy().copy())
                t[3].zero_()
            torch.cuda.synchronize()
            for _ in range(3):
                for st, (S, t, b) in zip(streams, data):
                    c.set_stream(st.cuda_stream)
                    call(S, b, B.FLAG_NO_SYNC)
        torch.cuda.synchronize()
        for w, (S, t, b) in zip(want, data):
            assert np.array_equal(t[3].cpu().numpy().view(np.uint32), w.view(np.uint32))
    finally:
        c.set_stream(0)
        c.destroy()


class _Prompts:
    """Prompts of several lengths on the GPU, each with the bits that it has alone."""

    def __init__(self, backend, lengths, H=8, Hkv=2):
        import torch
        self.torch, self.c, self.H, self.Hkv = torch, backend.create_context(0), H, Hkv
        self.data = []
        for i, S in enumerate(lengths):
            t = [torch.from_numpy(x).cuda() for x in _qkv(80 + i, 1, H, Hkv, S, S)]
            t.append(torch.zeros_like(t[0]))
            self.data.append((S, t, [self.c.wrap(x.data_ptr(), x.numel() * 4) for x in t]))
        torch.cuda.synchronize()
        self.want = []
        for i in range(len(lengths)):
            self.call(i, 0)
            self.want.append(self.data[i][1][3].cpu().numpy().view(np.uint32).copy())
            self.data[i][1][3].zero_()
        torch.cuda.synchronize()

    def call(self, i, flags=B.FLAG_NO_SYNC):
        S, _, b = self.data[i]
        self.c.sdpa(*b, 1, self.H, self.Hkv, S, S, 128, 1 / np.sqrt(128), flags=flags | B.FLAG_ATTN_CAUSAL)

    def check(self):
        self.torch.cuda.synchronize()
        for (_, t, _), w in zip(self.data, self.want):
            assert np.array_equal(t[3].cpu().numpy().view(np.uint32), w)

    def check_nothing_ran(self):
        self.torch.cuda.synchronize()
        assert not any(t[3].any().item() for _, t, _ in self.data)

    def clear(self):
        for _, t, _ in self.data:
            t[3].zero_()
        self.torch.cuda.synchronize()

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.torch.cuda.synchronize()
        self.c.set_stream(0)
        self.c.destroy()


def test_order_of_the_scratch_survives_a_capture_and_a_blocking_call(backend):
    """A long prompt on one stream; then on another, the context having been on a capturing stream or in a blocking
    call in between, a short one: it still begins behind the first."""
    with _Tuned(backend, attn_prefill=1), _Prompts(backend, (4000, 700, 130), H=16, Hkv=4) as pr:
        torch = pr.torch
        for between in ("capture", "blocking", "same handle"):
            a, b = torch.cuda.Stream(), torch.cuda.Stream()
            other = torch.zeros(1 << 20, device="cuda")
            ob = pr.c.wrap(other.data_ptr(), other.numel() * 4)
            pr.clear()
            pr.c.set_stream(a.cuda_stream)
            for _ in range(4):
                pr.call(0)
            if between == "capture":
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=b, capture_error_mode="relaxed"):
                    pr.c.set_stream(b.cuda_stream)
                    pr.c.rope_precompute_cache(ob, ob, 16, 128, 1e4, B.FLAG_NO_SYNC)
            elif between == "blocking":
                pr.c.set_stream(b.cuda_stream)
                pr.c.rope_precompute_cache(ob, ob, 16, 128, 1e4, 0)
            else:
                pr.c.set_stream(b.cuda_stream)
                pr.c.set_stream(b.cuda_stream)
            pr.call(1)
            pr.call(2)
            pr.check()


def test_replayed_prompts_and_direct_ones_share_nothing(backend):
    """Graphs that hold prompts are replayed on one stream, others, and direct calls, run beside them: every output keeps
    the bits that its call has alone.  What a graph had is given back when it is gone."""
    with _Tuned(backend, attn_prefill=1), _Prompts(backend, (3000, 900, 130, 2000), H=16, Hkv=4) as pr:
        torch = pr.torch
        a, b, c = (torch.cuda.Stream() for _ in range(3))
        def capture(stream, prompts):
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=stream):
                pr.c.set_stream(stream.cuda_stream)
                for i in prompts:
                    pr.call(i)
            return g
        free = []
        for _ in range(3):
            pr.clear()
            ga, gb = capture(a, (2, 0)), capture(b, (1,))           # the longer one last: a larger scratch for the same stream
            pr.check_nothing_ran()
            for _ in range(3):
                with torch.cuda.stream(a):
                    ga.replay()
                with torch.cuda.stream(b):
                    gb.replay()
                pr.c.set_stream(c.cuda_stream)
                pr.call(3)
            pr.check()
            del ga, gb
            torch.cuda.synchronize()
            pr.c.set_stream(c.cuda_stream)
            pr.call(2, 0)
            free.append(torch.cuda.mem_get_info()[0])
        assert free[1] == free[2]


def test_a_capture_that_forks_has_a_scratch_for_each_branch(backend):
    """Two streams within one capture: the branches run side by side in a replay."""
    with _Tuned(backend, attn_prefill=1), _Prompts(backend, (1500, 1400), H=4, Hkv=2) as pr:
        torch = pr.torch
        a, b = torch.cuda.Stream(), torch.cuda.Stream()
        pr.clear()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=a):
            b.wait_stream(a)
            pr.c.set_stream(b.cuda_stream)
            pr.call(1)
            pr.c.set_stream(a.cuda_stream)
            pr.call(0)
            a.wait_stream(b)
        for _ in range(3):
            pr.clear()
            g.replay()
            pr.check()


def test_a_context_takes_the_scratch_with_its_first_prompt(backend):
    """A host that never runs prompt attention does not pay for its scratch; one call takes it, the next no more."""
    import torch
    free = lambda: (torch.cuda.synchronize(), torch.cuda.mem_get_info()[0])[1]
    q, k, v = _qkv(70, 1, 2, 1, 64, 64)
    warm = backend.create_context(0)                 # what the first context of a process sets up
    warm.destroy()
    before = free()
    c = backend.create_context(0)
    try:
        created = before - free()
        assert created < 64 << 20
        with _Tuned(backend, attn_prefill=1):
            _sdpa(c, q, k, v, True)
            first = before - free()
            assert first >= 131072 * 1536
            _sdpa(c, q, k, v, True)
            assert before - free() == first
    finally:
        c.destroy()
    assert before - free() < 32 << 20


@pytest.mark.parametrize("gain", [1e-6, 1.0, 1e7])
def test_a_row_with_one_key_is_its_value_bit_for_bit(ctx, backend, gain):
    """The first row of a causal prompt, and a row whose other keys weigh nothing, are that key's V; the log-sum-exp of such a row
    is its score, to the rounding of the score and of a product by ln 2."""
    q, k, v = _qkv(90, 2, 4, 2, 200, 200)
    v *= np.float32(gain)
    q[:, :, 150] = 0
    q[:, :, 150, 0] = 4000.0
    k[:, :, :, 0] = np.where(np.arange(200) == 77, 3.0, -1.0)            # scores of about 1060 and -350
    q[:, :, 0, 0] = 0
    with _Tuned(backend, attn_prefill=1):
        got, lse = _sdpa(ctx, q, k, v, True)
    assert np.array_equal(got[:, :, 0].view(np.uint32), np.repeat(v[:, :, 0], 2, axis=1).view(np.uint32))
    assert np.array_equal(got[:, :, 150].view(np.uint32), np.repeat(v[:, :, 77], 2, axis=1).view(np.uint32))
    want = np.einsum("bhd,bhd->bh", q[:, :, 0].astype(np.float64), np.repeat(k[:, :, 0], 2, axis=1).astype(np.float64)) / np.sqrt(128)
    # a score is a sum of 128 products of N(0, 1) values, 1 / 11 each, with an error of 2^-24 of its largest partial sums (below 4)
    np.testing.assert_allclose(lse[:, :, 0], want, rtol=0, atol=4 * 4 * 2.0 ** -24)


@pytest.mark.parametrize("peak", [1.0, 6.0])
def test_outputs_have_no_mean_error(ctx, backend, peak):
    """What the tensor core's chains cut off is added back: over many rows with so many keys the outputs are neither too large
    nor too small by more than 2e-8 of themselves (3 to 8e-8 if it were not; a row of ones is off by up to 9e-8 where the
    denominator carries the correction).  The mean of 2^18 errors of 3e-7 at most is known to 1e-9."""
    q, k, v = _qkv(91, 4, 16, 16, 256, 256)
    q *= np.float32(peak)
    with _Tuned(backend, attn_prefill=1):
        got, _ = _sdpa(ctx, q, k, v, True)
    want = _sdpa64(q, k, v, True)
    for lo, hi in ((1, 32), (32, 64), (64, 128), (128, 256)):
        w, e = want[:, :, lo:hi], got[:, :, lo:hi] - want[:, :, lo:hi]
        assert abs((e * w).sum() / (w * w).sum()) < 2e-8, (lo, hi)


@pytest.mark.parametrize("tiles", [1, 2, 5])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("B_,H,Hkv,Sq,Skv", [(1, 2, 2, 127, 128), (1, 1, 1, 129, 191), (2, 4, 2, 65, 65), (1, 5, 1, 300, 640), (1, 3, 3, 257, 449), (1, 8, 2, 385, 1000),
                                             (1, 2, 2, 500, 130), (2, 2, 1, 70, 0)])
def test_passes_over_ranges_of_the_keys(ctx, backend, B_, H, Hkv, Sq, Skv, causal, tiles):
    """So many key tiles per pass, blocks carrying what they have from one to the next: blocks that see no key of a pass, passes that end
    inside a block's diagonal, odd pairs; against 64 bits, and the log-sum-exp against one pass."""
    q, k, v = _qkv(Sq + Skv + tiles, B_, H, Hkv, Sq, Skv)
    with _Tuned(backend, attn_prefill=1):
        one, one_lse = _sdpa(ctx, q, k, v, causal)
    before = backend.launch_count()
    with _Tuned(backend, attn_prefill=1, attn_pass_tiles=tiles):
        got, lse = _sdpa(ctx, q, k, v, causal)
        assert backend.last_kernel_name() == "lux_attn_prefill_mma_f32" and ctx.last_device_status() == 0
    seen = -(-(min(Sq, Skv) if causal else Skv) // 64)
    assert backend.launch_count() - before == (2 * -(-seen // tiles) if seen else 1)
    if not Skv:
        assert not got.any()
        return
    assert orc.rel_l2(got, _sdpa64(q, k, v, causal)) < TOL
    np.testing.assert_allclose(lse, one_lse, rtol=2.0 ** -22, atol=2.0 ** -22)      # four roundings each


@pytest.mark.parametrize("tiles", [1, 3])
def test_passes_keep_what_one_pass_keeps(ctx, backend, tiles):
    """The tests above on ranges, extremes and fallbacks, with their bounds, in passes."""
    with _Tuned(backend, attn_pass_tiles=tiles):
        for bad in (np.nan, np.inf):
            test_values_a_row_must_not_see_do_not_reach_it(ctx, backend, bad)
        for row in (0, 77, 149):
            test_a_non_finite_query_is_noticed_by_every_warp(ctx, backend, row, np.nan)
        test_no_keys_and_large_scores(ctx, backend, 1)
        test_magnitudes_far_apart(ctx, backend)
        for key in (63, 149):
            for factor in (1e5, 1e30):
                test_large_finite_values_behind_the_mask_do_not_reach_earlier_rows(ctx, backend, key, factor)
        for lo, hi in ((-6, 12), (-30, 0)):
            test_keys_of_very_different_magnitude(ctx, backend, lo, hi)
        for drop in (14, 30, 80):
            test_small_weights_under_a_dominant_key_without_a_value(ctx, backend, drop)
        for scale in (1e-28, 1e-31, 1e-37):
            for columns in (slice(None), slice(5, 6)):
                test_values_close_to_the_smallest_normal_number(ctx, backend, scale, columns)
        for qs, ks in ((1e15, 1e-15), (1e-37, 1e37)):
            test_scores_of_ordinary_size_from_extreme_operands(ctx, backend, qs, ks)
        for value in (np.float32(1), np.float32(3e-30)):
            test_a_constant_v_comes_back(ctx, backend, value)
        for where, bad in (("q", np.nan), ("k", np.inf), ("v", np.nan), ("v", 1e30)):
            test_a_block_out_of_range_leaves_the_others_alone(ctx, backend, where, bad)
            test_an_odd_pair_with_one_block_out_of_range(ctx, backend, where)
        test_output_over_the_queries(ctx, backend)
        test_replays_of_a_captured_call_do_not_remember(backend)
        test_a_row_with_one_key_is_its_value_bit_for_bit(ctx, backend, 1.0)
        test_outputs_have_no_mean_error(ctx, backend, 1.0)
