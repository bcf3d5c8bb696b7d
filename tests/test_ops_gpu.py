"""Parity of every kernel entry point with the CPU oracle, through the C ABI.

Bit-exact for integer/byte work (dequantisation, f16 cache rows, argmax);
fp32 results differ from the oracle only by summation order, so they are held
to a relative-L2 of 1e-5 and a max-abs of 1e-4 of the largest output -- two
orders tighter than the end-to-end logits tolerance (max-abs 1e-2, rel-L2 1e-3).
"""
import ctypes as C

import numpy as np
import pytest

import oracle_bind as ob
import quant_np as qn

pytestmark = pytest.mark.gpu

HEADS, ROT = 32, 128
DIM = HEADS * ROT


def close(got, want, rel_l2=1e-5, max_abs_frac=1e-4):
    got, want = np.asarray(got, np.float64).ravel(), np.asarray(want, np.float64).ravel()
    assert got.shape == want.shape
    assert np.all(np.isfinite(got))
    denom = np.linalg.norm(want) or 1.0
    l2 = np.linalg.norm(got - want) / denom
    mx = np.abs(got - want).max()
    assert l2 <= rel_l2, f"rel-L2 {l2:.3e}"
    assert mx <= max_abs_frac * (np.abs(want).max() or 1.0), f"max-abs {mx:.3e}"


def workers_for(cols):
    return 32 if cols == 5120 else 128      # llava_session.cpp:357-371


def u32_dev(gpu, value):
    return gpu.upload(np.array([value, value, value, value], np.uint32))   # config_buffer: token_count x4


@pytest.mark.parametrize("wtype", [qn.Q4_0, qn.Q8_0])
def test_dequant_rows_bit_exact(gpu, pkg, wtype):
    rng = np.random.default_rng(20)
    vocab, cols = 64, 4096
    table = qn.quantize((rng.standard_normal((vocab, cols)) * 0.02).astype(np.float32), wtype)
    ids = np.array([0, 63, 17, 17, 5], np.uint32)
    d_out = gpu.alloc(ids.size * cols * 4)
    pkg.check(gpu.lib.lv_dequant_rows(gpu.handle, d_out, gpu.upload(table), wtype, gpu.upload(ids), None, cols, vocab, ids.size))
    gpu.sync()
    got = gpu.download(d_out, np.float32, ids.size * cols).reshape(ids.size, cols)
    rb = qn.row_bytes(wtype, cols)
    for z, t in enumerate(ids):
        want = ob.dequant(table[t * rb:(t + 1) * rb], wtype, cols)
        assert np.array_equal(got[z].view(np.uint32), want.view(np.uint32))
    # ids taken from a device-resident token log at a device-resident position
    pkg.check(gpu.lib.lv_dequant_rows(gpu.handle, d_out, gpu.upload(table), wtype, gpu.upload(ids), u32_dev(gpu, 2), cols, vocab, 2))
    gpu.sync()
    got = gpu.download(d_out, np.float32, 2 * cols).reshape(2, cols)
    for z, t in enumerate(ids[2:4]):
        assert np.array_equal(got[z], ob.dequant(table[t * rb:(t + 1) * rb], wtype, cols))


@pytest.mark.parametrize("dim,batch", [(4096, 1), (5120, 3)])
def test_norm(gpu, pkg, dim, batch):
    rng = np.random.default_rng(21)
    x = (rng.standard_normal((batch, dim)) * 3 + 0.2).astype(np.float32)
    w = (1 + 0.01 * rng.standard_normal(dim)).astype(np.float32)
    d_out = gpu.alloc(x.nbytes)
    pkg.check(gpu.lib.lv_norm_f32(gpu.handle, d_out, gpu.upload(x), gpu.upload(w), dim, batch))
    gpu.sync()
    got = gpu.download(d_out, np.float32, x.size).reshape(batch, dim)
    for z in range(batch):
        close(got[z], ob.norm(x[z], w), rel_l2=2e-6, max_abs_frac=2e-6)


@pytest.mark.parametrize("nbytes", [1, 4099, 128000, 256 * 1024, 256 * 1024 + 1, 1 << 20])
def test_download_through_either_way(gpu, pkg, nbytes):
    data = np.random.default_rng(nbytes).integers(0, 256, nbytes + 1, dtype=np.uint8)
    d, got = gpu.upload(data), np.full(nbytes + 2, 7, np.uint8)
    pkg.check(gpu.lib.lv_download(gpu.handle, C.c_void_p(got.ctypes.data + 1), pkg.offset(d, 1), nbytes))
    assert np.array_equal(got[1:-1], data[1:]) and got[0] == 7 and got[-1] == 7
    pinned = C.c_void_p()
    pkg.check(gpu.lib.lv_host_alloc(gpu.handle, nbytes + 2, C.byref(pinned)))
    got = np.frombuffer((C.c_uint8 * (nbytes + 2)).from_address(pinned.value), np.uint8)
    got[:] = 7
    pkg.check(gpu.lib.lv_download(gpu.handle, pkg.offset(pinned, 1), pkg.offset(d, 1), nbytes))
    assert np.array_equal(got[1:-1], data[1:]) and got[0] == 7 and got[-1] == 7
    del got
    pkg.check(gpu.lib.lv_host_free(gpu.handle, pinned))
    gpu.free(d)


GEMV_SHAPES = [
    (qn.Q4_0, 4096, 4096), (qn.Q4_0, 4096, 11008), (qn.Q4_0, 5120, 13824), (qn.Q4_0, 5120, 5120),
    (qn.Q4_0, 32000, 4096), (qn.Q8_0, 4096, 4096), (qn.Q8_0, 4096, 11008), (qn.Q8_0, 1024, 5120),
    (qn.Q4_0, 4, 256), (qn.Q8_0, 8, 512),
]


@pytest.mark.parametrize("wtype,rows,cols", GEMV_SHAPES)
def test_gemv_and_residual_add(gpu, pkg, wtype, rows, cols):
    rng = np.random.default_rng(rows + cols)
    W = qn.quantize((rng.standard_normal((rows, cols)) * 0.02).astype(np.float32), wtype)
    x = rng.standard_normal(cols).astype(np.float32)
    base = rng.standard_normal(rows).astype(np.float32)
    dW, dx = gpu.upload(W), gpu.upload(x)
    d_out = gpu.upload(base)
    pkg.check(gpu.lib.lv_gemv(gpu.handle, d_out, dW, wtype, dx, rows, cols, 1, 0))
    gpu.sync()
    want = ob.gemv(W, wtype, x, rows, cols, workers_for(cols))
    close(gpu.download(d_out, np.float32, rows), want)
    pkg.check(gpu.lib.lv_upload(gpu.handle, d_out, base.ctypes.data_as(C.c_void_p), base.nbytes))
    pkg.check(gpu.lib.lv_gemv(gpu.handle, d_out, dW, wtype, dx, rows, cols, 1, 1))      # matmul_add_*
    gpu.sync()
    close(gpu.download(d_out, np.float32, rows), base + want)
    for d in (dW, dx, d_out):
        gpu.free(d)


@pytest.mark.parametrize("rows,cols", [(4096, 4096), (4096, 11008), (5120, 13824), (8, 512)])
def test_gemv_on_version_1_blocks(gpu, pkg, rows, cols):
    """q4_0 as ggjt version 1 files store it (f32 scale, byte j = elements 2j and 2j+1; matmul_dim.comp / matmul_ff.comp
    without the _fp16 suffix, llava_buffer.cpp:193-224): plain, add-in-place, with a norm in front, and the SiLU pair."""
    rng = np.random.default_rng(rows * 3 + cols)
    W = qn.quantize_q4_0_v1((rng.standard_normal((rows, cols)) * 0.02).astype(np.float32))
    x = rng.standard_normal(cols).astype(np.float32)
    base = rng.standard_normal(rows).astype(np.float32)
    dW, dx, d_out = gpu.upload(W), gpu.upload(x), gpu.upload(base)
    want = ob.gemv(W, qn.Q4_0, x, rows, cols, workers_for(cols), version=1)
    pkg.check(gpu.lib.lv_gemv(gpu.handle, d_out, dW, qn.Q4_0_V1, dx, rows, cols, 1, 1))
    gpu.sync()
    close(gpu.download(d_out, np.float32, rows), base + want)
    nw = (1 + 0.01 * rng.standard_normal(cols)).astype(np.float32)
    pkg.check(gpu.lib.lv_norm_gemv(gpu.handle, d_out, dW, qn.Q4_0_V1, dx, gpu.upload(nw), rows, cols, 1))
    gpu.sync()
    close(gpu.download(d_out, np.float32, rows), ob.gemv(W, qn.Q4_0, ob.norm(x, nw), rows, cols, workers_for(cols), version=1))
    if rows % 2 == 0 and rows >= 4096:
        half = rows // 2
        d_g = gpu.alloc(half * 4)
        rb = cols // 32 * 20
        pkg.check(gpu.lib.lv_gemv_silu(gpu.handle, d_g, dW, pkg.offset(dW, half * rb), qn.Q4_0_V1, dx, half, cols, 1))
        gpu.sync()
        close(gpu.download(d_g, np.float32, half), ob.gemv_silu(W[:half * rb], W[half * rb:], qn.Q4_0, x, half, cols, workers_for(cols), version=1))
        gpu.free(d_g)
    for d in (dW, dx, d_out):
        gpu.free(d)


def test_dequant_rows_of_version_1_blocks_bit_exact(gpu, pkg):
    rng = np.random.default_rng(41)
    vocab, cols = 64, 4096
    table = qn.quantize_q4_0_v1((rng.standard_normal((vocab, cols)) * 0.02).astype(np.float32))
    ids = np.array([5, 0, 63, 17], np.uint32)
    d_out = gpu.alloc(ids.size * cols * 4)
    pkg.check(gpu.lib.lv_dequant_rows(gpu.handle, d_out, gpu.upload(table), qn.Q4_0_V1, gpu.upload(ids), None, cols, vocab, ids.size))
    gpu.sync()
    got = gpu.download(d_out, np.float32, ids.size * cols).reshape(ids.size, cols)
    rb = cols // 32 * 20
    for z, t in enumerate(ids):
        assert np.array_equal(got[z].view(np.uint32), ob.dequant(table[t * rb:(t + 1) * rb], qn.Q4_0, cols, version=1).view(np.uint32))


def _outlier_activations(rng, cols):
    """Activations as a trained LLaMA's residual stream has them: a few channels two to three orders of
    magnitude above the rest -- alone in a 32-block, several in one block, in many blocks -- plus an
    all-zero block and a block of denormals.  The GEMV stores each block of activations as fixed point
    relative to the block's largest magnitude, so these are the inputs that stress it most."""
    x = rng.standard_normal(cols).astype(np.float32)
    x[5] *= 1000.0                                   # one outlier alone in its block
    x[64:96:7] *= 300.0                              # several in one block
    x[3 * 32 + 1] = -850.0
    x[np.arange(7, cols, 416)] *= 120.0              # spread over many blocks
    x[10 * 32:11 * 32] = 0.0                         # an all-zero block
    x[12 * 32:13 * 32] = (rng.standard_normal(32) * 1e-41).astype(np.float32)    # denormals only
    x[14 * 32:15 * 32] = 0.0
    x[14 * 32 + 9] = 512.0                           # a block that is one outlier and nothing else
    return x


@pytest.mark.parametrize("wtype,rows,cols", [(qn.Q4_0, 4096, 4096), (qn.Q4_0, 4096, 11008), (qn.Q8_0, 4096, 4096), (qn.Q8_0, 1024, 11008)])
def test_gemv_with_outlier_activations(gpu, pkg, wtype, rows, cols):
    rng = np.random.default_rng(77 + rows + cols + wtype)
    W = qn.quantize((rng.standard_normal((rows, cols)) * 0.02).astype(np.float32), wtype)
    x = _outlier_activations(rng, cols)
    dW, dx = gpu.upload(W), gpu.upload(x)
    d_out = gpu.alloc(rows * 4)
    pkg.check(gpu.lib.lv_gemv(gpu.handle, d_out, dW, wtype, dx, rows, cols, 1, 0))
    gpu.sync()
    close(gpu.download(d_out, np.float32, rows), ob.gemv(W, wtype, x, rows, cols, workers_for(cols)))
    for d in (dW, dx, d_out):
        gpu.free(d)


def test_norm_gate_up_silu_with_outlier_activations(gpu, pkg):
    rng = np.random.default_rng(78)
    ff, dim = 11008, 4096
    w3 = qn.quantize_q4_0((rng.standard_normal((ff, dim)) * 0.02).astype(np.float32))
    w1 = qn.quantize_q4_0((rng.standard_normal((ff, dim)) * 0.02).astype(np.float32))
    x = _outlier_activations(rng, dim)
    nw = (1 + 0.01 * rng.standard_normal(dim)).astype(np.float32)
    d_out = gpu.alloc(ff * 4)
    pkg.check(gpu.lib.lv_norm_gate_up_silu(gpu.handle, d_out, gpu.upload(w3), gpu.upload(w1), qn.Q4_0, gpu.upload(x), gpu.upload(nw), ff, dim, 1))
    gpu.sync()
    close(gpu.download(d_out, np.float32, ff), ob.gemv_silu(w3, w1, qn.Q4_0, ob.norm(x, nw), ff, dim, 128))


@pytest.mark.parametrize("wtype,ff,dim", [(qn.Q4_0, 11008, 4096), (qn.Q8_0, 11008, 4096), (qn.Q4_0, 13824, 5120)])
def test_gemv_silu(gpu, pkg, wtype, ff, dim):
    rng = np.random.default_rng(ff)
    w3 = qn.quantize((rng.standard_normal((ff, dim)) * 0.02).astype(np.float32), wtype)
    w1 = qn.quantize((rng.standard_normal((ff, dim)) * 0.02).astype(np.float32), wtype)
    x = rng.standard_normal(dim).astype(np.float32)
    d3, d1, dx = gpu.upload(w3), gpu.upload(w1), gpu.upload(x)
    d_out = gpu.alloc(ff * 4)
    pkg.check(gpu.lib.lv_gemv_silu(gpu.handle, d_out, d3, d1, wtype, dx, ff, dim, 1))
    gpu.sync()
    close(gpu.download(d_out, np.float32, ff), ob.gemv_silu(w3, w1, wtype, x, ff, dim, workers_for(dim)))
    for d in (d3, d1, dx, d_out):
        gpu.free(d)


def test_gemv_batch_rows_are_independent(gpu, pkg):
    rng = np.random.default_rng(22)
    rows, cols, batch = 512, 4096, 3
    W = qn.quantize_q4_0((rng.standard_normal((rows, cols)) * 0.02).astype(np.float32))
    x = rng.standard_normal((batch, cols)).astype(np.float32)
    d_out = gpu.alloc(batch * rows * 4)
    pkg.check(gpu.lib.lv_gemv(gpu.handle, d_out, gpu.upload(W), qn.Q4_0, gpu.upload(x), rows, cols, batch, 0))
    gpu.sync()
    got = gpu.download(d_out, np.float32, batch * rows).reshape(batch, rows)
    for z in range(batch):
        close(got[z], ob.gemv(W, qn.Q4_0, x[z], rows, cols, 128))


def test_norm_fused_gemv_matches_norm_then_gemv(gpu, pkg):
    rng = np.random.default_rng(23)
    rows, cols = 1024, 4096
    W = qn.quantize_q4_0((rng.standard_normal((rows, cols)) * 0.02).astype(np.float32))
    x = (rng.standard_normal(cols) * 2).astype(np.float32)
    nw = (1 + 0.01 * rng.standard_normal(cols)).astype(np.float32)
    d_out = gpu.alloc(rows * 4)
    pkg.check(gpu.lib.lv_norm_gemv(gpu.handle, d_out, gpu.upload(W), qn.Q4_0, gpu.upload(x), gpu.upload(nw), rows, cols, 1))
    gpu.sync()
    close(gpu.download(d_out, np.float32, rows), ob.gemv(W, qn.Q4_0, ob.norm(x, nw), rows, cols, 128))


def test_gemv_rejects_bad_arguments(gpu, pkg):
    lib = gpu.lib
    d = gpu.alloc(4096)
    assert lib.lv_gemv(gpu.handle, d, d, 3, d, 4, 256, 1, 0) == pkg.LV_ERR_BAD_ARGUMENTS        # q4_1 unsupported
    assert lib.lv_gemv(gpu.handle, d, d, qn.Q4_0, d, 4, 96, 1, 0) == pkg.LV_ERR_BAD_ARGUMENTS   # cols % 256
    assert lib.lv_gemv(gpu.handle, d, d, qn.Q4_0, d, 6, 256, 1, 0) == pkg.LV_ERR_BAD_ARGUMENTS  # rows % 4
    assert lib.lv_gemv(gpu.handle, d, pkg.offset(d, 2), qn.Q4_0, d, 4, 256, 1, 0) == pkg.LV_ERR_BAD_ARGUMENTS
    assert lib.lv_gemv(None, d, d, qn.Q4_0, d, 4, 256, 1, 0) == pkg.LV_ERR_BAD_ARGUMENTS
    assert b"" != lib.lv_last_error_string()


def test_kv_append_bit_exact(gpu, pkg):
    rng = np.random.default_rng(24)
    batch, ctx_rows, pos = 3, 16, 5
    x = np.concatenate([rng.standard_normal((batch, DIM - 6)) * 2, np.tile([1e-7, 65519.0, 7e4, -0.0, 6.1e-5, 1.0009766], (batch, 1))], 1).astype(np.float32)
    cache = gpu.zeros(ctx_rows * DIM * 2)
    pkg.check(gpu.lib.lv_kv_append_f16(gpu.handle, cache, gpu.upload(x), u32_dev(gpu, pos), DIM, batch, ctx_rows))
    gpu.sync()
    got = gpu.download(cache, np.uint16, ctx_rows * DIM).reshape(ctx_rows, DIM)
    want = np.zeros((ctx_rows, DIM), np.uint16)
    with np.errstate(over="ignore"):
        want[pos:pos + batch] = x.astype(np.float16).view(np.uint16)
    assert np.array_equal(got, want)
    assert np.array_equal(want[pos], ob.f32_to_f16_bits(x[0]))
    # a row outside the cache is refused and reported, never written
    pkg.check(gpu.lib.lv_kv_append_f16(gpu.handle, cache, gpu.upload(x), u32_dev(gpu, ctx_rows - 1), DIM, batch, ctx_rows))
    with pytest.raises(pkg.LvError) as e:
        gpu.sync()
    assert e.value.code == pkg.LV_ERR_DEVICE_WAIT
    gpu.sync()      # the error word was cleared


def _caches(rng, n, rows):
    k = np.zeros((rows, DIM), np.float16)
    v = np.zeros((rows, DIM), np.float16)
    k[:n] = (rng.standard_normal((n, DIM)) * 0.7).astype(np.float16)
    v[:n] = (rng.standard_normal((n, DIM)) * 0.7).astype(np.float16)
    return k.view(np.uint16), v.view(np.uint16)


@pytest.fixture(scope="module")
def rope_table(gpu, pkg):
    t = gpu.alloc(2048 * ROT * 4)
    pkg.check(gpu.lib.lv_rope_table_build(gpu.handle, t, 2048, ROT))
    return t


@pytest.mark.parametrize("pos,backlog", [(0, 128), (1, 128), (63, 128), (64, 128), (127, 128), (300, 512)])
def test_three_attention_ops_match_reference_shaders(gpu, pkg, rope_table, pos, backlog):
    rng = np.random.default_rng(100 + pos)
    k, v = _caches(rng, pos + 1, backlog)
    q = rng.standard_normal(DIM).astype(np.float32)
    lib, h = gpu.lib, gpu.handle
    dk, dv, dq, dpos = gpu.upload(k), gpu.upload(v), gpu.upload(q), u32_dev(gpu, pos)
    d_scores = gpu.alloc(backlog * HEADS * 4)
    d_out = gpu.alloc(DIM * 4)
    pkg.check(lib.lv_attn_scores_rope(h, d_scores, dk, dq, dpos, rope_table, backlog, HEADS, ROT, 1))
    gpu.sync()
    scores = gpu.download(d_scores, np.float32, backlog * HEADS).reshape(backlog, HEADS)
    want_scores = ob.mhsa(k, q, pos, HEADS, ROT)
    close(scores[: pos + 1], want_scores, rel_l2=2e-6, max_abs_frac=1e-5)
    assert np.all(scores[pos + 1:] == 0)
    pkg.check(lib.lv_softmax_masked(h, d_scores, dpos, backlog, HEADS, ROT, 1))
    gpu.sync()
    probs = gpu.download(d_scores, np.float32, backlog * HEADS).reshape(backlog, HEADS)
    want_probs = ob.softmax(want_scores, pos, backlog, HEADS, ROT)
    close(probs, want_probs, rel_l2=5e-6, max_abs_frac=1e-5)
    assert np.all(probs[pos + 1:] == 0)
    pkg.check(lib.lv_attn_values(h, d_out, dv, d_scores, backlog, HEADS, ROT, 1))
    gpu.sync()
    close(gpu.download(d_out, np.float32, DIM), ob.kqv(v, want_probs, backlog, HEADS, ROT), rel_l2=5e-6, max_abs_frac=2e-5)
    for d in (dk, dv, dq, d_scores, d_out):
        gpu.free(d)


@pytest.mark.parametrize("grid", ["whole-cache", "backlog"])
@pytest.mark.parametrize("pos", [0, 1, 31, 32, 63, 64, 65, 127, 128, 255, 256, 300, 511, 1023, 1500, 2047])
def test_fused_attention(gpu, pkg, rope_table, pos, grid):
    """grid "whole-cache": one CTA per 256 rows of the 2048-row cache (more CTAs than SMs: the variant with
    the compact rotation table); "backlog": only the current backlog, as a session launches it (at most
    one CTA per SM up to a backlog of 1024: exact table rows staged)."""
    rng = np.random.default_rng(200 + pos)
    backlog = 128
    while backlog <= pos:
        backlog *= 2
    max_ctx = 2048 if grid == "whole-cache" else backlog
    k, v = _caches(rng, pos + 1, max_ctx)
    q = rng.standard_normal(DIM).astype(np.float32)
    nbytes = gpu.lib.lv_attention_scratch_bytes(HEADS, ROT, max_ctx, 1)
    assert nbytes > 0
    scratch = gpu.zeros(nbytes)
    dk, dv, dq = gpu.upload(k), gpu.upload(v), gpu.upload(q)
    d_out = gpu.alloc(DIM * 4)
    want = ob.attention(k, v, q, pos, backlog, HEADS, ROT)
    for _ in range(2):       # the second launch proves the arrival counters were reset
        pkg.check(gpu.lib.lv_memset(gpu.handle, d_out, 0xFF, DIM * 4))
        pkg.check(gpu.lib.lv_attention_fused(gpu.handle, d_out, dq, dk, dv, u32_dev(gpu, pos), rope_table, scratch,
                                             HEADS, ROT, max_ctx, 1))
        gpu.sync()
        # grids with more CTAs than SMs (here: the 2048-row cache) form cos/sin of a distance from two table
        # rows; a few units in the last place per rotation add up over two thousand rows
        close(gpu.download(d_out, np.float32, DIM), want, rel_l2=5e-6 if max_ctx < 2048 else 1e-5, max_abs_frac=2e-5)
    for d in (dk, dv, dq, d_out, scratch):
        gpu.free(d)


def test_fused_attention_refuses_a_position_outside_the_cache(gpu, pkg, rope_table):
    """A position word at or beyond max_ctx would index past the caches and the rotation table: the kernel
    reports it through the error word and writes nothing (like lv_kv_append_f16), and the arrival counters
    stay clear, so the next call with a valid position is unaffected."""
    rng = np.random.default_rng(32)
    for batch, max_ctx in ((1, 256), (6, 512)):         # one CTA per SM / the two-CTAs-per-SM variant
        k, v = _caches(rng, max_ctx, max_ctx)
        q = rng.standard_normal((batch, DIM)).astype(np.float32)
        scratch = gpu.zeros(gpu.lib.lv_attention_scratch_bytes(HEADS, ROT, max_ctx, batch))
        dk, dv, dq = gpu.upload(k), gpu.upload(v), gpu.upload(q)
        d_out = gpu.alloc(batch * DIM * 4)
        pkg.check(gpu.lib.lv_memset(gpu.handle, d_out, 0xA5, batch * DIM * 4))
        pkg.check(gpu.lib.lv_attention_fused(gpu.handle, d_out, dq, dk, dv, u32_dev(gpu, max_ctx), rope_table, scratch, HEADS, ROT, max_ctx, batch))
        with pytest.raises(pkg.LvError) as e:
            gpu.sync()
        assert e.value.code == pkg.LV_ERR_DEVICE_WAIT
        assert np.all(gpu.download(d_out, np.uint8, batch * DIM * 4) == 0xA5)
        # the refused call left no trace: the next one, with every row of the batch inside the cache, is correct
        pos = max_ctx - batch
        pkg.check(gpu.lib.lv_attention_fused(gpu.handle, d_out, dq, dk, dv, u32_dev(gpu, pos), rope_table, scratch, HEADS, ROT, max_ctx, batch))
        gpu.sync()
        got = gpu.download(d_out, np.float32, batch * DIM).reshape(batch, DIM)
        for z in range(batch):
            close(got[z], ob.attention(k, v, q[z], pos + z, max_ctx, HEADS, ROT), rel_l2=1e-5, max_abs_frac=2e-5)
        for d in (dk, dv, dq, d_out, scratch):
            gpu.free(d)


def test_fused_attention_batch_is_causal(gpu, pkg, rope_table):
    rng = np.random.default_rng(31)
    batch, pos, max_ctx = 4, 70, 256
    k, v = _caches(rng, pos + batch, max_ctx)
    q = rng.standard_normal((batch, DIM)).astype(np.float32)
    scratch = gpu.zeros(gpu.lib.lv_attention_scratch_bytes(HEADS, ROT, max_ctx, batch))
    d_out = gpu.alloc(batch * DIM * 4)
    pkg.check(gpu.lib.lv_attention_fused(gpu.handle, d_out, gpu.upload(q), gpu.upload(k), gpu.upload(v), u32_dev(gpu, pos),
                                         rope_table, scratch, HEADS, ROT, max_ctx, batch))
    gpu.sync()
    got = gpu.download(d_out, np.float32, batch * DIM).reshape(batch, DIM)
    for z in range(batch):       # row z sees cache rows 0 .. pos + z (softmax.comp:35)
        close(got[z], ob.attention(k, v, q[z], pos + z, 128, HEADS, ROT), rel_l2=5e-6, max_abs_frac=2e-5)


@pytest.mark.parametrize("batch,pos,max_ctx", [(12, 0, 128), (64, 0, 128), (16, 120, 256), (17, 111, 128), (64, 64, 128), (33, 300, 512), (64, 512, 1024), (50, 974, 1024),
                                               (9, 1015, 2048), (64, 1984, 2048), (63, 1985, 2048), (70, 90, 256), (130, 640, 1024), (12, 19, 31),
                                               (13, 100, 128), (14, 0, 128), (14, 16, 31), (18, 238, 256), (19, 1, 257)])
def test_prompt_attention(gpu, pkg, rope_table, batch, pos, max_ctx):
    """Steps of many rows go through the matrix products of attention_prompt.cu: chunks of 128 keys that end inside a block of 16, one or
    several CTAs and passes per head, one or several tiles of 64 rows.  Bounds as for the compact table of test_fused_attention: the angle of
    a distance of 2000 is an f32 with half an ulp of 2^-14, and the sum of two angles rounds elsewhere than the angle of the sum, which
    for queries of at most unit size moves scores by about 1e-5."""
    rng = np.random.default_rng(500 + batch + pos)
    k, v = _caches(rng, pos + batch, max_ctx)
    q = (rng.standard_normal((batch, DIM)) * np.exp2(rng.integers(-12, 1, (batch, 1)))).astype(np.float32)
    q[0, :ROT] = 0                                          # a head's query of zeros weighs its keys equally
    dk, dv, dq = gpu.upload(k), gpu.upload(v), gpu.upload(q)
    d_out, scratch = gpu.alloc((batch + 1) * DIM * 4), gpu.zeros(gpu.lib.lv_attention_scratch_bytes(HEADS, ROT, max_ctx, batch))
    pkg.check(gpu.lib.lv_memset(gpu.handle, d_out, 0xFF, (batch + 1) * DIM * 4))
    pkg.check(gpu.lib.lv_attention_fused(gpu.handle, d_out, dq, dk, dv, u32_dev(gpu, pos), rope_table, scratch, HEADS, ROT, max_ctx, batch))
    gpu.sync()
    got = gpu.download(d_out, np.float32, (batch + 1) * DIM).reshape(batch + 1, DIM)
    assert np.all(got[batch].view(np.uint32) == 0xFFFFFFFF)
    backlog = 128
    while backlog < pos + batch:
        backlog *= 2
    for z in sorted({0, 1, 7, min(15, batch - 1), batch // 2, batch - 2, batch - 1}):
        close(got[z], ob.attention(k, v, q[z], pos + z, backlog, HEADS, ROT), rel_l2=1e-5, max_abs_frac=2e-5)
    for d in (dk, dv, dq, d_out, scratch):
        gpu.free(d)


def exact_attention(table, k, v, q, P):
    """One row over positions 0 .. P in 64 bits, turned by the rows of the rotation table."""
    heads = q.size // ROT
    kk = k[:P + 1].view(np.float16).astype(np.float64).reshape(P + 1, heads, ROT // 2, 2)
    t = table[P - np.arange(P + 1)].astype(np.float64)[:, None]
    turned = np.stack([t[..., 0] * kk[..., 0] + t[..., 1] * kk[..., 1], t[..., 0] * kk[..., 1] - t[..., 1] * kk[..., 0]], -1).reshape(P + 1, heads, ROT)
    s = np.einsum("hd,phd->ph", q.astype(np.float64).reshape(heads, ROT), turned) / np.sqrt(ROT)
    e = np.exp(s - s.max(0))
    return np.einsum("ph,phd->hd", e / e.sum(0), v[:P + 1].view(np.float16).astype(np.float64).reshape(P + 1, heads, ROT)).ravel()


@pytest.mark.parametrize("batch,pos", [(64, 0), (50, 60)])
@pytest.mark.parametrize("size", [1.0, 1e-2, 1e-3, 2.0 ** -14, 30.0, 2.0 ** 12])
def test_prompt_attention_of_small_and_large_keys(gpu, pkg, rope_table, batch, pos, size):
    """Keys of any size of f16, with queries that make scores of a few units, are as exact as f32 sums make them: scores of 128 products, the
    rounding of the table's angles (2^-19 at distances of up to 63) and the sums of the weighted values each leave about 2^-23."""
    rng = np.random.default_rng(700 + batch)
    max_ctx = 128
    k, v = _caches(rng, pos + batch, max_ctx)
    k = np.zeros((max_ctx, DIM), np.float16)
    k[:pos + batch] = (rng.standard_normal((pos + batch, DIM)) * size).astype(np.float16)
    q = (rng.standard_normal((batch, DIM)) / size).astype(np.float32)
    q[0, :ROT] *= np.float32(1e-30)                         # scores of next to nothing
    d_out, scratch = gpu.alloc(batch * DIM * 4), gpu.zeros(gpu.lib.lv_attention_scratch_bytes(HEADS, ROT, max_ctx, batch))
    args = [gpu.upload(a) for a in (q, k.view(np.uint16), v)]
    pkg.check(gpu.lib.lv_attention_fused(gpu.handle, d_out, *args, u32_dev(gpu, pos), rope_table, scratch, HEADS, ROT, max_ctx, batch))
    gpu.sync()
    got = gpu.download(d_out, np.float32, batch * DIM).reshape(batch, DIM)
    table = gpu.download(rope_table, np.float32, 128 * ROT).reshape(128, ROT // 2, 2)
    for z in sorted({0, 1, 17, batch // 2, batch - 1}):
        close(got[z], exact_attention(table, k.view(np.uint16), v, q[z], pos + z), rel_l2=7e-7, max_abs_frac=3e-6)
    for d in args + [d_out, scratch]:
        gpu.free(d)


@pytest.mark.parametrize("batch,pos,max_ctx", [(64, 0, 128), (50, 100, 256), (64, 448, 512), (70, 90, 256), (64, 960, 1024)])
def test_prompt_attention_rows_do_not_depend_on_later_values(gpu, pkg, rope_table, batch, pos, max_ctx):
    """Values of the cache that are not finite (the append rounds to f16) reach the rows that see them, and no row before: against the same
    caches with 0 in their place every other output has the same bits."""
    rng = np.random.default_rng(600 + batch)
    k, v = _caches(rng, pos + batch, max_ctx)
    odd = [(pos + 3, 5, np.inf), (pos + 20, 5 + ROT, -np.inf), (pos + 21, 2 * ROT + 77, np.nan), (pos + batch - 1, 9, np.inf), (pos + batch - 1, 7 * ROT + 64, np.nan)]
    q = rng.standard_normal((batch, DIM)).astype(np.float32)
    dk, dq, at = gpu.upload(k), gpu.upload(q), u32_dev(gpu, pos)
    scratch, d_out = gpu.zeros(gpu.lib.lv_attention_scratch_bytes(HEADS, ROT, max_ctx, batch)), gpu.alloc(batch * DIM * 4)
    got = []
    for put in (False, True):
        w = v.copy().view(np.float16)
        for row, col, x in odd:
            w[row, col] = x if put else 0
        dv = gpu.upload(w)
        pkg.check(gpu.lib.lv_attention_fused(gpu.handle, d_out, dq, dk, dv, at, rope_table, scratch, HEADS, ROT, max_ctx, batch))
        gpu.sync()
        got.append(gpu.download(d_out, np.float32, batch * DIM).reshape(batch, DIM))
        gpu.free(dv)
    sees = np.zeros((batch, DIM), bool)
    for row, col, _ in odd:
        sees[row - pos:, col] = True
    assert not np.isfinite(got[1][sees]).any()
    assert np.array_equal(got[0][~sees].view(np.uint32), got[1][~sees].view(np.uint32))
    for d in (dk, dq, at, scratch, d_out):
        gpu.free(d)


@pytest.mark.parametrize("heads,batch,pos,max_ctx", [(4, 12, 100, 128), (4, 12, 400, 512), (2, 64, 60, 128), (5, 14, 480, 512), (4, 36, 20, 256)])
def test_attention_of_few_heads_keeps_the_exact_angles(gpu, pkg, rope_table, heads, batch, pos, max_ctx):
    """Steps whose rows fill no more than an SM each are turned by the table row of every distance: f32 sums are all that is left, 2^-22."""
    rng = np.random.default_rng(800 + batch)
    dim = heads * ROT
    k, v = ((rng.standard_normal((max_ctx, dim))).astype(np.float16) for _ in range(2))
    q = rng.standard_normal((batch, dim)).astype(np.float32)
    scratch, d_out = gpu.zeros(gpu.lib.lv_attention_scratch_bytes(heads, ROT, max_ctx, batch)), gpu.alloc(batch * dim * 4)
    args = [gpu.upload(a) for a in (q, k.view(np.uint16), v.view(np.uint16))]
    pkg.check(gpu.lib.lv_attention_fused(gpu.handle, d_out, *args, u32_dev(gpu, pos), rope_table, scratch, heads, ROT, max_ctx, batch))
    gpu.sync()
    got = gpu.download(d_out, np.float32, batch * dim).reshape(batch, dim)
    table = gpu.download(rope_table, np.float32, 2048 * ROT).reshape(2048, ROT // 2, 2)
    for z in (0, batch // 2, batch - 1):
        close(got[z], exact_attention(table, k.view(np.uint16), v.view(np.uint16), q[z], pos + z), rel_l2=4e-7, max_abs_frac=2e-6)
    for d in args + [scratch, d_out]:
        gpu.free(d)


@pytest.mark.parametrize("heads", [24, 40, 44, 52, 60])
@pytest.mark.parametrize("batch,pos,max_ctx", [(64, 960, 1024), (20, 700, 1024), (50, 1890, 2048), (64, 1984, 2048), (33, 1000, 2048)])
def test_prompt_attention_in_clusters_of_every_size(gpu, pkg, rope_table, heads, batch, pos, max_ctx):
    """Clusters are so small that all of them run at a time: 8, 6, 5, 4 and 4 CTAs for these heads on 148 SMs, with one to four passes of which the last is
    partial.  Bounds as in test_prompt_attention."""
    rng = np.random.default_rng(heads + pos)
    dim = heads * ROT
    k, v = (rng.standard_normal((max_ctx, dim), dtype=np.float32).astype(np.float16).view(np.uint16) for _ in range(2))
    q = rng.standard_normal((batch, dim)).astype(np.float32)
    scratch, d_out = gpu.zeros(gpu.lib.lv_attention_scratch_bytes(heads, ROT, max_ctx, batch)), gpu.zeros((batch + 1) * dim * 4)
    args = [gpu.upload(a) for a in (q, k, v)]
    pkg.check(gpu.lib.lv_attention_fused(gpu.handle, d_out, *args, u32_dev(gpu, pos), rope_table, scratch, heads, ROT, max_ctx, batch))
    gpu.sync()
    got = gpu.download(d_out, np.float32, (batch + 1) * dim).reshape(batch + 1, dim)
    table = gpu.download(rope_table, np.float32, 2048 * ROT).reshape(2048, ROT // 2, 2)
    for z in (0, 9, batch // 2 + 1, batch - 1):
        close(got[z], exact_attention(table, k, v, q[z], pos + z), rel_l2=1e-5, max_abs_frac=2e-5)
    assert not got[batch].any() and np.isfinite(got).all()
    for d in args + [scratch, d_out]:
        gpu.free(d)


@pytest.mark.parametrize("batch,pos,max_ctx", [(12, 30, 128), (64, 300, 512), (64, 1900, 2048)])
def test_attention_of_rows_that_are_not_aligned(gpu, pkg, rope_table, batch, pos, max_ctx):
    """Outputs 4 bytes behind a 16-byte boundary were always taken."""
    rng = np.random.default_rng(900 + batch)
    k, v = _caches(rng, pos + batch, max_ctx)
    q = rng.standard_normal((batch, DIM)).astype(np.float32)
    scratch, d_out = gpu.zeros(gpu.lib.lv_attention_scratch_bytes(HEADS, ROT, max_ctx, batch)), gpu.zeros((batch * DIM + 4) * 4)
    args = [gpu.upload(a) for a in (q, k, v)]
    pkg.check(gpu.lib.lv_attention_fused(gpu.handle, pkg.offset(d_out, 4), *args, u32_dev(gpu, pos), rope_table, scratch, HEADS, ROT, max_ctx, batch))
    gpu.sync()
    got = gpu.download(d_out, np.float32, batch * DIM + 4)
    assert got[0] == 0 and not got[-3:].any()
    backlog = 128
    while backlog < pos + batch:
        backlog *= 2
    for z in (0, batch - 1):
        close(got[1:-3].reshape(batch, DIM)[z], ob.attention(k, v, q[z], pos + z, backlog, HEADS, ROT), rel_l2=1e-5, max_abs_frac=2e-5)
    for d in args + [scratch, d_out]:
        gpu.free(d)


def test_prompt_attention_of_several_passes_repeats_itself(gpu, pkg, rope_table):
    """More than 1024 positions: a CTA brings new keys to where it kept probabilities.  The same bits from every launch, and the first
    rows of a step the same bits as in a shorter one."""
    rng = np.random.default_rng(35)
    batch, pos, max_ctx = 64, 1900, 2048
    k, v = _caches(rng, pos + batch, max_ctx)
    q = rng.standard_normal((batch, DIM)).astype(np.float32)
    dk, dv, dq, at = gpu.upload(k), gpu.upload(v), gpu.upload(q), u32_dev(gpu, pos)
    scratch, n = gpu.zeros(gpu.lib.lv_attention_scratch_bytes(HEADS, ROT, max_ctx, batch)), batch * DIM
    outs = [gpu.alloc(n * 4) for _ in range(20)]
    for d in outs:
        pkg.check(gpu.lib.lv_attention_fused(gpu.handle, d, dq, dk, dv, at, rope_table, scratch, HEADS, ROT, max_ctx, batch))
    part = gpu.alloc(n * 4)
    pkg.check(gpu.lib.lv_attention_fused(gpu.handle, part, dq, dk, dv, at, rope_table, scratch, HEADS, ROT, max_ctx, batch // 2))
    gpu.sync()
    first = gpu.download(outs[0], np.uint32, n)
    for d in outs[1:]:
        assert np.array_equal(first, gpu.download(d, np.uint32, n))
    assert np.array_equal(first[:n // 2], gpu.download(part, np.uint32, n // 2))
    for d in outs + [dk, dv, dq, at, scratch, part]:
        gpu.free(d)


def test_prompt_attention_leaves_out_rows_outside_the_cache(gpu, pkg, rope_table):
    rng = np.random.default_rng(34)
    batch, pos, max_ctx = 20, 245, 256                      # rows 0 .. 10 lie inside
    k, v = _caches(rng, max_ctx, max_ctx)
    q = rng.standard_normal((batch, DIM)).astype(np.float32)
    d_out, scratch = gpu.alloc(batch * DIM * 4), gpu.zeros(gpu.lib.lv_attention_scratch_bytes(HEADS, ROT, max_ctx, batch))
    pkg.check(gpu.lib.lv_memset(gpu.handle, d_out, 0xA5, batch * DIM * 4))
    pkg.check(gpu.lib.lv_attention_fused(gpu.handle, d_out, gpu.upload(q), gpu.upload(k), gpu.upload(v), u32_dev(gpu, pos), rope_table, scratch, HEADS, ROT, max_ctx, batch))
    with pytest.raises(pkg.LvError) as e:
        gpu.sync()
    assert e.value.code == pkg.LV_ERR_DEVICE_WAIT
    got = gpu.download(d_out, np.float32, batch * DIM).reshape(batch, DIM)
    close(got[10], ob.attention(k, v, q[10], pos + 10, max_ctx, HEADS, ROT), rel_l2=1e-5, max_abs_frac=2e-5)
    assert np.all(got[11:].view(np.uint8) == 0xA5)


def test_fused_attention_shares_one_scratch_between_batches_and_contexts(gpu, pkg, rope_table):
    """A session clears its scratch once and then launches short steps of several sizes, single tokens and growing backlogs on it, a group of
    sessions one row per member: what the launches with more than one chunk leave there must not reach the arrival counters of the others.
    (A negative batch: the members of a group.  Prompt steps of many rows take the matrix products, which use no scratch.)"""
    rng = np.random.default_rng(33)
    k, v = _caches(rng, 1100, 2048)
    dk, dv = gpu.upload(k), gpu.upload(v)
    shared = gpu.zeros(gpu.lib.lv_attention_scratch_bytes(HEADS, ROT, 2048, 64))
    for batch, pos, max_ctx in ((-64, 300, 512), (-37, 364, 512), (1, 401, 512), (-64, 512, 1024), (7, 576, 1024), (5, 584, 1024), (-12, 700, 1024), (64, 800, 1024), (1, 1024, 2048),
                                (-50, 1028, 2048), (2, 1030, 2048)):
        at, members = u32_dev(gpu, pos), None
        if batch < 0:
            batch = -batch
            members = gpu.upload(np.array([[dk.value, dv.value, at.value, 0]] * batch, np.uint64))
        dq = gpu.upload(rng.standard_normal((batch, DIM)).astype(np.float32))
        own = gpu.zeros(gpu.lib.lv_attention_scratch_bytes(HEADS, ROT, max_ctx, batch))
        got = []
        for scratch in (shared, own):
            d_out = gpu.alloc(batch * DIM * 4)
            pkg.check(gpu.lib.lv_memset(gpu.handle, d_out, 0xFF, batch * DIM * 4))
            if members is not None:
                pkg.check(gpu.lib.lv_attention_fused_group(gpu.handle, d_out, dq, members, rope_table, scratch, HEADS, ROT, max_ctx, batch))
            else:
                pkg.check(gpu.lib.lv_attention_fused(gpu.handle, d_out, dq, dk, dv, at, rope_table, scratch, HEADS, ROT, max_ctx, batch))
            gpu.sync()
            got.append(gpu.download(d_out, np.float32, batch * DIM))
            gpu.free(d_out)
        assert np.array_equal(got[0], got[1]), (batch, pos)
        gpu.free(dq)
        gpu.free(own)
    for d in (dk, dv, shared):
        gpu.free(d)


def test_qkv_fused_writes_cache_rows_and_query(gpu, pkg):
    rng = np.random.default_rng(32)
    ctx_rows, pos, batch = 8, 3, 2
    ws = [qn.quantize_q4_0((rng.standard_normal((DIM, DIM)) * 0.02).astype(np.float32)) for _ in range(3)]
    wq, wk, wv = ws
    x = (rng.standard_normal((batch, DIM)) * 2).astype(np.float32)
    nw = (1 + 0.01 * rng.standard_normal(DIM)).astype(np.float32)
    dkc, dvc = gpu.zeros(ctx_rows * DIM * 2), gpu.zeros(ctx_rows * DIM * 2)
    dq = gpu.alloc(batch * DIM * 4)
    pkg.check(gpu.lib.lv_norm_qkv_kvappend(gpu.handle, dq, dkc, dvc, gpu.upload(wq), gpu.upload(wk), gpu.upload(wv), qn.Q4_0,
                                           gpu.upload(x), gpu.upload(nw), u32_dev(gpu, pos), DIM, DIM, batch, ctx_rows))
    gpu.sync()
    gq = gpu.download(dq, np.float32, batch * DIM).reshape(batch, DIM)
    gk = gpu.download(dkc, np.uint16, ctx_rows * DIM).reshape(ctx_rows, DIM).view(np.float16).astype(np.float32)
    gv = gpu.download(dvc, np.uint16, ctx_rows * DIM).reshape(ctx_rows, DIM).view(np.float16).astype(np.float32)
    for z in range(batch):
        h = ob.norm(x[z], nw)
        close(gq[z], ob.gemv(wq, qn.Q4_0, h, DIM, DIM, 128))
        # f16 rounding of a value that differs in the last fp32 bits may land on the neighbouring half
        close(gk[pos + z], ob.gemv(wk, qn.Q4_0, h, DIM, DIM, 128), rel_l2=6e-4, max_abs_frac=1e-3)
        close(gv[pos + z], ob.gemv(wv, qn.Q4_0, h, DIM, DIM, 128), rel_l2=6e-4, max_abs_frac=1e-3)
    assert not gk[:pos].any() and not gk[pos + batch:].any()


def test_argmax_copy_add(gpu, pkg):
    rng = np.random.default_rng(33)
    lib, h = gpu.lib, gpu.handle
    d_idx = gpu.alloc(16)
    for case in range(4):
        v = rng.standard_normal(32000).astype(np.float32)
        if case == 1:
            v[[31999, 777, 12345]] = v.max() + 1        # ties: lowest index wins
        if case == 2:
            v[5] = np.nan
        if case == 3:
            v[0] = np.nan
        pkg.check(lib.lv_argmax_f32(h, d_idx, gpu.upload(v), v.size))
        gpu.sync()
        assert gpu.download(d_idx, np.uint32, 1)[0] == ob.load().orc_argmax(ob.ptr(v), v.size)
    a, b = rng.standard_normal(5000).astype(np.float32), rng.standard_normal(5000).astype(np.float32)
    da, db, dc = gpu.upload(a), gpu.upload(b), gpu.alloc(a.nbytes)
    pkg.check(lib.lv_copy_f32(h, dc, da, a.size))
    pkg.check(lib.lv_add_f32(h, da, db, a.size))
    gpu.sync()
    assert np.array_equal(gpu.download(dc, np.float32, a.size), a)
    assert np.array_equal(gpu.download(da, np.float32, a.size), a + b)


def test_argmax_odd_sizes_and_unaligned_start(gpu, pkg):
    rng = np.random.default_rng(35)
    lib, h = gpu.lib, gpu.handle
    d_idx = gpu.alloc(16)
    big = rng.standard_normal(40000).astype(np.float32)
    big[[3, 20001, 39999]] = 9.0                        # equal maxima at both ends of the vector paths
    d_big = gpu.upload(big)
    for first, n in ((0, 1), (0, 3), (1, 4097), (0, 32769), (2, 39998), (3, 37), (4, 36001)):
        pkg.check(lib.lv_argmax_f32(h, d_idx, C.c_void_p(d_big.value + 4 * first), n))
        gpu.sync()
        v = np.ascontiguousarray(big[first:first + n])
        assert gpu.download(d_idx, np.uint32, 1)[0] == ob.load().orc_argmax(ob.ptr(v), n), (first, n)


def test_argmax_advance_logs_the_token_and_moves_the_position(gpu, pkg):
    """One launch = lv_argmax_f32 + lv_decode_advance, plus the token in mapped host memory."""
    rng = np.random.default_rng(36)
    lib, h = gpu.lib, gpu.handle
    host = C.c_void_p()
    pkg.check(lib.lv_host_alloc(h, 64, C.byref(host)))
    word = (C.c_uint32 * 16).from_address(host.value)
    try:
        for case, batch in ((0, 1), (1, 3), (2, 1)):
            v = rng.standard_normal(32000).astype(np.float32)
            if case == 1:
                v[[31000, 42]] = v.max() + 2
            if case == 2:
                v[0] = np.nan
            want = ob.load().orc_argmax(ob.ptr(v), v.size)
            cfg, log, am = u32_dev(gpu, 7), gpu.upload(np.full(32, 0xFFFFFFFF, np.uint32)), gpu.zeros(4)
            word[5] = 0xDEADBEEF
            pkg.check(lib.lv_argmax_advance(h, gpu.upload(v), v.size, cfg, log, batch, 32, am, C.c_void_p(host.value + 20)))
            gpu.sync()
            assert word[5] == want
            assert gpu.download(am, np.uint32, 1)[0] == want
            got_log = gpu.download(log, np.uint32, 32)
            assert got_log[7 + batch] == want and (np.delete(got_log, 7 + batch) == 0xFFFFFFFF).all()
            assert (gpu.download(cfg, np.uint32, 4) == 7 + batch).all()
        # a log index outside the log is reported, not written
        cfg, log = u32_dev(gpu, 31), gpu.upload(np.full(32, 0xFFFFFFFF, np.uint32))
        pkg.check(lib.lv_argmax_advance(h, gpu.upload(np.ones(64, np.float32)), 64, cfg, log, 1, 32, None, None))
        assert lib.lv_stream_sync(h, 10000) == pkg.LV_ERR_DEVICE_WAIT
        assert (gpu.download(log, np.uint32, 32) == 0xFFFFFFFF).all()
    finally:
        pkg.check(lib.lv_host_free(h, host))


def test_graph_capture_replays_with_a_new_position(gpu, pkg, rope_table):
    """The recorded step reads the position from device memory, so one graph serves every token."""
    rng = np.random.default_rng(34)
    ctx_rows = 16
    x = rng.standard_normal((1, DIM)).astype(np.float32)
    cache = gpu.zeros(ctx_rows * DIM * 2)
    dpos, dx = u32_dev(gpu, 2), gpu.upload(x)
    g = C.c_void_p()
    pkg.check(gpu.lib.lv_graph_begin_capture(gpu.handle))
    pkg.check(gpu.lib.lv_kv_append_f16(gpu.handle, cache, dx, dpos, DIM, 1, ctx_rows))
    pkg.check(gpu.lib.lv_graph_end_capture(gpu.handle, C.byref(g)))
    for pos in (2, 9):
        p = np.array([pos] * 4, np.uint32)
        pkg.check(gpu.lib.lv_upload(gpu.handle, dpos, p.ctypes.data_as(C.c_void_p), 16))
        pkg.check(gpu.lib.lv_graph_launch(gpu.handle, g))
        gpu.sync()
    got = gpu.download(cache, np.uint16, ctx_rows * DIM).reshape(ctx_rows, DIM)
    want = x.astype(np.float16).view(np.uint16)[0]
    assert np.array_equal(got[2], want) and np.array_equal(got[9], want)
    assert not got[[0, 1, 3, 8, 10]].any()
    pkg.check(gpu.lib.lv_graph_destroy(g))


@pytest.mark.parametrize("two_phase", ["0", "1"], ids=["sum-per-cta", "sum-per-gpu"])
def test_exchange_fused_into_the_gemvs_on_one_rank(pkg, two_phase, monkeypatch):
    """lv_tp_arm_push / lv_tp_arm_pull with a single-rank window: the pushed rows of one GEMV come
    back as `x + rows` in the input of the next normalising GEMV, which also stores that sum.  Both
    ways of forming the sum (in every CTA; one slice per CTA, then shared through local flags)."""
    monkeypatch.setenv("LV_TP_TWO_PHASE", two_phase)
    rng = np.random.default_rng(60)
    K, rows_out, steps = 1024, 512, 3
    Wa = qn.quantize_q4_0((rng.standard_normal((K, 512)) * 0.05).astype(np.float32))      # K rows of 512 columns
    Wb = qn.quantize_q4_0((rng.standard_normal((rows_out, K)) * 0.05).astype(np.float32))
    nw = (1 + 0.1 * rng.standard_normal(K)).astype(np.float32)
    with pkg.Context(0) as g:
        lib, h = g.lib, g.handle
        handle = (C.c_uint8 * 64)()
        pkg.check(lib.lv_peer_window_create(h, 1, K, handle))
        pkg.check(lib.lv_peer_connect(h, 0, handle))
        cfg, dWa, dWb, dnw = u32_dev(g, 0), g.upload(Wa), g.upload(Wb), g.upload(nw)
        for step in range(steps):                       # a new step number (flag epoch) every round
            v = rng.standard_normal(512).astype(np.float32)
            x = rng.standard_normal(K).astype(np.float32)
            dx, dxo, dout, dummy = g.upload(x), g.zeros(K * 4), g.zeros(rows_out * 4), g.zeros(K * 4)
            for exchange in (0, 1):                     # both slot sets
                pkg.check(lib.lv_tp_arm_push(h, exchange, 2))
                pkg.check(lib.lv_gemv(h, dummy, dWa, qn.Q4_0, g.upload(v), K, 512, 1, 0))
                pkg.check(lib.lv_tp_arm_pull(h, exchange, 2, K, dxo))
                pkg.check(lib.lv_norm_gemv(h, dout, dWb, qn.Q4_0, dx, dnw, rows_out, K, 1))
                g.sync()
                partial = ob.gemv(Wa, qn.Q4_0, v, K, 512, 128)
                close(g.download(dxo, np.float32, K), x + partial, rel_l2=2e-6, max_abs_frac=2e-6)
                close(g.download(dout, np.float32, rows_out), ob.gemv(Wb, qn.Q4_0, ob.norm(x + partial, nw), rows_out, K, 128))
                assert not g.download(dummy, np.float32, K).any()          # a pushing GEMV does not write its `out`
            pkg.check(lib.lv_decode_advance(h, cfg, None, None, 1, 0))      # ends the step: the next epochs differ
        # an armed role without connected windows is refused, as is an exchange index outside the step
        assert lib.lv_tp_arm_push(h, 2, 2) == pkg.LV_ERR_BAD_ARGUMENTS
        pkg.check(lib.lv_peer_destroy(h))
        assert lib.lv_tp_arm_push(h, 0, 2) == pkg.LV_ERR_BAD_ARGUMENTS
