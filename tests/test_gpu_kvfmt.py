"""int8 (kvQ8) and f32 KV caches: the append of kv_store_q8 bit for bit, and attention over those caches against exact
attention over the values the cache holds (engine/wgsl/qwen35.js:97-139, :908-946; engine/wgsl/dense.js:22-136)."""
import numpy as np
import pytest

from oracle import po
from tests import util

pytestmark = pytest.mark.gpu


def _engine(fmt, nH, nKV, hd, max_seq, act="f32", max_cols=8, rope_mode="none", n_layers=1, n_seqs=1):
    import torch
    from pooled_b200 import AttnConfig, AttnEngine
    return AttnEngine(AttnConfig(n_heads=nH, n_kv_heads=nKV, head_dim=hd, n_rot=64, rope_theta=1e7, max_seq=max_seq, rope_mode=rope_mode, n_layers=n_layers,
                                 n_seqs=n_seqs, act_dtype=torch.float32 if act == "f32" else torch.float16, max_cols=max_cols, kv_format=fmt))


def _held(eng, fmt, li, rows):
    """The K and V values the cache holds, as float32 [rows][kv_dim]."""
    k, v = eng.cache(li, "k")[0, :rows].cpu().numpy(), eng.cache(li, "v")[0, :rows].cpu().numpy()
    if fmt == "q8":
        ks, vs = eng.cache_scales(li, "k")[0, :rows].cpu().numpy(), eng.cache_scales(li, "v")[0, :rows].cpu().numpy()
        return po.dequant_q8(k, ks), po.dequant_q8(v, vs), (k, ks, v, vs)
    return k, v, None


def test_q8_append_is_kv_store_q8_bit_for_bit():
    import torch
    nH, nKV, hd, n = 16, 2, 256, 40
    eng = _engine("q8", nH, nKV, hd, 64, max_cols=64)
    x = (po.normal(1, 2 * n * nKV * hd) * 2.5).astype(np.float32).reshape(2, n, nKV * hd)
    x[0, 3, :32] = 0.0                       # an all-zero block: scale 0, values 0
    x[0, 4, 32:64] = 1e-30                   # a block whose scale underflows towards zero
    x[1, 5, 7] = 1000.0                      # one outlier sets the block's scale
    x[0, 6, :32] = np.arange(32) - 15.5      # ties: x * inv lands on .5 values for some entries
    eng.kv_append(0, 0, 10, torch.from_numpy(x[0]).cuda(), torch.from_numpy(x[1]).cuda())
    eng.sync()
    _, _, (k, ks, v, vs) = _held(eng, "q8", 0, 64)
    wk, wks = po.kv_store_q8(x[0]); wv, wvs = po.kv_store_q8(x[1])
    assert np.array_equal(k[10:10 + n], wk) and np.array_equal(v[10:10 + n], wv), "int8 values differ from kv_store_q8"
    assert np.array_equal(ks[10:10 + n].view(np.uint32), wks.view(np.uint32)) and np.array_equal(vs[10:10 + n].view(np.uint32), wvs.view(np.uint32))
    nk, nks = po.np_kv_store_q8(x[0])        # the NumPy twin agrees with the C restatement
    assert np.array_equal(nk, wk) and np.array_equal(nks.view(np.uint32), wks.view(np.uint32))


@pytest.mark.parametrize("fmt", ["q8", "f32"])
@pytest.mark.parametrize("nH,nKV,hd", [(16, 2, 256), (16, 8, 128), (8, 2, 64)])
def test_decode_over_the_cache_equals_exact_attention_over_what_it_holds(fmt, nH, nKV, hd):
    import torch
    rows = 3001
    eng = _engine(fmt, nH, nKV, hd, 3100, max_cols=8)
    K = (po.normal(2, rows * nKV * hd) * 0.8).astype(np.float32).reshape(rows, nKV * hd); V = po.normal(3, rows * nKV * hd).astype(np.float32).reshape(rows, nKV * hd)
    for r0 in range(0, rows, 8):             # appended eight rows at a time
        eng.kv_append(0, 0, r0, torch.from_numpy(K[r0:r0 + 8]).cuda(), torch.from_numpy(V[r0:r0 + 8]).cuda())
    eng.sync()
    Kh, Vh, _ = _held(eng, fmt, 0, rows)
    if fmt == "f32":
        assert np.array_equal(Kh, K) and np.array_equal(Vh, V)
    for seq_len, nc in ((1, 1), (64, 1), (65, 1), (rows, 1), (rows, 5), (700, 3)):
        pos = seq_len - nc
        q = po.normal(10 + seq_len, nc * nH * hd).astype(np.float32).reshape(nc, nH * hd); g = po.normal(20 + seq_len, nc * nH * hd).astype(np.float32).reshape(nc, nH * hd)
        out = eng.decode(0, [(0, pos, nc)], util.torch_dev(q), util.torch_dev(g)).cpu().numpy()
        eng.sync()
        ref = po.attn_f64_kv32(q, Kh, Vh, nH, nKV, hd, pos, nc, g)
        assert np.all(np.isfinite(out)) and util.errs(out, ref)[1] < util.REF_REL, f"{fmt} seq_len {seq_len} x {nc}"


@pytest.mark.parametrize("fmt", ["q8", "f32"])
def test_layer_call_and_prefill_on_other_formats(fmt):
    # RoPE + append + attend + gate in one call: k is rotated (float64 expression, f32 result) and then stored in the
    # layer's format; a 300-column prefill chunk, then one token, then a 5-token block
    import torch
    nH, nKV, hd, n_rot, theta = 16, 2, 256, 64, 1e7
    eng = _engine(fmt, nH, nKV, hd, 512, act="f16", max_cols=320, rope_mode="f64")
    T = 306
    q = util.normal_f16(1, (T, nH * hd)); k = util.normal_f16(2, (T, nKV * hd)); v = util.normal_f16(3, (T, nKV * hd)); g = util.normal_f16(4, (T, nH * hd))
    d = lambda a: util.torch_dev(a, torch.float16)
    outs = [eng.encode_layer(0, 0, d(q[:300]), d(k[:300]), d(v[:300]), d(g[:300]), mode="prefill"),
            eng.encode_layer(0, 300, d(q[300:301]), d(k[300:301]), d(v[300:301]), d(g[300:301]), mode="decode"),
            eng.encode_layer(0, 301, d(q[301:]), d(k[301:]), d(v[301:]), d(g[301:]), mode="decode")]
    eng.sync()
    out = torch.cat(outs).float().cpu().numpy()
    k_rot = np.stack([po.rope_neox_f64(k[c], nKV, hd, n_rot, c, theta) for c in range(T)])
    Kh, Vh, held = _held(eng, fmt, 0, T)
    if fmt == "q8":
        wk, wks = po.kv_store_q8(k_rot); wv, wvs = po.kv_store_q8(v)
        assert np.array_equal(held[0], wk) and np.array_equal(held[2], wv) and np.array_equal(held[1].view(np.uint32), wks.view(np.uint32))
    else:
        assert np.array_equal(Kh.view(np.uint32), k_rot.view(np.uint32)) and np.array_equal(Vh, v)
    q_rot = np.stack([po.rope_neox_f64(q[c], nH, hd, n_rot, c, theta) for c in range(T)])
    ref = np.concatenate([po.attn_f64_kv32(q_rot[c:c + 1], Kh, Vh, nH, nKV, hd, c, 1, g[c:c + 1]) for c in range(T)])
    util.assert_close(out, ref, f"{fmt} layer calls")


@pytest.mark.parametrize("fmt,nH,nKV,hd", [("q8", 16, 1, 256), ("q8", 6, 2, 128), ("q8", 3, 1, 64), ("f32", 4, 4, 256), ("f32", 8, 4, 128), ("f32", 8, 2, 64), ("f32", 12, 4, 64)])
def test_row_groups_splits_and_magnitudes(fmt, nH, nKV, hd):
    # query rows of one, two and four 8-row groups and of several row tiles, contexts from one row to many splits, few
    # and many records per row; scales from 1e-9 to 1e4 and q from 1e-6 to 30, which f16 operands cannot hold unscaled
    import torch
    rows = 2900
    eng = _engine(fmt, nH, nKV, hd, rows + 4, max_cols=600)
    rng = np.random.default_rng(5)
    K = rng.standard_normal((rows, nKV * hd)).astype(np.float32); V = rng.standard_normal((rows, nKV * hd)).astype(np.float32)
    mag = np.repeat(10.0 ** rng.uniform(-9, 0, (rows, nKV * hd // 32)), 32, axis=1).astype(np.float32)      # a scale per block
    for k0 in range(0, rows, 580):
        eng.kv_append(0, 0, k0, torch.from_numpy(K[k0:k0 + 580] * np.sqrt(mag[k0:k0 + 580])).cuda(), torch.from_numpy(V[k0:k0 + 580] * mag[k0:k0 + 580] * 1e4).cuda())
    eng.sync()
    Kh, Vh, _ = _held(eng, fmt, 0, rows)
    for seq_len, nc in ((1, 1), (17, 1), (127, 2), (129, 3), (1500, 5), (rows, 1), (rows, 7), (500, 300), (2900, 70)):
        pos = seq_len - nc
        q = po.normal(10 + seq_len, nc * nH * hd).astype(np.float32).reshape(nc, nH, hd)
        q *= (10.0 ** rng.uniform(-6, 1, (nc, nH, 1))).astype(np.float32)
        if nc == 1:
            q[0, 0] *= np.float32(30.0 / np.abs(q[0, 0]).max())     # logits stay below 50: f32 scores err by 50 * 2^-24 at most
        q = q.reshape(nc, nH * hd)
        out = eng.decode(0, [(0, pos, nc)], util.torch_dev(q)).cpu().numpy() if nc <= 8 else eng.prefill(0, 0, pos, util.torch_dev(q)).cpu().numpy()
        eng.sync()
        ref = po.attn_f64_kv32(q, Kh, Vh, nH, nKV, hd, pos, nc, None)
        assert np.all(np.isfinite(out)) and util.errs(out, ref)[1] < util.REF_REL, f"{fmt} seq_len {seq_len} x {nc}: {util.errs(out, ref)}"
        e = _block_errs(out, ref, nH, hd)            # the blocks differ by up to nine decades: each by itself
        assert e.max() < util.REF_REL, f"{fmt} seq_len {seq_len} x {nc}: {e.max(axis=(0, 1))}"


@pytest.mark.parametrize("fmt,nH,nKV,hd", [("q8", 16, 2, 256), ("q8", 6, 2, 128), ("q8", 3, 1, 64), ("f32", 4, 2, 128), ("f32", 6, 1, 256)])
@pytest.mark.parametrize("pos,n_cols", [(0, 70), (37, 21), (1000, 5), (59, 8)])
@pytest.mark.parametrize("bad", [np.inf, np.nan, 1e30])
def test_rows_a_column_does_not_see_leave_no_trace(fmt, nH, nKV, hd, pos, n_cols, bad):
    # columns of one call, the last few of whose K or V rows hold an infinity, a NaN or values that dwarf all others: the bits
    # of the columns before them are those of the same call over ordinary rows
    import torch
    eng = _engine(fmt, nH, nKV, hd, 1100, max_cols=1024)
    T, cut = pos + n_cols, n_cols // 2
    K, V = (torch.from_numpy(po.normal(40 + i, T * nKV * hd).astype(np.float32).reshape(T, -1)).cuda() for i in range(2))
    q = util.torch_dev(po.normal(50, n_cols * nH * hd).astype(np.float32).reshape(n_cols, -1))
    run = lambda: eng.decode(0, [(0, pos, n_cols)], q) if n_cols <= 8 else eng.prefill(0, 0, pos, q)
    eng.kv_append(0, 0, 0, K, V)
    clean = run()
    Kb, Vb = K[pos + cut:].clone(), V[pos + cut:].clone()
    Kb[1::2, 3::40] = bad
    Vb[:, ::33] = bad
    eng.kv_append(0, 0, pos + cut, Kb, Vb)
    dirty = run()
    eng.sync()
    assert torch.isfinite(clean).all() and not torch.equal(clean[cut:], dirty[cut:])
    assert torch.equal(clean[:cut].view(torch.int32), dirty[:cut].view(torch.int32))


def _block_errs(got, ref, nH, hd):
    """Largest error of each 32-dim block of each head, relative to the block's own largest output."""
    d, r = (np.abs(x.astype(np.float64)).reshape(-1, nH, hd // 32, 32).max(axis=3) for x in (got - ref, ref))
    return d / r


@pytest.mark.parametrize("fmt", ["q8", "f32"])
@pytest.mark.parametrize("nH,nKV,hd,rows,n_cols", [(16, 2, 256, 3000, 1), (16, 8, 128, 700, 5), (4, 2, 64, 2000, 33), (8, 2, 128, 64, 20)])
@pytest.mark.parametrize("log2_v", [-30, -16, 24])
def test_value_blocks_of_any_magnitude_keep_f32_precision(fmt, nH, nKV, hd, rows, n_cols, log2_v):
    # the V of every other 32-dim block 2^-30 or 2^-16 of its neighbours', or one row's V 2^24 times all others where the row has next
    # to no weight.  Judged per block of the output, relative to its own largest value: scores below 8 in 32 bits leave 8 * 2^-24
    # in a weight, and the sums as much again (their terms add up without their signs to some 8 times the largest output): 1e-6,
    # doubled for the largest of several thousand blocks
    import torch
    eng = _engine(fmt, nH, nKV, hd, rows, max_cols=rows)
    g = np.random.default_rng(9)
    K, V, q = (g.standard_normal(s).astype(np.float32) for s in ((rows, nKV * hd), (rows, nKV * hd), (n_cols, nH * hd)))
    if log2_v < 0:
        V.reshape(rows, -1, 2, 32)[:, :, 1] *= np.float32(2.0 ** log2_v)
    else:
        V[7] *= np.float32(2.0 ** log2_v)
        K[7] = -np.abs(K[7]) * 4
        q = np.abs(q)                                             # row 7 scores about -2.5 sqrt(hd)
    eng.kv_append(0, 0, 0, util.torch_dev(K), util.torch_dev(V))
    dq, pos = util.torch_dev(q), rows - n_cols
    out = (eng.decode(0, [(0, pos, n_cols)], dq) if n_cols <= 8 else eng.prefill(0, 0, pos, dq)).cpu().numpy()
    eng.sync()
    Kh, Vh, _ = _held(eng, fmt, 0, rows)
    e = _block_errs(out, po.attn_f64_kv32(q, Kh, Vh, nH, nKV, hd, pos, n_cols, None), nH, hd)
    assert e.max() < 2e-6, f"{e.max(axis=(0, 1))}"


@pytest.mark.parametrize("fmt", ["q8", "f32"])
@pytest.mark.parametrize("nH,nKV,hd,rows,n_cols", [(16, 2, 256, 3000, 1), (16, 8, 128, 700, 5), (4, 2, 64, 2000, 33)])
@pytest.mark.parametrize("log2_q", [-16, -30])
def test_query_blocks_of_any_magnitude_keep_f32_precision(fmt, nH, nKV, hd, rows, n_cols, log2_q):
    # q of every other 32-dim block small, K there as much larger, so that all blocks weigh alike in the scores (bound as above)
    eng = _engine(fmt, nH, nKV, hd, rows, max_cols=rows)
    g = np.random.default_rng(10)
    K, V, q = (g.standard_normal(s).astype(np.float32) for s in ((rows, nKV * hd), (rows, nKV * hd), (n_cols, nH * hd)))
    K.reshape(rows, -1, 2, 32)[:, :, 1] *= np.float32(2.0 ** -log2_q)
    q.reshape(n_cols, -1, 2, 32)[:, :, 1] *= np.float32(2.0 ** log2_q)
    eng.kv_append(0, 0, 0, util.torch_dev(K), util.torch_dev(V))
    dq, pos = util.torch_dev(q), rows - n_cols
    out = (eng.decode(0, [(0, pos, n_cols)], dq) if n_cols <= 8 else eng.prefill(0, 0, pos, dq)).cpu().numpy()
    eng.sync()
    Kh, Vh, _ = _held(eng, fmt, 0, rows)
    e = _block_errs(out, po.attn_f64_kv32(q, Kh, Vh, nH, nKV, hd, pos, n_cols, None), nH, hd)
    assert e.max() < 2e-6, f"{e.max(axis=(0, 1))}"


@pytest.mark.parametrize("fmt,nH,nKV,hd", [("q8", 16, 2, 256), ("q8", 6, 2, 128), ("q8", 3, 1, 64), ("f32", 4, 2, 256), ("f32", 4, 1, 128), ("f32", 2, 2, 64), ("f32", 6, 2, 128)])
@pytest.mark.parametrize("rows,n_cols", [(1, 1), (70, 1), (70, 20), (2900, 1), (2900, 5)])
@pytest.mark.parametrize("top", [1e31, 3.2e38])
def test_scores_down_to_the_lowest_f32_still_weigh(fmt, nH, nKV, hd, rows, n_cols, top):
    # q . k between -top / 2 and -top: every row's weight goes to its least negative score (what the V of that row holds comes out)
    eng = _engine(fmt, nH, nKV, hd, rows, max_cols=rows)
    g = np.random.default_rng(12)
    b = np.float32(np.sqrt(top / hd))
    K = np.repeat(-b * g.uniform(0.5, 1.0, (rows, 1)).astype(np.float32), nKV * hd, axis=1)
    V, q = g.standard_normal((rows, nKV * hd)).astype(np.float32), np.full((n_cols, nH * hd), b, np.float32)
    eng.kv_append(0, 0, 0, util.torch_dev(K), util.torch_dev(V))
    dq, pos = util.torch_dev(q), rows - n_cols
    out = (eng.decode(0, [(0, pos, n_cols)], dq) if n_cols <= 8 else eng.prefill(0, 0, pos, dq)).cpu().numpy()
    eng.sync()
    Kh, Vh, _ = _held(eng, fmt, 0, rows)
    ref = po.attn_f64_kv32(q, Kh, Vh, nH, nKV, hd, pos, n_cols, None)
    assert np.all(np.isfinite(out)) and util.errs(out, ref)[1] < util.REF_REL


@pytest.mark.parametrize("hd,bound", [(64, 2.6e-7), (128, 2.6e-7), (256, 3.9e-7)])
def test_long_sums_over_int8_rows_stay_as_close_as_f32_loops(hd, bound):
    # 40 columns x 2 heads over 5000 rows in one split: 312 steps of a warp, one after the other.  2-norm error against float64
    # over the exact products value * scale.  An f32 addition is off by 0.72 * 2^-23 / sqrt(12) = 2.5e-8 of the sum at random, N
    # of them on a sum that grows like a random walk by sqrt(N / 2) times that, on one that grows steadily (the weights')
    # by sqrt(N / 3); scores and weights themselves leave 1.5e-7.  One output sum of 312 (head_dim 256): 3.5e-7; in two levels
    # of 16 and 20: 1.9e-7; weights in one of 1248 per thread: another 2.5e-7, 4.3e-7 in all
    import torch
    from pooled_b200 import AttnConfig, AttnEngine
    nH, nKV, rows, n_cols = 2, 1, 5000, 40
    eng = AttnEngine(AttnConfig(n_heads=nH, n_kv_heads=nKV, head_dim=hd, n_rot=64, rope_theta=1e7, max_seq=rows, rope_mode="none", act_dtype=torch.float32, max_cols=rows, splits=1,
                                kv_format="q8"))
    g = np.random.default_rng(14)
    K, V, q = (g.standard_normal(s).astype(np.float32) for s in ((rows, hd), (rows, hd), (n_cols, nH * hd)))
    eng.kv_append(0, 0, 0, util.torch_dev(K), util.torch_dev(V))
    out = eng.prefill(0, 0, rows - n_cols, util.torch_dev(q)).cpu().numpy().astype(np.float64).reshape(n_cols, nH, hd)
    eng.sync()
    k, ks, v, vs = _held(eng, "q8", 0, rows)[2]
    K, V = ((x.reshape(rows, -1, 32) * sc.astype(np.float64)[..., None]).reshape(rows, hd) for x, sc in ((k, ks), (v, vs)))
    s = np.einsum("chd,rd->chr", q.reshape(n_cols, nH, hd).astype(np.float64), K) / np.sqrt(hd)
    s = np.where(np.arange(rows) <= (rows - n_cols + np.arange(n_cols))[:, None, None], s, -np.inf)
    w = np.exp(s - s.max(axis=2, keepdims=True))
    ref = np.einsum("chr,rd->chd", w / w.sum(axis=2, keepdims=True), V)
    err = float(np.linalg.norm(out - ref) / np.linalg.norm(ref))
    assert err < bound, f"{err:.3e}"


@pytest.mark.parametrize("fmt,hd,n_rot,act,n_cols", [("q8", 256, 64, "f16", 1), ("q8", 128, 128, "f32", 3), ("q8", 128, 64, "f32", 70), ("f32", 64, 64, "f16", 2), ("f32", 256, 32, "f32", 5)])
def test_front_of_a_layer_call_with_head_norm_keeps_the_bits(fmt, hd, n_rot, act, n_cols):
    # head-norm, rotation and the format's append (in one launch where n_rot is 64, or 128 of 128): cache bytes as the CPU twins give them
    import torch
    from pooled_b200 import AttnConfig, AttnEngine
    nH, nKV, theta, pos, eps = 4, 2, 1e6, 37, 1e-6
    td = torch.float16 if act == "f16" else torch.float32
    eng = AttnEngine(AttnConfig(n_heads=nH, n_kv_heads=nKV, head_dim=hd, n_rot=n_rot, rope_theta=theta, max_seq=256, act_dtype=td, max_cols=128, kv_format=fmt))
    rng = np.random.default_rng(3)
    mk = (lambda *s: util.normal_f16(int(rng.integers(1 << 20)), s)) if act == "f16" else (lambda *s: rng.standard_normal(s).astype(np.float32))
    k0, v0 = mk(pos, nKV * hd), mk(pos, nKV * hd)
    eng.kv_append(0, 0, 0, util.torch_dev(k0), util.torch_dev(v0))
    q, k, v = mk(n_cols, 2 * nH * hd), mk(n_cols, nKV * hd), mk(n_cols, nKV * hd)       # q and gate interleaved
    qw, kw = (1 + 0.1 * rng.standard_normal(hd)).astype(np.float32), (1 + 0.1 * rng.standard_normal(hd)).astype(np.float32)
    eng.set_head_norm(0, util.torch_dev(qw), util.torch_dev(kw), eps)
    dq = util.torch_dev(q, td)
    out = eng.encode_layer(0, pos, dq, util.torch_dev(k, td), util.torch_dev(v, td), dq[:, hd:], q_head_stride=2 * hd, gate_head_stride=2 * hd).float().cpu().numpy()
    eng.sync()
    act_of = (lambda x: po.h2f(po.f16_rne(x))) if act == "f16" else (lambda x: x)
    qh = np.ascontiguousarray(q.reshape(n_cols, nH, 2, hd)[:, :, 0]).reshape(n_cols, -1); g = np.ascontiguousarray(q.reshape(n_cols, nH, 2, hd)[:, :, 1]).reshape(n_cols, -1)
    rot = lambda x, n, w: np.stack([po.rope_neox_f64(act_of(po.head_norm_f64(x[c], n, hd, w, eps)), n, hd, n_rot, pos + c, theta) for c in range(n_cols)])
    kr, qr = rot(k, nKV, kw), rot(qh, nH, qw)
    Kh, Vh, held = _held(eng, fmt, 0, pos + n_cols)
    if fmt == "q8":
        wk, wks = po.kv_store_q8(kr); wv, wvs = po.kv_store_q8(v)
        assert np.array_equal(held[0][pos:], wk) and np.array_equal(held[2][pos:], wv)
        assert np.array_equal(held[1][pos:].view(np.uint32), wks.view(np.uint32)) and np.array_equal(held[3][pos:].view(np.uint32), wvs.view(np.uint32))
    else:
        assert np.array_equal(Kh[pos:].view(np.uint32), kr.view(np.uint32)) and np.array_equal(Vh[pos:], v)
    util.assert_close(out, po.attn_f64_kv32(qr, Kh, Vh, nH, nKV, hd, pos, n_cols, g), f"{fmt} layer call")


def test_q8_state_round_trip_and_refusals():
    import torch
    from pooled_b200.lib import PaError
    nH, nKV, hd, pos = 16, 2, 256, 200
    a = _engine("q8", nH, nKV, hd, 256, max_cols=8)
    K = po.normal(5, pos * nKV * hd).astype(np.float32).reshape(pos, nKV * hd)
    for r0 in range(0, pos, 8):
        a.kv_append(0, 0, r0, torch.from_numpy(K[r0:r0 + 8]).cuda(), torch.from_numpy(K[r0:r0 + 8] * 0.5).cuda())
    st = a.export_state(pos)
    assert [len(p) for p in st["parts"]] == [pos * 512, pos * 512, pos * 16 * 4, pos * 16 * 4]      # K, V, K scales, V scales (kvQ8 _stateParts)
    b = _engine("q8", nH, nKV, hd, 256, max_cols=8)
    b.import_state(st)
    q = util.torch_dev(po.normal(6, nH * hd).astype(np.float32).reshape(1, -1))
    oa, ob = a.decode(0, [(0, pos - 1, 1)], q), b.decode(0, [(0, pos - 1, 1)], q)
    a.sync(); b.sync()
    assert torch.equal(oa.view(torch.int32), ob.view(torch.int32))
    with pytest.raises(PaError, match="different model"):
        _engine("f32", nH, nKV, hd, 256).import_state(st)
    with pytest.raises(PaError) as e:
        a.save_slot("x", pos)
    assert e.value.code == -2
    with pytest.raises(PaError) as e:
        a.decode_partial(0, [(0, pos - 1, 1)], q)
    assert e.value.code == -2


def test_an_int8_call_wider_than_the_grid():
    # 16 heads per kv head: 131 070 columns fill the grid's 65 535 row tiles; 131 200 into an empty cache, a column of the first
    # and the last rows and those around the seam against the oracle (one block of 64 columns of values, repeated)
    import torch
    nH, nKV, hd, T = 16, 1, 64, 131200
    eng = _engine("q8", nH, nKV, hd, T, act="f16", max_cols=T)
    K, V, q = (util.normal_f16(60 + i, (64, d)) for i, d in enumerate((hd, hd, nH * hd)))
    wide = lambda a: util.torch_dev(a, torch.float16).repeat(T // 64, 1)
    eng.kv_append(0, 0, 0, wide(K), wide(V))
    out = eng.prefill(0, 0, 0, wide(q))
    eng.sync()
    Kh, Vh, _ = _held(eng, "q8", 0, 64)
    for c in (0, 1, 63, 5000, 131069, 131070, 131071, T - 1):
        reps = c // 64
        # every whole block weighs as one: a column sees `reps` copies of the 64 rows and the first c % 64 + 1 of another
        s = q[c % 64].reshape(nH, hd).astype(np.float64) @ Kh.T.astype(np.float64) / np.sqrt(hd)
        w = np.exp(s - s.max(axis=1, keepdims=True)) * (reps + (np.arange(64) <= c % 64))
        ref = (w / w.sum(axis=1, keepdims=True)) @ Vh.astype(np.float64)
        util.assert_close(out[c].float().cpu().numpy(), ref.reshape(-1), f"column {c}")


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("n_cols", [9, 16, 17, 288, 289, 300])
def test_int8_row_tiles_of_32_and_64(hd, n_cols):
    # two heads per kv head: just past 16 query rows, one whole tile of 32 and a remainder, and either side of where 64-row tiles fill the chip
    nH, nKV, pos = 32, 16, 77
    rows = pos + n_cols
    eng = _engine("q8", nH, nKV, hd, rows, max_cols=rows)
    g = np.random.default_rng(19)
    K, V, q = (g.standard_normal(s).astype(np.float32) for s in ((rows, nKV * hd), (rows, nKV * hd), (n_cols, nH * hd)))
    eng.kv_append(0, 0, 0, util.torch_dev(K), util.torch_dev(V))
    out = eng.prefill(0, 0, pos, util.torch_dev(q)).cpu().numpy()
    eng.sync()
    Kh, Vh, _ = _held(eng, "q8", 0, rows)
    assert util.errs(out, po.attn_f64_kv32(q, Kh, Vh, nH, nKV, hd, pos, n_cols, None))[1] < util.REF_REL


@pytest.mark.parametrize("nH,nKV,hd", [(16, 2, 256), (6, 2, 128), (3, 1, 64)])
@pytest.mark.parametrize("rows,n_cols", [(64, 1), (129, 2), (1100, 3), (2900, 40), (9003, 3), (8963, 8)])
def test_f32_plans_of_many_waves(nH, nKV, hd, rows, n_cols):
    # head counts of the chunked f32 kernel at odd numbers of 64-row tiles, few and many columns: both split plans
    eng = _engine("f32", nH, nKV, hd, rows, max_cols=rows)
    g = np.random.default_rng(16)
    K, V, q = (g.standard_normal(s).astype(np.float32) for s in ((rows, nKV * hd), (rows, nKV * hd), (n_cols, nH * hd)))
    eng.kv_append(0, 0, 0, util.torch_dev(K), util.torch_dev(V))
    dq, pos = util.torch_dev(q), rows - n_cols
    out = (eng.decode(0, [(0, pos, n_cols)], dq) if n_cols <= 8 else eng.prefill(0, 0, pos, dq)).cpu().numpy()
    eng.sync()
    assert util.errs(out, po.attn_f64_kv32(q, K, V, nH, nKV, hd, pos, n_cols, None))[1] < util.REF_REL


@pytest.mark.parametrize("nH,nKV,hd,n_rot", [(4, 1, 256, 64), (4, 2, 256, 64), (2, 2, 256, 64), (8, 2, 128, 128), (16, 8, 128, 64), (4, 4, 128, 128), (4, 1, 64, 64), (4, 2, 64, 64), (2, 2, 64, 64)])
@pytest.mark.parametrize("act", ["f32", "f16"])
def test_f32_tokens_with_front_and_merge_in_the_kernel(nH, nKV, hd, n_rot, act, monkeypatch):
    # against the three-kernel chain bit for bit, cache rows too: tokens straight behind an append and one another, two layers, contexts
    # from none to several batches of rows per warp and either side of their edges
    import torch
    from pooled_b200 import AttnConfig, AttnEngine
    td, T, n = (torch.float32 if act == "f32" else torch.float16), 2200, 3
    outs = []
    rnd = lambda seed, *shape: torch.from_numpy(po.normal(seed, int(np.prod(shape))).astype(np.float32).reshape(shape)).cuda().to(td)
    K, V, q, k, v, g = (rnd(70 + i, T if i < 2 else 2 * n, (nH if i in (2, 5) else nKV) * hd) for i in range(6))
    for chain in (False, True):
        for var in ("POOLED_ATTN_NO_FUSE", "POOLED_ATTN_NO_MERGE"):
            monkeypatch.setenv(var, "1") if chain else monkeypatch.delenv(var, raising=False)
        eng = AttnEngine(AttnConfig(n_heads=nH, n_kv_heads=nKV, head_dim=hd, n_rot=n_rot, rope_theta=1e6, max_seq=T + n, n_layers=2, act_dtype=td, max_cols=T, kv_format="f32"))
        o = []
        for ctx in (0, 1, 15, 16, 127, 128, 129, 1000, 2047, T):
            for li in range(2):
                if ctx:
                    eng.kv_append(li, 0, 0, K[:ctx], V[:ctx])
                before = eng.stats()["kernel_launches"]
                for t in range(n):
                    o.append(eng.encode_layer(li, ctx + t, q[li * n + t:li * n + t + 1], k[li * n + t:li * n + t + 1], v[li * n + t:li * n + t + 1], g[li * n + t:li * n + t + 1]))
                assert chain or eng.stats()["kernel_launches"] - before == n
            o += [eng.cache(li, w)[0, :ctx + n].clone() for li in range(2) for w in "kv"]
        eng.sync()
        outs.append(o)
    for a, b in zip(*outs):
        assert torch.isfinite(a).all() and torch.equal(a, b)


@pytest.mark.parametrize("nH,nKV,hd", [(4, 1, 256), (8, 4, 256), (8, 2, 128), (16, 8, 128), (16, 16, 128), (2, 1, 64), (8, 2, 64)])
def test_f32_splits_around_the_end_of_eight(nH, nKV, hd):
    # contexts below, at and past one, two and three batches of rows per warp of eight splits, one token and three
    batch = 512 // hd * (2 if nH // nKV == 4 else 4) * 64
    rows = 3 * batch + 65
    eng = _engine("f32", nH, nKV, hd, rows, max_cols=rows)
    g = np.random.default_rng(18)
    K, V, q = (g.standard_normal(s).astype(np.float32) for s in ((rows, nKV * hd), (rows, nKV * hd), (3, nH * hd)))
    eng.kv_append(0, 0, 0, util.torch_dev(K), util.torch_dev(V))
    dq = util.torch_dev(q)
    for n in sorted({3, *(f * batch // 4 + d for f in (4, 7, 8, 12) for d in (-1, 0, 1, 64))}):
        for nc in (1, 3):
            out = eng.decode(0, [(0, n - nc, nc)], dq[:nc]).cpu().numpy()
            eng.sync()
            assert util.errs(out, po.attn_f64_kv32(q[:nc], K, V, nH, nKV, hd, n - nc, nc, None))[1] < util.REF_REL, f"{n} rows x {nc}"


@pytest.mark.parametrize("nH,nKV,n_cols,ctx", [(13, 13, 1, (128, 129, 1000)), (16, 16, 1, (129, 131, 700)), (8, 8, 2, (129, 300)), (5, 5, 3, (129, 300)), (2, 2, 1, (3585, 4000)),
                                               (1, 1, 1, (3585, 5003)), (8, 8, 1, (3585,)), (12, 12, 1, (4736, 4737)), (24, 12, 1, (4737,)), (13, 13, 1, (2500,))])
def test_f32_records_of_one_head_of_64_dims(nH, nKV, n_cols, ctx, monkeypatch):
    # the CTAs of one query head x 64 dims leave 66 floats each: merged in the kernel as by the kernel behind it, bit for bit, where more
    # than eight CTAs a (kv head, column) merge there
    hd, outs = 64, []
    rows = max(ctx)
    rnd = lambda seed, *shape: util.torch_dev(po.normal(seed, int(np.prod(shape))).astype(np.float32).reshape(shape))
    K, V, q, g = rnd(90, rows, nKV * hd), rnd(91, rows, nKV * hd), rnd(92, n_cols, nH * hd), rnd(93, n_cols, nH * hd)
    for chain in (False, True):
        monkeypatch.setenv("POOLED_ATTN_NO_MERGE", "1") if chain else monkeypatch.delenv("POOLED_ATTN_NO_MERGE", raising=False)
        eng = _engine("f32", nH, nKV, hd, rows, max_cols=rows)
        eng.kv_append(0, 0, 0, K, V)
        o = [eng.decode(0, [(0, n - n_cols, n_cols)], q, gate) for n in ctx for gate in (None, g) for _ in range(2)]
        eng.sync()
        outs.append([x.cpu().numpy() for x in o])
    assert all(np.isfinite(a).all() and np.array_equal(a, b) for a, b in zip(*outs))
    assert util.errs(outs[0][-3], po.attn_f64_kv32(q.cpu().numpy(), K.cpu().numpy(), V.cpu().numpy(), nH, nKV, hd, ctx[-1] - n_cols, n_cols, None))[1] < util.REF_REL


@pytest.mark.parametrize("fmt", ["f16", "f32"])
def test_merged_records_of_many_calls_keep_their_bits(fmt):
    # calls of different plans, one straight behind the other, through the one buffer of records that say themselves when they are there
    import torch
    nH, nKV, hd, ctx = 4, 2, 128, (9000, 3001, 12000, 7777)
    eng = _engine(fmt, nH, nKV, hd, max(ctx))
    g = torch.Generator(device="cuda").manual_seed(9)
    for w in "kv":
        c = eng.cache(0, w)
        x = torch.randn(c.shape, device="cuda", generator=g)
        c.copy_(x.half().view(torch.int16) if fmt == "f16" else x)
    q = torch.randn((1, nH * hd), device="cuda", generator=g)
    outs = [eng.decode(0, [(0, n - 1, 1)], q) for _ in range(60) for n in ctx]
    eng.sync()
    assert torch.isfinite(torch.stack(outs)).all() and all(torch.equal(o, outs[i % len(ctx)]) for i, o in enumerate(outs))


@pytest.mark.parametrize("nH,nKV,hd,pos,n_cols", [(24, 4, 256, 1000, 24), (24, 4, 256, 1000, 8), (24, 4, 256, 4096, 48), (16, 2, 256, 300, 48), (16, 2, 256, 300, 150), (16, 2, 256, 9000, 17),
                                                 (16, 8, 128, 2048, 48), (16, 8, 128, 1000, 64), (16, 8, 128, 4096, 200), (16, 8, 64, 300, 150), (16, 8, 64, 300, 200), (24, 4, 256, 0, 400)])
def test_int8_blocks_in_either_form(nH, nKV, hd, pos, n_cols):
    # more than 16 query rows: by four warps that convert for themselves and by eight that share a conversion, split in clusters, by records and not at all
    rows = pos + n_cols
    eng = _engine("q8", nH, nKV, hd, rows, max_cols=rows)
    g = np.random.default_rng(23)
    K, V, q = (g.standard_normal(s).astype(np.float32) for s in ((rows, nKV * hd), (rows, nKV * hd), (n_cols, nH * hd)))
    eng.kv_append(0, 0, 0, util.torch_dev(K), util.torch_dev(V))
    dq = util.torch_dev(q)
    outs = [eng.prefill(0, 0, pos, dq).cpu().numpy() for _ in range(2)]
    eng.sync()
    Kh, Vh, _ = _held(eng, "q8", 0, rows)
    assert np.array_equal(*outs)
    assert util.errs(outs[0], po.attn_f64_kv32(q, Kh, Vh, nH, nKV, hd, pos, n_cols, None))[1] < util.REF_REL
