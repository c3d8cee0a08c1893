"""Tiled causal prefill (tcgen05 + TMEM) on the GPU against the float64 oracle, through the C ABI."""
import numpy as np
import pytest

from oracle import po
from tests import util

pytestmark = pytest.mark.gpu


def _engine(nH, nKV, hd, max_seq, act="f32", max_cols=1024, n_rot=64, theta=1e7, rope_mode="none", n_seqs=1):
    import torch
    from pooled_b200 import AttnConfig, AttnEngine
    return AttnEngine(AttnConfig(n_heads=nH, n_kv_heads=nKV, head_dim=hd, n_rot=n_rot, rope_theta=theta, max_seq=max_seq, n_seqs=n_seqs,
                                 rope_mode=rope_mode, act_dtype=torch.float32 if act == "f32" else torch.float16, max_cols=max_cols))


# ---- the reference's own tile test, retargeted: tests/unit/attn_tile_test.js:118-131 --------------------------------
# (all six cases, in the reference's order: the LCG seed carries over from case to case)
TILE_CASES = [
    dict(name="MoE shape, first pass", hd=256, nH=16, nKV=2, nc=16, basePos=0, maxSeq=512),
    dict(name="MoE shape, 5 splits, partial tile", hd=256, nH=16, nKV=2, nc=16, basePos=301, maxSeq=4096),
    dict(name="27B shape, 2 big splits", hd=256, nH=24, nKV=4, nc=16, basePos=173, maxSeq=512),
    dict(name="27B shape, TK 16", hd=256, nH=24, nKV=4, nc=16, basePos=90, maxSeq=4096),
    dict(name="small head, 1 split target", hd=64, nH=8, nKV=2, nc=16, basePos=219, maxSeq=2048),
    dict(name="8-column batch", hd=128, nH=12, nKV=2, nc=8, basePos=77, maxSeq=1024),
]


def test_attn_tile_js_cases():
    import torch
    seed = 12345
    for t in TILE_CASES:
        hd, nH, nKV, nc, base, max_seq = t["hd"], t["nH"], t["nKV"], t["nc"], t["basePos"], t["maxSeq"]
        s0, s1 = nH * hd + 12, nH * hd + 20                       # padded column strides (attn_tile_test.js:51)
        K, V, q, seed = po.gen_attn_tile(seed, max_seq, nKV * hd, base + nc, nc, s0)
        eng = _engine(nH, nKV, hd, max_seq, act="f32", max_cols=64)
        util.load_cache(eng, 0, 0, K, V)                          # rows at or past base + nc hold the NaN pattern 0x7e00
        out = torch.full((nc, s1), float("nan"), device="cuda")
        eng.prefill(0, 0, base, util.torch_dev(q), out=out)
        eng.sync()
        o = out.cpu().numpy()
        ref = po.attn_f64(q, K, V, nH, nKV, hd, base, nc)
        assert np.all(np.isfinite(o[:, :nH * hd])), t["name"]
        ma, mr = util.assert_close(o[:, :nH * hd], ref, t["name"])
        assert np.all(np.isnan(o[:, nH * hd:])), "wrote into the padding between columns"   # attn_tile_test.js:80
        print(f"{t['name']}: max-abs {ma:.2e} max-rel {mr:.2e}")


def test_head_dims_outside_64_128_256_are_refused():
    # attnTileConfig takes any multiple of 16 up to 256 (engine/wgsl/attn_tile.js:44); the TMA boxes and the tensor-core
    # tiles here are built from 64-element chunks, so 64, 128 and 256 (every shape pooled's models use) are what exists
    from pooled_b200 import PaError
    for hd in (96, 80, 512):
        with pytest.raises(PaError) as e:
            _engine(8, 2, hd, 2048)
        assert e.value.code == -2


@pytest.mark.parametrize("n_cols,pos,act", [(700, 0, "f16"), (130, 219, "f32")])
def test_head_dim_64_prefill_chunks_and_decode(n_cols, pos, act):
    # head_dim 64 (the reference's "small head" case) beyond the 16-column pass of its unit test: several 128-column
    # CTA tiles, a chunk that starts past row 0, and the decode kernel on the same cache
    import torch
    nH, nKV, hd = 8, 2, 64
    td = torch.float16 if act == "f16" else torch.float32
    eng = _engine(nH, nKV, hd, pos + n_cols + 8, act=act, max_cols=1024, n_rot=64, rope_mode="f64")
    q, k, v, g = _inputs(9, nH, nKV, hd, pos + n_cols)
    d = lambda a: util.torch_dev(a, td)
    if pos:
        eng.encode_layer(0, 0, d(q[:pos]), d(k[:pos]), d(v[:pos]), d(g[:pos]), mode="prefill")
    out = eng.encode_layer(0, pos, d(q[pos:]), d(k[pos:]), d(v[pos:]), d(g[pos:]), mode="prefill").float().cpu().numpy()
    eng.sync()
    ref, Kf, Vf = _oracle_layer(q, k, v, g, nH, nKV, hd, 64, 1e7, 0)
    gk, gv = util.read_cache(eng, 0, 0, 0, pos + n_cols)
    assert np.array_equal(gk, Kf) and np.array_equal(gv, Vf), "KV append is not bit-exact"
    util.assert_close(out, ref[pos:], f"head_dim 64 prefill at {pos}")
    for c in (0, pos, pos + n_cols - 1):
        qr = eng.rope(d(q[c:c + 1]), nH, c)
        one = eng.decode(0, [(0, c, 1)], qr, d(g[c:c + 1])).float().cpu().numpy()
        util.assert_close(one[0], ref[c], f"head_dim 64 decode at {c}")
    eng.sync()


@pytest.mark.parametrize("n_rot", [64, 128])
@pytest.mark.parametrize("n_cols,pos", [(130, 0), (48, 300), (257, 5)])
def test_head_dim_128_prompts_rotated_in_part_and_in_full(n_rot, n_cols, pos):
    # rotated in part, the 64 dims no rotation touches come from the caller's q: interleaved with its gate, as the q projection delivers both
    import torch
    nH, nKV, hd = 6, 2, 128
    eng = _engine(nH, nKV, hd, pos + n_cols + 8, act="f16", max_cols=512, n_rot=n_rot, rope_mode="f64")
    q, k, v, g = _inputs(8, nH, nKV, hd, pos + n_cols)
    d = lambda a: util.torch_dev(a, torch.float16)
    both = torch.cat([d(q).view(-1, nH, hd), d(g).view(-1, nH, hd)], 2).view(pos + n_cols, -1)
    run = lambda a, b: eng.encode_layer(0, a, both[a:b], d(k[a:b]), d(v[a:b]), both[a:b, hd:], mode="prefill", q_head_stride=2 * hd, gate_head_stride=2 * hd)
    if pos:
        run(0, pos)
    out = run(pos, pos + n_cols).float().cpu().numpy()
    eng.sync()
    ref, Kf, Vf = _oracle_layer(q, k, v, g, nH, nKV, hd, n_rot, 1e7, 0)
    gk, gv = util.read_cache(eng, 0, 0, 0, pos + n_cols)
    assert np.array_equal(gk, Kf) and np.array_equal(gv, Vf), "KV append is not bit-exact"
    util.assert_close(out, ref[pos:], f"{n_cols} columns at {pos}, {n_rot} rotated dims")


def _inputs(cfg_id, nH, nKV, hd, n_cols):
    q = util.normal_f16(0xA11CE + cfg_id, (n_cols, nH * hd)); k = util.normal_f16(0xB0B + cfg_id, (n_cols, nKV * hd))
    v = util.normal_f16(0xC0DE + cfg_id, (n_cols, nKV * hd)); g = util.normal_f16(0x6A7E + cfg_id, (n_cols, nH * hd))
    return q, k, v, g


def _oracle_layer(q, k, v, g, nH, nKV, hd, n_rot, theta, pos, cols=None):
    n = q.shape[0]
    Kf = np.stack([po.f16_rne(po.rope_neox_f64(k[c], nKV, hd, n_rot, pos + c, theta)) for c in range(n)])
    Vf = po.f16_rne(v)
    cols = range(n) if cols is None else cols
    outs = []
    for c in cols:
        qr = po.rope_neox_f64(q[c], nH, hd, n_rot, pos + c, theta)[None]
        outs.append(po.attn_f64(qr, Kf, Vf, nH, nKV, hd, pos + c, 1, None if g is None else g[c:c + 1])[0])
    return np.stack(outs), Kf, Vf


@pytest.mark.parametrize("n_cols,act,gate", [(1024, "f16", False), (300, "f32", True), (129, "f16", True), (1, "f16", False)])
def test_config3_shape_reduced(n_cols, act, gate):
    # 24 q / 4 kv heads, head_dim 256, partial RoPE 64 dims theta 1e7, prompt into an empty cache: RoPE + append + prefill
    import torch
    nH, nKV, hd = 24, 4, 256
    td = torch.float16 if act == "f16" else torch.float32
    eng = _engine(nH, nKV, hd, n_cols + 8, act=act, max_cols=n_cols, rope_mode="f64")
    q, k, v, g = _inputs(3, nH, nKV, hd, n_cols)
    out = eng.encode_layer(0, 0, util.torch_dev(q, td), util.torch_dev(k, td), util.torch_dev(v, td), util.torch_dev(g, td) if gate else None,
                           mode="prefill").float().cpu().numpy()
    eng.sync()
    ref, Kf, Vf = _oracle_layer(q, k, v, g if gate else None, nH, nKV, hd, 64, 1e7, 0)
    gk, gv = util.read_cache(eng, 0, 0, 0, n_cols)
    assert np.array_equal(gk, Kf) and np.array_equal(gv, Vf), "KV append is not bit-exact"
    ma, mr = util.assert_close(out, ref, f"prefill {n_cols}")
    print(f"prefill {n_cols} {act}: max-abs {ma:.2e} max-rel {mr:.2e}")


@pytest.mark.parametrize("hd,n_rot,n_cols", [(256, 96, 150), (256, 128, 40), (256, 192, 203), (128, 48, 77), (64, 48, 19)])
def test_prompts_of_other_rotary_widths(hd, n_rot, n_cols):
    # widths whose groups of eight do not divide the rotation kernel's 64 threads, with (96) and without unrotated dims copied
    import torch
    nH, nKV = 6, 2
    eng = _engine(nH, nKV, hd, n_cols + 8, act="f16", max_cols=n_cols, rope_mode="f64", n_rot=n_rot)
    q, k, v, g = _inputs(31, nH, nKV, hd, n_cols)
    d = lambda a: util.torch_dev(a, torch.float16)
    out = eng.encode_layer(0, 0, d(q), d(k), d(v), d(g), mode="prefill").float().cpu().numpy()
    eng.sync()
    ref, Kf, Vf = _oracle_layer(q, k, v, g, nH, nKV, hd, n_rot, 1e7, 0)
    gk, gv = util.read_cache(eng, 0, 0, 0, n_cols)
    assert np.array_equal(gk, Kf) and np.array_equal(gv, Vf), "KV append is not bit-exact"
    util.assert_close(out, ref, f"n_rot {n_rot}")


@pytest.mark.parametrize("nH,nKV,hd", [(24, 4, 256), (16, 8, 128)])
def test_prefill_gives_the_same_bits_twice(nH, nKV, hd):
    # two threads issue the score products of alternate tiles and two softmax groups take alternate tiles: the order of
    # every sum is fixed all the same, so a repeated pass over the same cache carries the same bits
    import torch
    n_cols = 1500
    eng = _engine(nH, nKV, hd, n_cols + 8, act="f16", max_cols=n_cols, rope_mode="f64")
    q, k, v, g = _inputs(5, nH, nKV, hd, n_cols)
    d = lambda a: util.torch_dev(a, torch.float16)
    dq, dk, dv, dg = d(q), d(k), d(v), d(g)
    outs = [eng.encode_layer(0, 0, dq, dk, dv, dg, mode="prefill").cpu().numpy().view(np.uint16) for _ in range(3)]
    eng.sync()
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2])


def test_chunked_prefill_and_prefill_vs_decode():
    # a second chunk against the first chunk's rows; every column also equals the decode kernel's answer at its position
    import torch
    nH, nKV, hd, n1, n2 = 16, 2, 256, 200, 333
    eng = _engine(nH, nKV, hd, 1024, act="f32", max_cols=512, rope_mode="f64")
    q, k, v, g = _inputs(7, nH, nKV, hd, n1 + n2)
    d = lambda a: util.torch_dev(a)
    o1 = eng.encode_layer(0, 0, d(q[:n1]), d(k[:n1]), d(v[:n1]), d(g[:n1]), mode="prefill").cpu().numpy()
    o2 = eng.encode_layer(0, n1, d(q[n1:]), d(k[n1:]), d(v[n1:]), d(g[n1:]), mode="prefill").cpu().numpy()
    ref, _, _ = _oracle_layer(q, k, v, g, nH, nKV, hd, 64, 1e7, 0)
    util.assert_close(np.concatenate([o1, o2]), ref, "chunked prefill")
    for c in (0, 1, 199, 200, 333, 532):
        qr = eng.rope(d(q[c:c + 1]), nH, c)
        one = eng.decode(0, [(0, c, 1)], qr, d(g[c:c + 1])).cpu().numpy()
        util.assert_close(one[0], ref[c], f"decode at {c}")
    eng.sync()


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("n_cols,pos", [(1, 0), (64, 0), (65, 63), (127, 1), (128, 128), (129, 127), (300, 85)])
@pytest.mark.parametrize("act,order", [("f16", "cols"), ("f16", "heads"), ("f16", "padded"), ("f32", "cols"), ("f32", "heads")])
def test_prefill_at_the_edges_of_its_tiles_and_any_order_of_heads(hd, n_cols, pos, act, order):
    # 128 columns x 128 keys a tile; q and gate as [column][head][dim] with the gate beside q (every copy by TMA), [head][column][dim]
    # (none), or with column strides of no whole 64-dim chunks
    import torch
    nH, nKV = 6, 2
    td = torch.float16 if act == "f16" else torch.float32
    T = pos + n_cols
    eng = _engine(nH, nKV, hd, T + 70, act=act, max_cols=512, rope_mode="none")
    q, g = util.normal_f16(31, (n_cols, nH * hd)), util.normal_f16(32, (n_cols, nH * hd))
    K, V = (po.np_f16_rne(po.normal(33 + i, T * nKV * hd)).reshape(T, -1) for i in range(2))
    poison = np.full((70, nKV * hd), 0x7e00, np.uint16)      # rows past the last one hold NaN
    util.load_cache(eng, 0, 0, np.concatenate([K, poison]), np.concatenate([V, poison]))
    tq, tg = (util.torch_dev(x, td).view(n_cols, nH, hd) for x in (q, g))
    if order == "cols":
        both = torch.cat([tq, tg], 2).view(n_cols, -1)
        out = eng.prefill(0, 0, pos, both, both[:, hd:], q_head_stride=2 * hd, gate_head_stride=2 * hd)
    elif order == "heads":
        q2, g2 = (x.permute(1, 0, 2).contiguous() for x in (tq, tg))
        out = eng.prefill(0, 0, pos, q2.view(-1)[:n_cols * hd].view(n_cols, hd), g2.view(-1)[:n_cols * hd].view(n_cols, hd), q_head_stride=n_cols * hd, gate_head_stride=n_cols * hd)
    else:
        q2, g2 = (torch.nn.functional.pad(x.reshape(n_cols, -1), (0, 8)) for x in (tq, tg))
        out = eng.prefill(0, 0, pos, q2, g2)
    eng.sync()
    util.assert_close(out.float().cpu().numpy(), po.attn_f64(q, K, V, nH, nKV, hd, pos, n_cols, g), f"{n_cols} columns at {pos}, {act} {order}")


@pytest.mark.parametrize("nH,nKV,hd,n_cols,pos,act,gate", [
    (24, 4, 256, 203, 3001, "f32", True),     # two q tiles, the second with 75 rows
    (16, 2, 256, 48, 1500, "f16", True),      # less than one q tile
    (8, 2, 256, 128, 1216, "f16", False),     # 21 tiles in fifths: the last split is one tile, out of sight of half of the rows
    (16, 8, 128, 129, 1000, "f16", True), (8, 2, 64, 65, 700, "f32", False)])
def test_few_columns_behind_a_long_context_split_their_keys(nH, nKV, hd, n_cols, pos, act, gate):
    import torch
    td = torch.float16 if act == "f16" else torch.float32
    eng = _engine(nH, nKV, hd, pos + n_cols + 70, act=act, max_cols=n_cols, rope_mode="none")
    T = pos + n_cols
    q = util.normal_f16(21, (n_cols, nH * hd)); K = po.np_f16_rne(po.normal(22, T * nKV * hd)).reshape(T, -1); V = po.np_f16_rne(po.normal(23, T * nKV * hd)).reshape(T, -1)
    g = util.normal_f16(24, (n_cols, nH * hd)) if gate else None
    poison = np.full((70, nKV * hd), 0x7e00, np.uint16)      # rows past the last one hold NaN
    util.load_cache(eng, 0, 0, np.concatenate([K, poison]), np.concatenate([V, poison]))
    before = eng.stats()["kernel_launches"]
    out = eng.prefill(0, 0, pos, util.torch_dev(q, td), util.torch_dev(g, td) if gate else None)
    eng.sync()
    assert eng.stats()["kernel_launches"] - before == 2      # the keys were split: prefill and merge
    util.assert_close(out.float().cpu().numpy(), po.attn_f64(q, K, V, nH, nKV, hd, pos, n_cols, g), f"split prefill {n_cols} at {pos}")


def test_config3_full_size_properties():
    # the whole 8192-token prompt (0.82 TFLOP): checked on sampled columns against the oracle (the float64 oracle over
    # all 8192 columns takes minutes) and through size-independent properties
    import torch
    nH, nKV, hd, T = 24, 4, 256, 8192
    eng = _engine(nH, nKV, hd, T, act="f16", max_cols=T, rope_mode="f64")
    q, k, v, g = _inputs(3, nH, nKV, hd, T)
    d = lambda a: util.torch_dev(a, torch.float16)
    out = eng.encode_layer(0, 0, d(q), d(k), d(v), None, mode="prefill").float().cpu().numpy()
    eng.sync()
    assert np.all(np.isfinite(out))
    # the first, the last and one interior column of each of the 64 CTA tiles of 128 columns (every CTA of the
    # 24-head x 64-tile schedule has columns under the oracle), plus the first 64-key tile's edges
    rng = np.random.default_rng(3)
    cols = sorted({0, 1, 63, 64} | {t * 128 + o for t in range(T // 128) for o in (0, 127, int(rng.integers(1, 127)))})
    ref, Kf, Vf = _oracle_layer(q, k, v, None, nH, nKV, hd, 64, 1e7, 0, cols)
    ma, mr = util.assert_close(out[cols], ref, "config 3 sampled columns")
    print(f"config 3 full size: {len(cols)} columns, max-abs {ma:.2e} max-rel {mr:.2e}")
    gk, gv = util.read_cache(eng, 0, 0, 0, T)
    assert np.array_equal(gk, Kf) and np.array_equal(gv, Vf), "KV append is not bit-exact at full size"
    # column 0 attends one key: its output is exactly that V row (per kv head), whatever q is
    v0 = po.h2f(Vf[0]).reshape(nKV, hd)
    assert np.allclose(out[0].reshape(nH, hd), np.repeat(v0, nH // nKV, axis=0), atol=1e-3)
    # every output lies inside the range of the V values it can see (a convex combination)
    vmax = np.maximum.accumulate(po.h2f(Vf).reshape(T, nKV, hd), axis=0)[::512]
    o = out[::512].reshape(-1, nKV, nH // nKV, hd)
    assert np.all(o <= vmax[:, :, None, :] + 2e-3)


def _prefill_splits(pos, n_cols, n_heads, hd, sms, slots):
    longest, avg = (pos + n_cols + 63) // 64, (pos + n_cols // 2 + 63) // 64
    rows, ctas, best, best_t = n_cols * n_heads, -(-n_cols // 128) * n_heads, 1, 0.0
    for ns in range(1, 9):
        if ns > 1 and (rows * ns > slots or longest / ns < 4):
            break
        waves = ctas * ns / sms
        t = longest / ns + 8 if waves <= 1 else np.ceil(waves) * (longest / ns + 8) if avg >= 0.8 * longest else waves * (avg / ns + 8) + 0.5 * longest / ns
        if ns > 1:
            t += 6 + rows * ns * (hd * 8.0) / 3.0e6 / 0.8
        if ns == 1 or t < 0.95 * best_t:
            best, best_t = ns, t
    return best


def _rounded_weights(q, K, V, nH, nKV, hd, pos, ns):
    """Attention whose softmax weights are f16 values in the running reference maximum of 64 keys after 64 (moved when it grows by more
    than 2^8), the rest in float64: the keys of each 128 columns in ns splits of whole 64s, each with a reference of its own."""
    n, G, out = q.shape[0], nH // nKV, np.zeros((q.shape[0], nH * hd))
    q, K, V = q.astype(np.float64), po.np_h2f(K).astype(np.float64), po.np_h2f(V).astype(np.float64)
    for c0 in range(0, n, 128):
        cols = np.arange(c0, min(n, c0 + 128))
        keys = pos + cols[-1] + 1
        per = -(-(-(-keys // 64)) // ns) * 64
        for h in range(nH):
            sl, kl = slice(h * hd, (h + 1) * hd), slice(h // G * hd, (h // G + 1) * hd)
            x = q[cols, sl] @ K[:keys, kl].T * (1.4426950408889634 / np.sqrt(hd))
            x[np.arange(keys)[None] > (pos + cols)[:, None]] = -np.inf
            parts = []
            for z in range(0, keys, per):
                m, l, o = np.full(len(cols), -1e30), np.zeros(len(cols)), np.zeros((len(cols), hd))
                for b in range(z, min(keys, z + per), 64):
                    e = min(keys, z + per, b + 64)
                    top = x[:, b:e].max(1)
                    new = np.where((b == 0) | (top > m + 8), np.maximum(top, -1e30), m)
                    w = np.exp2(x[:, b:e] - new[:, None])
                    a = np.exp2(np.maximum(m - new, -2000.0))
                    l, o, m = l * a + w.sum(1), o * a[:, None] + w.astype(np.float16).astype(np.float64) @ V[b:e, kl], new
                parts.append((m, l, o))
            M = np.max([p[0] for p in parts], 0)
            L = sum(l * np.exp2(m - M) for m, l, o in parts)
            out[cols, sl] = sum(o * np.exp2(m - M)[:, None] for m, l, o in parts) / L[:, None]
    return out


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("nH,nKV,pos,n_cols", [(4, 2, 0, 300), (4, 1, 0, 500), (4, 2, 3000, 40), (6, 2, 4031, 130), (6, 1, 1100, 200)])
def test_weights_round_in_the_running_reference_of_64_keys(hd, nH, nKV, pos, n_cols):
    # a result carries the f16 roundings of its weights (2e-4 of itself): they are those of this reference and of these splits, which is
    # what keeps a prompt's f32 outputs the same whatever the kernel's tiles.  What is left are weights that an error of some 3e-6 in 2^y, the
    # sum of a score's products, takes across a rounding's edge: one in 300, 3e-5 of the result
    import torch
    rows = pos + n_cols
    eng = _engine(nH, nKV, hd, rows, max_cols=512)
    K = po.np_f16_rne(po.normal(41, rows * nKV * hd)).reshape(rows, nKV * hd); V = po.np_f16_rne(po.normal(42, rows * nKV * hd)).reshape(rows, nKV * hd)
    util.load_cache(eng, 0, 0, K, V)
    q = util.normal_f16(43, (n_cols, nH * hd))
    out = eng.prefill(0, 0, pos, util.torch_dev(q)).cpu().numpy().astype(np.float64)
    eng.sync()
    slots = max(16384, min(32768, 512 * nH * 8))
    ns = _prefill_splits(pos, n_cols, nH, hd, torch.cuda.get_device_properties(0).multi_processor_count, slots)
    assert (ns > 1) == (pos > 1000)
    ref = _rounded_weights(q, K, V, nH, nKV, hd, pos, ns)
    assert np.linalg.norm(out - ref) / np.linalg.norm(ref) < 8e-5


@pytest.mark.parametrize("hd,nH,nKV,pos,n_cols", [(64, 8, 4, 0, 3000), (128, 8, 4, 0, 3000), (256, 8, 4, 0, 3000), (64, 4, 1, 20000, 70), (128, 4, 1, 20000, 70), (256, 4, 1, 20000, 70)])
def test_many_tiles_repeat_bit_for_bit(hd, nH, nKV, pos, n_cols):
    # scores and weights of up to 160 tiles take turns in the same tensor-memory columns
    import torch
    eng = _engine(nH, nKV, hd, pos + n_cols, act="f32", max_cols=n_cols)
    g = torch.Generator(device="cuda").manual_seed(5)
    for w in "kv":
        c = eng.cache(0, w)
        c.copy_(torch.randn(c.shape, device="cuda", generator=g).half().view(torch.int16))
    q = torch.randn((n_cols, nH * hd), device="cuda", generator=g).half().float()
    outs = [eng.prefill(0, 0, pos, q) for _ in range(12)]
    eng.sync()
    assert torch.isfinite(outs[0]).all() and all(torch.equal(outs[0], o) for o in outs[1:])
    K, V = (eng.cache(0, w)[0].cpu().numpy().view(np.uint16) for w in "kv")
    last = [n_cols - 1]
    ref = po.attn_f64(q[last].cpu().numpy(), K, V, nH, nKV, hd, pos + n_cols - 1, 1)
    util.assert_close(outs[0][last].cpu().numpy(), ref, "last column")


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("pos,n_cols,bad", [(1, 256, 144), (1, 300, 200), (0, 300, 130), (70, 250, 208), (3000, 260, 3136)])
def test_infinite_values_of_later_rows_stay_out_of_earlier_tiles(hd, pos, n_cols, bad):
    # the columns of the first 128 do not see row `bad`, nor do the 16 rows that hold the last that one of them sees: an infinity there leaves
    # them as they are, bit for bit
    import torch
    nH, nKV = 4, 2
    assert bad >= (pos + 128 + 15) // 16 * 16
    eng = _engine(nH, nKV, hd, pos + n_cols, act="f32", max_cols=512)
    g = torch.Generator(device="cuda").manual_seed(6)
    for w in "kv":
        c = eng.cache(0, w)
        c.copy_(torch.randn(c.shape, device="cuda", generator=g).half().view(torch.int16))
    q = torch.randn((n_cols, nH * hd), device="cuda", generator=g).half().float()
    want = eng.prefill(0, 0, pos, q)
    eng.cache(0, "v")[0, bad:bad + 8] = 0x7c00
    got = eng.prefill(0, 0, pos, q)
    eng.sync()
    assert torch.isfinite(want).all() and torch.equal(got[:128], want[:128])
    assert not torch.isfinite(got[bad - pos:]).all()


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("act", ["f16", "f32"])
@pytest.mark.parametrize("n_cols", [100, 300])
def test_prompts_of_any_stride_carry_the_same_bits(hd, act, n_cols):
    # tiles of q, gate and output travel by tensor map, by lanes and by rows, each as its stride and alignment allow
    import torch
    nH, nKV, pos = 4, 2, 37
    td = torch.float16 if act == "f16" else torch.float32
    eng = _engine(nH, nKV, hd, pos + n_cols, act=act, max_cols=512)
    g = torch.Generator(device="cuda").manual_seed(8)
    for w in "kv":
        c = eng.cache(0, w)
        c.copy_(torch.randn(c.shape, device="cuda", generator=g).half().view(torch.int16))
    q, gate = (torch.randn((n_cols, nH * hd), device="cuda", generator=g).to(td) for _ in range(2))
    def at(x, pad, skip=0):      # the same values, rows `pad` values further apart, `skip` past an aligned address
        buf = torch.full((n_cols * (nH * hd + pad) + 64,), float("nan"), device="cuda", dtype=td)
        v = buf[skip:skip + n_cols * (nH * hd + pad)].view(n_cols, -1)[:, :nH * hd]
        return v.copy_(x), buf
    for gt in (None, gate):
        want = eng.prefill(0, 0, pos, q, gt).clone()
        ref = po.attn_f64(q.float().cpu().numpy(), *(eng.cache(0, w)[0].cpu().numpy().view(np.uint16) for w in "kv"), nH, nKV, hd, pos, n_cols, None if gt is None else gt.float().cpu().numpy())
        util.assert_close(want.float().cpu().numpy(), ref, f"{act} {hd}")
        for qp, op in ((0, 8), (8, 0), (64, 72)):
            for gp, skip in ((0, 0), (8, 0), (8, 8), (4, 0), (0, 2), (5, 1)) if gt is not None else ((0, 0),):
                out, buf = at(torch.zeros_like(want), op)
                got = eng.prefill(0, 0, pos, at(q, qp)[0], None if gt is None else at(gt, gp, skip)[0], out=out)
                eng.sync()
                assert torch.equal(got, want), (qp, op, gp, skip)
                assert torch.isnan(buf).sum() == buf.numel() - want.numel()      # nothing written between the rows
