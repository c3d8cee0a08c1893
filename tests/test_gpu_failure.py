"""A bounded device-side wait that runs out: the kernel returns by itself with a status the host reads, the context
latches until pa_reset, and the next step is correct again.  The failure is made on the host side of the protocol: a
two-rank exchange in which the second rank never publishes (its buffer lives on this GPU and nothing writes to it),
with a short polling limit.  Nothing traps, faults or hangs."""
import ctypes as C

import numpy as np
import pytest

from oracle import po
from tests import util

pytestmark = pytest.mark.gpu


def test_exchange_wait_runs_out_then_reset_recovers():
    import torch
    from pooled_b200 import AttnConfig, AttnEngine
    from pooled_b200.lib import PaError
    nH, nKV, hd, rows = 16, 2, 256, 3000
    eng = AttnEngine(AttnConfig(n_heads=nH, n_kv_heads=nKV, head_dim=hd, n_rot=64, rope_theta=1e7, max_seq=4096, rope_mode="none", act_dtype=torch.float32))
    L = eng.L
    K = po.np_f16_rne(po.normal(1, rows * nKV * hd) * 0.7).reshape(rows, nKV * hd); V = po.np_f16_rne(po.normal(2, rows * nKV * hd)).reshape(rows, nKV * hd)
    util.load_cache(eng, 0, 0, K, V)
    q = po.normal(3, nH * hd).astype(np.float32).reshape(1, -1)
    qd = util.torch_dev(q)
    # world 2, this process is rank 0; "rank 1" is a second buffer on this GPU that no one ever writes
    nbytes = L.pa_exchange_bytes(eng.ctx, 2, 64)
    bufs = (C.c_void_p * 2)()
    for r in range(2):
        p = C.c_void_p()
        eng._ck(L.pa_alloc(eng.ctx, nbytes, C.byref(p)))
        bufs[r] = p.value
    # zero both buffers through torch (plain device memory)
    from pooled_b200.attn import _DevArray
    for r in range(2):
        torch.as_tensor(_DevArray(bufs[r], (nbytes,), "|u1"), device="cuda").zero_()
    torch.cuda.synchronize()
    eng._ck(L.pa_exchange_init(eng.ctx, 0, 2, bufs, 64))
    eng.set_wait_limit(3000)                       # a few milliseconds instead of about a second
    out = eng.decode_exchange(0, [(0, rows - 1, 1)], qd)
    with pytest.raises(PaError) as ei:
        eng.sync()                                 # the kernel came back by itself; the host reads its status
    assert ei.value.code == -5                     # PA_ETIMEOUT
    with pytest.raises(PaError) as ei:
        eng.decode(0, [(0, rows - 1, 1)], qd)      # latched: every call is refused until reset
    assert ei.value.code == -6                     # PA_ESTATE
    eng.reset()
    eng.set_wait_limit(0)
    got = eng.decode(0, [(0, rows - 1, 1)], qd).cpu().numpy()
    eng.sync()
    ref = po.attn_f64(q, K, V, nH, nKV, hd, rows - 1, 1)
    assert util.errs(got, ref)[1] < util.REF_REL
    # the unfinished exchange left its partial answer: finite, and the merge over the one rank that did publish
    assert np.all(np.isfinite(out.cpu().numpy()))
    for r in range(2):
        L.pa_free(eng.ctx, C.c_void_p(bufs[r]))


def _f16_and_f32_token(fmt, nH, nKV, hd, rows, monkeypatch=None):
    import torch
    from pooled_b200 import AttnConfig, AttnEngine
    eng = AttnEngine(AttnConfig(n_heads=nH, n_kv_heads=nKV, head_dim=hd, n_rot=64, rope_theta=1e7, max_seq=rows, rope_mode="none", act_dtype=torch.float32, kv_format=fmt))
    g = torch.Generator(device="cuda").manual_seed(11)
    for w in "kv":
        c = eng.cache(0, w)
        x = torch.randn(c.shape, device="cuda", generator=g)
        c.copy_(x.half().view(torch.int16) if fmt == "f16" else x)
    q, gate = torch.randn((2, 1, nH * hd), device="cuda", generator=g)
    return eng, q, gate


def test_merge_wait_runs_out_then_reset_recovers():
    # one look for the records of CTAs that are still at their rows: the call comes back by itself with a status, records that came late
    # stay in the buffer, and after a reset the bits are those of before
    import torch
    from pooled_b200.lib import PaError
    rows = 40000
    eng, q, gate = _f16_and_f32_token("f16", 16, 2, 256, rows)
    want = eng.decode(0, [(0, rows - 1, 1)], q, gate).clone()
    eng.sync()
    for _ in range(3):
        eng.set_wait_limit(1)
        for _ in range(50):                        # (CTAs in step may all be in time, in one call)
            eng.decode(0, [(0, rows - 1, 1)], q, gate)
        with pytest.raises(PaError) as ei:
            eng.sync()
        assert ei.value.code == -5                 # PA_ETIMEOUT
        with pytest.raises(PaError) as ei:
            eng.decode(0, [(0, rows - 1, 1)], q, gate)
        assert ei.value.code == -6                 # PA_ESTATE
        eng.reset()
        eng.set_wait_limit(0)
        got = [eng.decode(0, [(0, n - 1, 1)], q, gate).clone() for n in (rows, 9000, rows)]
        eng.sync()
        assert torch.equal(got[0], want) and torch.equal(got[2], want) and torch.isfinite(got[1]).all()


@pytest.mark.parametrize("nH,nKV,hd,rows", [(1, 1, 256, 40000), (4, 1, 256, 9000), (16, 8, 128, 3000), (16, 8, 128, 6000), (2, 2, 64, 5000), (13, 13, 64, 1000)])
def test_f32_units_left_to_the_last_cta_carry_the_same_bits(nH, nKV, hd, rows, monkeypatch):
    # from a single look for the others' records, which leaves nearly every unit, to none left
    import torch
    monkeypatch.setenv("POOLED_ATTN_NO_MERGE", "1")
    ref, q, gate = _f16_and_f32_token("f32", nH, nKV, hd, rows)
    ctx = (rows, rows // 2 + 1, rows)
    want = [ref.decode(0, [(0, n - 1, 1)], q, g).clone() for n in ctx for g in (None, gate)]
    ref.sync()
    monkeypatch.delenv("POOLED_ATTN_NO_MERGE")
    eng, q, gate = _f16_and_f32_token("f32", nH, nKV, hd, rows)
    for limit in (1, 2, 3, 5, 9, 20, 0):
        eng.set_wait_limit(limit)
        for _ in range(20):
            got = [eng.decode(0, [(0, n - 1, 1)], q, g) for n in ctx for g in (None, gate)]
        eng.sync()
        assert all(torch.equal(a, b) for a, b in zip(got, want)), limit


def test_f32_token_beside_a_long_kernel_of_another_stream():
    # the call has a CTA for every SM, sixteen of which merge, and a kernel that watches the clock for three seconds and ends leaves it eight
    # SMs: no CTA waits for one that has none, and the call is right and done before that kernel is
    import torch
    rows = 40000
    eng, q, gate = _f16_and_f32_token("f32", 4, 1, 256, rows)      # (whose CTAs take all registers of an SM)
    want = eng.decode(0, [(0, rows - 1, 1)], q, gate).clone()
    eng.sync()
    got, side, main = [torch.empty_like(want) for _ in range(3)], torch.cuda.Stream(), torch.cuda.Stream()
    watch = torch.cuda._compile_kernel("""extern "C" __global__ void watch(long long ns) {
        long long t0, t;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
        do { __nanosleep(1000); asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t)); } while (t >= t0 && t - t0 < ns);
    }""", "watch")
    n = torch.cuda.get_device_properties(0).multi_processor_count - 8
    end = torch.cuda.Event()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        watch(grid=(n, 1, 1), block=(1024, 1, 1), args=[3_000_000_000])
        end.record()
    with torch.cuda.stream(main):
        for g in got:
            eng.decode(0, [(0, rows - 1, 1)], q, gate, out=g)
        eng.sync()
    assert not end.query()
    torch.cuda.synchronize()
    assert all(torch.equal(g, want) for g in got)
