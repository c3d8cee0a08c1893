"""ctypes binding of libpooled_attn.so (include/pooled_attn.h).  Fails loudly when the library is missing."""
from __future__ import annotations

import ctypes as C
import importlib.machinery
import importlib.util
import os
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
SO_PATH = os.path.join(HERE, "libpooled_attn.so")
CALL_PATH = os.path.join(HERE, "_pa_call" + sysconfig.get_config_var("EXT_SUFFIX"))   # of this interpreter's ABI only

PA_F32, PA_F16 = 0, 1
PA_ROPE_NONE, PA_ROPE_F64, PA_ROPE_TABLE = 0, 1, 2
PA_KV_F16, PA_KV_Q8, PA_KV_F32 = 0, 1, 2
PA_FLAG_FAST = 1
PA_MODE_AUTO, PA_MODE_DECODE, PA_MODE_PREFILL = 0, 1, 2
STATUS = {0: "PA_OK", -1: "PA_EINVAL", -2: "PA_EUNSUPPORTED", -3: "PA_ENOMEM", -4: "PA_ECUDA", -5: "PA_ETIMEOUT", -6: "PA_ESTATE"}


class PaError(RuntimeError):
    def __init__(self, code: int, msg: str):
        super().__init__(f"{STATUS.get(code, code)}: {msg}")
        self.code = code


class PaConfig(C.Structure):
    _fields_ = [("n_heads", C.c_uint32), ("n_kv_heads", C.c_uint32), ("head_dim", C.c_uint32), ("n_rot", C.c_uint32),
                ("rope_theta", C.c_double), ("rope_mode", C.c_uint32), ("act_dtype", C.c_uint32), ("max_cols", C.c_uint32),
                ("splits", C.c_uint32), ("flags", C.c_uint32), ("reserved", C.c_uint32 * 5)]


class PaItem(C.Structure):
    _fields_ = [("seq", C.c_uint32), ("pos", C.c_uint32), ("n_cols", C.c_uint32), ("reserved", C.c_uint32)]


class PaStats(C.Structure):
    _fields_ = [("kernel_launches", C.c_uint64), ("kv_bytes_streamed", C.c_uint64), ("calls", C.c_uint64)]


# name -> (restype, argtypes): every symbol include/pooled_attn.h declares
_vp, _u32, _u64, _i, _sz = C.c_void_p, C.c_uint32, C.c_uint64, C.c_int, C.c_size_t
SYMBOLS = {
    "pa_create": (_i, [_i, C.POINTER(PaConfig), C.POINTER(_vp)]),
    "pa_destroy": (_i, [_vp]),
    "pa_layer_create": (_i, [_vp, _u32, _u32, C.POINTER(_vp)]),
    "pa_layer_create_fmt": (_i, [_vp, _u32, _u32, _i, C.POINTER(_vp)]),
    "pa_layer_destroy": (_i, [_vp]),
    "pa_layer_set_origin": (_i, [_vp, _u32]),
    "pa_layer_set_next": (_i, [_vp, _vp]),
    "pa_cache_ptr": (_vp, [_vp, _i]),
    "pa_cache_export": (_i, [_vp, _u32, _u32, _u32, _i, _vp, C.POINTER(_u32), _vp]),
    "pa_cache_import": (_i, [_vp, _u32, _u32, _u32, _i, _vp, C.POINTER(_u32), _vp]),
    "pa_slot_save": (_i, [_vp, _u32, _u32, C.POINTER(_vp), _vp]),
    "pa_slot_load": (_i, [_vp, _u32, _vp, C.POINTER(_u32), _vp]),
    "pa_slot_export": (_i, [_vp, _i, _vp, _vp]),
    "pa_slot_info": (_i, [_vp, C.POINTER(_u32), C.POINTER(_u32), C.POINTER(_u32)]),
    "pa_slot_drop": (_i, [_vp]),
    "pa_last_error": (C.c_char_p, [_vp]),
    "pa_version": (C.c_char_p, []),
    "pa_sync": (_i, [_vp, _vp]),
    "pa_reset": (_i, [_vp]),
    "pa_alloc": (_i, [_vp, _sz, C.POINTER(_vp)]),
    "pa_free": (_i, [_vp, _vp]),
    "pa_alloc_host": (_i, [_vp, _sz, C.POINTER(_vp)]),
    "pa_free_host": (_i, [_vp, _vp]),
    "pa_upload": (_i, [_vp, _vp, _vp, _sz, _vp]),
    "pa_download": (_i, [_vp, _vp, _vp, _sz, _vp]),
    "pa_dec_config": (_u32, [_u32, _u32, _u32, _u32]),
    "pa_dec_split_len": (_u32, [_u32, _u32]),
    "pa_dec_splits": (_u32, [_u32, _u32]),
    "pa_tile_split_len": (_u32, [_u32, _u32, _u32, _u32]),
    "pa_plan_splits": (_u32, [_vp, _u32, _u32]),
    "pa_rope": (_i, [_vp, _vp, _u64, _u64, _u32, _u32, _u32, _vp, _vp, _u64, _vp]),
    "pa_kv_append": (_i, [_vp, _u32, _u32, _u32, _vp, _vp, _u64, _i, _vp]),
    "pa_rope_append": (_i, [_vp, _u32, _u32, _u32, _vp, _u64, _u64, _vp, _vp, _u64, _vp, _vp, _vp]),
    "pa_rope_append_items": (_i, [_vp, _vp, _u32, _vp, _u64, _u64, _vp, _vp, _u64, _vp, _vp]),
    "pa_decode": (_i, [_vp, C.POINTER(PaItem), _u32, _vp, _i, _u64, _u64, _vp, _u64, _u64, _vp, _u64, _vp]),
    "pa_decode_gather": (_i, [_vp, _u32, _u32, _vp, _u32, _vp, _i, _u64, _u64, _vp, _u64, _u64, _vp, _u64, _vp]),
    "pa_decode_partial": (_i, [_vp, C.POINTER(PaItem), _u32, _vp, _i, _u64, _u64, _vp, _vp]),
    "pa_merge": (_i, [_vp, _vp, _u32, _u32, _vp, _u64, _u64, _vp, _u64, _vp]),
    "pa_exchange_bytes": (_sz, [_vp, _u32, _u32]),
    "pa_shared_alloc": (_i, [_vp, _sz, C.POINTER(_vp), _vp]),
    "pa_shared_open": (_i, [_vp, _vp, C.POINTER(_vp)]),
    "pa_shared_close": (_i, [_vp, _vp]),
    "pa_exchange_init": (_i, [_vp, _u32, _u32, C.POINTER(_vp), _u32]),
    "pa_decode_exchange": (_i, [_vp, C.POINTER(PaItem), _u32, _vp, _i, _u64, _u64, _vp, _u64, _u64, _vp, _u64, _vp]),
    "pa_attn_items": (_i, [_vp, _vp, _u32, _vp, _u64, _u64, _vp, _vp, _u64, _vp, _u64, _u64, _vp, _u64, C.c_int, _vp]),
    "pa_attn_layer_sharded": (_i, [_vp, _u32, _u32, _u32, _vp, _u64, _u64, _vp, _vp, _u64, _vp, _u64, _u64, _vp, _vp, _u64, _vp]),
    "pa_prefill": (_i, [_vp, _u32, _u32, _u32, _vp, _i, _u64, _u64, _vp, _u64, _u64, _vp, _u64, _vp]),
    "pa_sigmoid_mul": (_i, [_vp, _vp, _u64, _vp, _u64, _u64, _u32, _vp]),
    "pa_layer_set_head_norm": (_i, [_vp, _vp, _vp, C.c_double]),
    "pa_head_norm": (_i, [_vp, _vp, _u64, _u64, _u32, _u32, _vp, C.c_double, _vp, _u64, _u64, _vp]),
    "pa_attn_layer": (_i, [_vp, _u32, _u32, _u32, _i, _vp, _u64, _u64, _vp, _vp, _u64, _vp, _u64, _u64, _vp, _vp, _u64, _vp]),
    "pa_attn_layer_host": (_i, [_vp, _u32, _u32, _u32, _i, _vp, _u64, _u64, _vp, _vp, _u64, _vp, _u64, _u64, _vp, _vp, _u64, _vp]),
    "pa_attn_step_host": (_i, [C.POINTER(_vp), _u32, _u32, _u32, _u32, _i, _vp, _u64, _u64, _u64, _vp, _vp, _u64, _u64, _vp, _u64, _u64, _u64, _vp, _u64, _u64, _vp]),
    "pa_decode_static": (_i, [_i, _vp, _vp, _u32, _u32, _u32, _u32, _u32, _u32, _vp, _vp, _vp, _vp, C.c_char_p, _sz]),
    "pa_decode_static_status": (_i, [_i, _vp, C.POINTER(_u32)]),
    "pa_set_wait_limit": (_i, [_vp, _u32]),
    "pa_get_stats": (_i, [_vp, C.POINTER(PaStats)]),
    "pa_timing_begin": (_i, [_vp, _u32]),
    "pa_set_core_only": (_i, [_vp, _i]),
    "pa_timing_end": (_i, [_vp, C.POINTER(C.c_double), C.POINTER(_u64)]),
}


def _ptr(t):
    return None if t is None else t.data_ptr()


def _gate(t, head_stride):
    return (None, 0, 0) if t is None else (t.data_ptr(), t.stride(0), head_stride)


class CtypesCalls:
    """What csrc/pa_call.c does, by ctypes (`entry` is not needed: the functions are the library's)."""

    def __init__(self, lib):
        self.lib = lib

    def attn_layer(self, entry, layer, seq, pos, mode, q, q_head_stride, k, v, gate, gate_head_stride, cs_table, out, stream):
        return self.lib.pa_attn_layer(layer, seq, pos, q.shape[0], mode, _ptr(q), q.stride(0), q_head_stride, _ptr(k), _ptr(v), k.stride(0),
                                      *_gate(gate, gate_head_stride), _ptr(cs_table), _ptr(out), out.stride(0), stream)

    def attn_items(self, entry, layer, seqs_pos, q, q_head_stride, k, v, gate, gate_head_stride, out, exchange, stream):
        items = (PaItem * max(1, len(seqs_pos)))(*[PaItem(s, p, 1, 0) for s, p in seqs_pos])
        return self.lib.pa_attn_items(layer, items, len(seqs_pos), _ptr(q), q.stride(0), q_head_stride, _ptr(k), _ptr(v), k.stride(0),
                                      *_gate(gate, gate_head_stride), _ptr(out), out.stride(0), exchange, stream)

    def rope_append(self, entry, layer, seq, pos, q, q_head_stride, k, v, cs_table, q_rot, stream):
        return self.lib.pa_rope_append(layer, seq, pos, q.shape[0], _ptr(q), q.stride(0), q_head_stride, _ptr(k), _ptr(v), k.stride(0), _ptr(cs_table),
                                       _ptr(q_rot), stream)

    def decode_gather(self, entry, layer, seq, lists, list_stride, q, q_dtype, q_head_stride, gate, gate_head_stride, out, stream):
        return self.lib.pa_decode_gather(layer, seq, q.shape[0], _ptr(lists), list_stride, _ptr(q), q_dtype, q.stride(0), q_head_stride,
                                         *_gate(gate, gate_head_stride), _ptr(out), out.stride(0), stream)


class Lib:
    """The loaded shared library with typed entry points."""

    def __init__(self, path: str = SO_PATH):
        if not os.path.exists(path):
            raise PaError(-4, f"{path} is missing: build it with `python -m pooled_b200.build` (nvcc, sm_100a). "
                              "There is no CPU or PyTorch fallback for the attention path.")
        self.path = path
        self.dll = C.CDLL(path)
        for name, (res, args) in SYMBOLS.items():
            fn = getattr(self.dll, name)   # AttributeError when the library lacks a declared symbol
            fn.restype, fn.argtypes = res, args
            setattr(self, name, fn)
        self.call = self._load_call()

    def _load_call(self):
        """The CPython module with the per-layer calls (csrc/pa_call.c), which takes their addresses in this library from
        `entry`; the same calls through ctypes where it was not built for this interpreter."""
        self.entry = {n: C.cast(getattr(self.dll, n), C.c_void_p).value for n in ("pa_attn_layer", "pa_attn_items", "pa_rope_append", "pa_decode_gather")}
        if not os.path.exists(CALL_PATH):
            return CtypesCalls(self)
        loader = importlib.machinery.ExtensionFileLoader("_pa_call", CALL_PATH)
        mod = importlib.util.module_from_spec(importlib.util.spec_from_file_location("_pa_call", CALL_PATH, loader=loader))
        loader.exec_module(mod)
        return mod

    def check(self, rc: int, ctx=None):
        if rc != 0:
            msg = self.pa_last_error(ctx)
            raise PaError(rc, msg.decode() if msg else "")


_lib: Lib | None = None


def load() -> Lib:
    global _lib
    if _lib is None:
        _lib = Lib()
    return _lib
