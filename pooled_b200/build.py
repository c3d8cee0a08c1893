"""Builds libpooled_attn.so in-tree with nvcc for sm_100a (no other architecture, no JIT cache)."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "libpooled_attn.so")
CALL_OUT = os.path.join(HERE, "_pa_call" + sysconfig.get_config_var("EXT_SUFFIX"))   # CPython module: the per-layer calls without ctypes
SOURCES = ["pa_api.cu", "pa_rope_append.cu", "pa_decode.cu", "pa_prefill.cu", "pa_verify.cu", "pa_kvfmt.cu", "pa_q8.cu", "pa_front.cu", "pa_noalloc.cu"]
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo", "--use_fast_math=false",
         "-Xcompiler", "-fPIC,-fvisibility=hidden", "--expt-relaxed-constexpr"]


def nvcc() -> str:
    for c in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if c and os.path.exists(c):
            return c
    raise RuntimeError("nvcc not found: libpooled_attn.so cannot be built (there is no CPU fallback)")


def _deps() -> list[str]:
    return [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(HERE, "..", "include", "pooled_attn.h")]


def _call_cmd() -> list[str] | None:
    """The command that builds the call module; None without a C compiler or this Python's headers (ctypes makes the calls then)."""
    cc, inc = shutil.which("gcc") or shutil.which("cc"), sysconfig.get_paths()["include"]
    if not cc or not os.path.exists(os.path.join(inc, "Python.h")):
        return None
    return [cc, "-O2", "-shared", "-fPIC", "-I" + inc, os.path.join(CSRC, "pa_call.c"), "-o", CALL_OUT]


def needs_build() -> bool:
    outs = [OUT, CALL_OUT] if _call_cmd() else [OUT]
    if not all(os.path.exists(o) for o in outs):
        return True
    t = min(os.path.getmtime(o) for o in outs)
    return any(os.path.getmtime(d) > t for d in _deps())


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return OUT
    objs = []
    bdir = os.path.join(HERE, "build")
    os.makedirs(bdir, exist_ok=True)
    procs = []
    for s in SOURCES:
        o = os.path.join(bdir, s.replace(".cu", ".o"))
        objs.append(o)
        cmd = [nvcc(), *[f for f in FLAGS if f != "--use_fast_math=false"], "-c", os.path.join(CSRC, s), "-o", o]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((s, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for s, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            sys.stderr.write(f"--- {s} ---\n{out}\n")
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    cmd = _call_cmd()
    if cmd:
        subprocess.check_call(cmd)
    else:
        sys.stderr.write("no C compiler or no Python headers: the per-layer calls go through ctypes, some 5 us slower each\n")
        if os.path.exists(CALL_OUT):
            os.remove(CALL_OUT)       # of an older source
    subprocess.check_call([nvcc(), "-shared", "-o", OUT, *objs, "-lcudart_static", "-lpthread", "-ldl", "-lrt"])
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
