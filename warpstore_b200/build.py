"""Builds libwarpstore_b200.so in-tree (sm_100a) with nvcc.

Steps: embed the device headers the code generator compiles at run time (ws_types.h, ws_dev.cuh,
ws_kern.cuh) as string literals, compile every translation unit for
`-gencode arch=compute_100a,code=sm_100a`, link against cudart, the driver API and NVRTC.
Objects go to warpstore_b200/_build/; unchanged sources are not recompiled.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(ROOT, "include")
BUILD = os.path.join(HERE, "_build")
LIB = os.path.join(HERE, "libwarpstore_b200.so")

# the interpreter instantiations first: they take longest
SOURCES = ["ws_interp_priv.cu", "ws_interp_hash.cu", "ws_interp_agg.cu", "ws_interp_select.cu", "ws_runtime.cu",
           "ws_plan.cpp", "ws_codegen.cpp", "ws_ops.cu", "ws_select_join.cu", "ws_noalloc.cu", "ws_rel.cu",
           "ws_encode.cu", "ws_estimate.cu", "ws_serve.cpp", "ws_tune.cpp", "ws_tier.cu"]
EMBED = [("kWsTypesSrc", os.path.join(INCLUDE, "ws_types.h")),
         ("kWsDevSrc", os.path.join(CSRC, "ws_dev.cuh")),
         ("kWsKernSrc", os.path.join(CSRC, "ws_kern.cuh"))]
HEADERS = [p for _, p in EMBED] + [os.path.join(CSRC, f) for f in ("ws_internal.h", "ws_interp.cuh", "ws_shape.h")] + \
    [os.path.join(INCLUDE, "ws_b200.h")]


def cuda_home() -> str:
    nvcc = shutil.which("nvcc")
    if nvcc:
        return os.path.dirname(os.path.dirname(os.path.realpath(nvcc)))
    return "/usr/local/cuda"


def _embed() -> str:
    out = os.path.join(BUILD, "ws_jit_sources.h")
    parts = ["// Generated by warpstore_b200/build.py: device headers for run-time compilation.\n#pragma once\n"]
    for name, path in EMBED:
        src = open(path).read()
        assert ")WSSRC\"" not in src
        parts.append(f'static const char* const {name} = R"WSSRC({src})WSSRC";\n')
    text = "".join(parts)
    if not os.path.exists(out) or open(out).read() != text:
        with open(out, "w") as f:
            f.write(text)
    return out


def _stale(obj: str, deps: list[str]) -> bool:
    if not os.path.exists(obj):
        return True
    t = os.path.getmtime(obj)
    return any(os.path.getmtime(d) > t for d in deps)


def _compile(src: str, nvcc: str, verbose: bool) -> str:
    obj = os.path.join(BUILD, os.path.basename(src) + ".o")
    deps = [src] + HEADERS + [os.path.join(BUILD, "ws_jit_sources.h")]
    if not _stale(obj, deps):
        return obj
    cmd = [nvcc, "-c", src, "-o", obj, "-std=c++17", "-O3", "-lineinfo",
           "-gencode", "arch=compute_100a,code=sm_100a",
           "--default-stream", "per-thread", "-Xcompiler", "-fPIC,-Wall",
           "--expt-relaxed-constexpr", "-I", INCLUDE, "-I", CSRC, "-I", BUILD]
    if src.endswith(".cpp"):
        cmd[1:1] = ["-x", "cu"]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
    if verbose and r.stderr:
        sys.stderr.write(r.stderr)
    return obj


def build(verbose: bool = False) -> str:
    os.makedirs(BUILD, exist_ok=True)
    _embed()
    home = cuda_home()
    nvcc = os.path.join(home, "bin", "nvcc")
    srcs = [os.path.join(CSRC, s) for s in SOURCES]
    with cf.ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 4)) as ex:
        objs = list(ex.map(lambda s: _compile(s, nvcc, verbose), srcs))
    if _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-o", LIB + ".tmp"] + objs + [
            "-gencode", "arch=compute_100a,code=sm_100a",
            "-L", os.path.join(home, "lib64"),
            "-lcudart", "-lnvrtc", "-Xlinker", "-rpath," + os.path.join(home, "lib64")]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
        os.replace(LIB + ".tmp", LIB)
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv))
