"""Builds libddf_b200.so from the CUDA sources in this directory with nvcc for
sm_100a (cross-compiles without a GPU).  The library links the CUDA runtime
statically and has no other dependency, so it loads in any process.
Then builds _native.so (native.cpp, g++ against the installed torch): the host
path of the Python operator.

    python -m ddfnet_b200.csrc.build [--force] [-DNAME=VALUE ...] [--out NAME]
"""
from __future__ import annotations

import concurrent.futures as cf
import hashlib
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.dirname(HERE)
SOURCES = ["abi.cu", "bwd_stream.cu", "layout.cu", "channel_branch.cu", "probe.cu", "nhwc.cu", "sfnorm.cu", "stream_inst_f32.cu", "stream_inst_f16.cu",
           "stream_inst_bf16.cu", "ring_inst_f16.cu", "ring_inst_bf16.cu", "row_inst_f16.cu", "row_inst_bf16.cu", "row_inst_f32.cu", "bwd_inst_f32.cu", "bwd_inst_f16.cu", "bwd_inst_bf16.cu",
           "maxpool.cu", "band.cu", "band_bwd_inst_f32.cu", "band_bwd_inst_f16.cu", "band_bwd_inst_bf16.cu", "band_inst_f32.cu",
           "band_inst_f16.cu", "band_inst_bf16.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
              "-Xcompiler", "-fPIC"]


def _nvcc() -> str:
    cand = os.environ.get("NVCC") or "/usr/local/cuda/bin/nvcc"
    return cand if os.path.exists(cand) else "nvcc"


def _deps() -> list[str]:
    return sorted(os.path.join(HERE, f) for f in os.listdir(HERE)
                  if f.endswith((".cu", ".cuh", ".inc", ".h"))) + [
        os.path.join(os.path.dirname(PKG), "include", "ddf_b200.h")]


def _fingerprint(defines: list[str]) -> str:
    h = hashlib.sha256()
    for p in _deps():
        h.update(p.encode())
        with open(p, "rb") as f:
            h.update(f.read())
    h.update(" ".join(NVCC_FLAGS + defines).encode())
    return h.hexdigest()


def build(force: bool = False, defines: list[str] | None = None,
          out_name: str = "libddf_b200.so", verbose: bool = False) -> str:
    defines = list(defines or [])
    out = os.path.join(PKG, out_name)
    stamp = out + ".stamp"
    fp = _fingerprint(defines)
    if not force and os.path.exists(out) and os.path.exists(stamp):
        with open(stamp) as f:
            if f.read().strip() == fp:
                return out
    bdir = os.path.join(HERE, "build", out_name.replace(".so", ""))
    os.makedirs(bdir, exist_ok=True)
    nvcc = _nvcc()

    def compile_one(src: str) -> str:
        obj = os.path.join(bdir, src.replace(".cu", ".o"))
        cmd = [nvcc] + NVCC_FLAGS + defines + ["-c", os.path.join(HERE, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
        if verbose:
            sys.stderr.write(r.stderr)
        return obj

    with cf.ThreadPoolExecutor(max_workers=min(8, len(SOURCES))) as ex:
        objs = list(ex.map(compile_one, SOURCES))
    link = [nvcc, "-shared", "-cudart", "static", "-gencode", "arch=compute_100a,code=sm_100a",
            "-o", out + ".tmp"] + objs
    r = subprocess.run(link, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    os.replace(out + ".tmp", out)
    with open(stamp, "w") as f:
        f.write(fp)
    return out


def build_native(force: bool = False) -> str:
    """Compiles native.cpp into ddfnet_b200/_native.so."""
    import sysconfig

    import torch
    src, out = os.path.join(HERE, "native.cpp"), os.path.join(PKG, "_native.so")
    root = os.path.dirname(os.path.abspath(torch.__file__))
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-I{root}/include", f"-I{root}/include/torch/csrc/api/include", f"-I{cuda}/include",
           f"-I{sysconfig.get_paths()['include']}", src, "-o", out + ".tmp", f"-L{root}/lib",
           "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", f"-Wl,-rpath,{root}/lib"]
    h = hashlib.sha256((" ".join(cmd) + torch.__version__).encode())
    for p in (src, os.path.join(os.path.dirname(PKG), "include", "ddf_b200.h")):
        with open(p, "rb") as f:
            h.update(f.read())
    stamp = out + ".stamp"
    if not force and os.path.exists(out) and os.path.exists(stamp):
        with open(stamp) as f:
            if f.read() == h.hexdigest():
                return out
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed on native.cpp:\n{r.stderr}")
    os.replace(out + ".tmp", out)
    with open(stamp, "w") as f:
        f.write(h.hexdigest())
    return out


if __name__ == "__main__":
    args = sys.argv[1:]
    force = "--force" in args
    verbose = "-v" in args
    defs = [a for a in args if a.startswith("-D")]
    name = "libddf_b200.so"
    if "--out" in args:
        name = args[args.index("--out") + 1]
    print(build(force=force, defines=defs, out_name=name, verbose=verbose))
    print(build_native(force=force))
