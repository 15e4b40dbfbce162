"""Builds the sm_100a CUDA library of torchturbo_b200 with plain nvcc.

The kernels expose a C ABI (`extern "C"`), take raw device pointers plus the CUDA
stream handle, and are loaded with ctypes, so no torch headers are needed and a
full rebuild takes seconds.  The shared object is written next to the package
(`torchturbo_b200/_lib/libttb200.so`).  `host.cpp`, the launch functions of the hot
operators, is a small extension module against the framework's headers beside it
(`ttb_host.so`).
"""
from __future__ import annotations

import hashlib
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import torch

CSRC = Path(__file__).resolve().parent
LIB_DIR = CSRC.parent / "_lib"
LIB_PATH = LIB_DIR / "libttb200.so"
HOST_SOURCE, HOST_PATH = CSRC / "host.cpp", LIB_DIR / "ttb_host.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC,-fvisibility=hidden",
    "--expt-relaxed-constexpr",
]
# Approximate exponentials, divisions and roots wherever a result leaves in bf16 anyway.  Sources whose fp32 results stand in
# for fp32 torch operations are compiled without; -ftz alone keeps an exp2f at one instruction.
FAST_MATH = ["--use_fast_math"]
PRECISE = {"delta_chunk.cu": [], "delta_chunk_vec.cu": ["-ftz=true"], "gates.cu": []}
HOST_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
HOST_LIBS = ["-ltorch_python", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-ltorch"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _digest(paths: list[Path]) -> str:
    h = hashlib.sha256()
    for p in sorted(paths) + sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.h")) + [HOST_SOURCE]:
        h.update(p.name.encode())
        h.update(p.read_bytes())
    h.update(" ".join(NVCC_FLAGS + FAST_MATH + HOST_FLAGS + HOST_LIBS).encode())
    h.update(repr(sorted(PRECISE.items())).encode())
    h.update(f"{torch.__version__} {sys.version}".encode())
    return h.hexdigest()


def _host_command() -> list[str]:
    inc = Path(torch.__file__).resolve().parent
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    return [os.environ.get("CXX", "g++"), *HOST_FLAGS,
            f"-I{inc}/include", f"-I{inc}/include/torch/csrc/api/include", f"-I{cuda}/include", f"-I{sysconfig.get_paths()['include']}",
            str(HOST_SOURCE), "-o", str(HOST_PATH), f"-L{inc}/lib", *HOST_LIBS, f"-L{LIB_DIR}", f"-l:{LIB_PATH.name}", "-Wl,-rpath,$ORIGIN"]


def build(force: bool = False, verbose: bool = False, ptxas_info: bool = False) -> Path:
    """Compile every `.cu` under csrc/ and link them into one shared object."""
    LIB_DIR.mkdir(exist_ok=True)
    srcs = sources()
    stamp = LIB_DIR / "build.stamp"
    digest = _digest(srcs)
    if not force and LIB_PATH.exists() and HOST_PATH.exists() and stamp.exists() and stamp.read_text() == digest:
        return LIB_PATH
    nvcc = _nvcc()
    obj_dir = LIB_DIR / "obj"
    obj_dir.mkdir(exist_ok=True)
    flags = list(NVCC_FLAGS) + (["-Xptxas", "-v"] if ptxas_info else [])

    def compile_one(src: Path) -> Path:
        obj = obj_dir / (src.stem + ".o")
        cmd = [nvcc, *flags, *PRECISE.get(src.name, FAST_MATH), "-I", str(CSRC), "-c", str(src), "-o", str(obj)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{res.stdout}\n{res.stderr}")
        if verbose or ptxas_info:
            sys.stderr.write(res.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        objs = list(ex.map(compile_one, srcs))
    cmd = [nvcc, "-shared", "-o", str(LIB_PATH), *map(str, objs), "-lcudart"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    res = subprocess.run(_host_command(), capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"{HOST_SOURCE.name} failed:\n{res.stdout}\n{res.stderr}")
    stamp.write_text(digest)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True, ptxas_info="--ptxas" in sys.argv))
