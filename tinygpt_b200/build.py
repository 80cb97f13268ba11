"""Build the sm_100a shared library in-tree with nvcc (no JIT cache: the .so travels with the repo snapshot).

    python -m tinygpt_b200.build [--force] [--verbose]

Output: tinygpt_b200/lib/libb200decode.so  (C ABI declared in include/b200_decode.h) and, linked to torch alone,
tinygpt_b200/lib/b200ops.so  (the operators of ops.py as native functions, csrc/torch_ops.cpp).
"""
from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
ROOT = PKG.parent
CSRC = PKG / "csrc"
LIB_DIR = PKG / "lib"
OBJ_DIR = LIB_DIR / "obj"
LIB_PATH = LIB_DIR / "libb200decode.so"
NATIVE_PATH = LIB_DIR / "b200ops.so"

SOURCES = ["common.cu", "gemv.cu", "gemv_batch.cu", "gemm.cu", "prefill.cu", "prefill_attn.cu", "prefill_attn_tc.cu", "sampling.cu", "ops.cu", "attn.cu", "engine.cu", "api.cu", "tp.cu", "stack_ops.cu",
           "stack_mix.cu", "stack_rec.cu", "stack_hyper.cu", "stack_pool.cu", "stack_pool_mma.cu", "engine_stack.cu"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr",
    "-Xcompiler", "-fPIC,-fno-exceptions,-fvisibility=hidden",
    "-Xptxas", "-v",
    *os.environ.get("B200_NVCC_EXTRA", "").split(),   # extra -D… for one-off diagnostic builds (part of the build digest)
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found: the B200 library cannot be built (there is no CPU fallback)")


def _hash(paths, *also: str) -> str:
    h = hashlib.sha256()
    for p in sorted([*paths, ROOT / "include" / "b200_decode.h"]):
        h.update(p.name.encode())
        h.update(p.read_bytes())
    for text in also:
        h.update(text.encode())
    return h.hexdigest()


def _digest() -> str:
    return _hash([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")], " ".join(NVCC_FLAGS))


def _cxx_flags() -> list[str]:
    import torch
    return ["-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]


def _native_digest() -> str:
    """The extension is bound to the torch and the Python that it was compiled against.  Without paths: the built files travel with the tree."""
    import torch
    return _hash([CSRC / "torch_ops.cpp"], torch.__version__, str(torch.version.git_version), sys.version, *_cxx_flags())


def _native_command() -> list[str]:
    """g++ for the torch extension: torch's own headers and libraries.  The library's functions come from the one that _lib.py loads."""
    import sysconfig

    import torch
    home = Path(torch.__file__).parent
    nvcc_home = Path(_nvcc()).resolve().parent.parent
    includes = [home / "include", home / "include/torch/csrc/api/include", nvcc_home / "include", sysconfig.get_paths()["include"]]
    return ["g++", *_cxx_flags(), *[x for i in includes for x in ("-isystem", str(i))], "-I", str(ROOT / "include"), str(CSRC / "torch_ops.cpp"),
            "-o", str(NATIVE_PATH), f"-L{home / 'lib'}", "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]


def build(force: bool = False, verbose: bool = False) -> Path:
    """Both files, each when it or what it is made from has changed since its stamp was written; the library first, which needs no torch."""
    LIB_DIR.mkdir(exist_ok=True)
    OBJ_DIR.mkdir(exist_ok=True)
    for made, digest, stamp, make in ((LIB_PATH, _digest, "build", _build_library), (NATIVE_PATH, _native_digest, "native", _build_native)):
        stamp, now = LIB_DIR / f"{stamp}.stamp", digest()
        if not force and made.exists() and stamp.exists() and stamp.read_text().strip() == now:
            continue
        log = make()
        stamp.with_suffix(".log").write_text(log)
        stamp.write_text(now)
        if verbose:
            print(log)
    return LIB_PATH


def _build_library() -> str:
    nvcc = _nvcc()
    log_lines: list[str] = []

    def compile_one(src: str) -> Path:
        obj = OBJ_DIR / (src[:-3] + ".o")
        cmd = [nvcc, *NVCC_FLAGS, "-I", str(ROOT / "include"), "-c", str(CSRC / src), "-o", str(obj)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        log_lines.append(f"$ {' '.join(cmd)}\n{r.stdout}{r.stderr}")
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(SOURCES))) as ex:
        objs = list(ex.map(compile_one, SOURCES))
    cmd = [nvcc, "-shared", "-o", str(LIB_PATH), *map(str, objs), "-gencode", "arch=compute_100a,code=sm_100a"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    log_lines.append(f"$ {' '.join(cmd)}\n{r.stdout}{r.stderr}")
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    return "\n".join(log_lines)


def _build_native() -> str:
    cmd = _native_command()
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed on torch_ops.cpp:\n{r.stdout}\n{r.stderr}")
    return f"$ {' '.join(cmd)}\n{r.stdout}{r.stderr}"


if __name__ == "__main__":
    p = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(p)
