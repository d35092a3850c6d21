"""In-tree build of liblocal_cuda.so for sm_100a with nvcc.

The library is rebuilt when the hash of its sources (csrc/*.cu, csrc/*.h,
include/local_cuda.h) differs from the hash recorded beside the built file,
so a stale binary is never loaded.  Each .cu is compiled to an object file in
parallel, then linked.  The CPython extension of fastcall.py (the argument
conversion of the Python mirror) is generated from the header and built beside it;
a machine that cannot build it calls through ctypes (slowcall.py).
"""
from __future__ import annotations

import hashlib
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
ROOT = PKG.parent
CSRC = PKG / "csrc"
OBJ = PKG / "build"
LIB = PKG / "liblocal_cuda.so"
HASH = PKG / "liblocal_cuda.build_hash"
FAST = PKG / ("_fastcall" + sysconfig.get_config_var("EXT_SUFFIX"))
FAST_HASH = PKG / "_fastcall.build_hash"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC,-fvisibility=hidden,-ffp-contract=off",
]


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def source_hash() -> str:
    h = hashlib.sha256()
    files = sources() + sorted(CSRC.glob("*.h")) + sorted(CSRC.glob("*.cuh")) + [ROOT / "include" / "local_cuda.h"]
    for f in files:
        h.update(f.name.encode())
        h.update(f.read_bytes())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()


def is_current() -> bool:
    return LIB.exists() and HASH.exists() and HASH.read_text().strip() == source_hash()


def find_nvcc() -> str | None:
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    return None


def fastcall_hash() -> str:
    h = hashlib.sha256(FAST.name.encode())
    for f in (PKG / "fastcall.py", ROOT / "include" / "local_cuda.h"):
        h.update(f.read_bytes())
    return h.hexdigest()


def build_fastcall(force: bool = False) -> Path:
    """Generate and compile the CPython extension for the running interpreter."""
    if not force and FAST.exists() and FAST_HASH.exists() and FAST_HASH.read_text().strip() == fastcall_hash():
        return FAST
    spec = importlib.util.spec_from_file_location("local_ai_b200_fastcall_gen", PKG / "fastcall.py")
    gen = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(gen)
    OBJ.mkdir(exist_ok=True)
    src = OBJ / "_fastcall.c"
    src.write_text(gen.generate(ROOT / "include" / "local_cuda.h"))
    cc = shutil.which("gcc") or shutil.which("cc")
    if cc is None:
        raise RuntimeError("no C compiler: cannot build the _fastcall extension")
    cmd = [cc, "-O2", "-std=gnu11", "-shared", "-fPIC", "-fvisibility=hidden", f"-I{sysconfig.get_paths()['include']}",
           f"-I{ROOT / 'include'}", str(src), "-o", str(FAST)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(f"$ {' '.join(cmd)}\n{r.stdout}{r.stderr}")
        raise RuntimeError("gcc failed on the _fastcall extension")
    FAST_HASH.write_text(fastcall_hash() + "\n")
    return FAST


def build_library(force: bool = False, verbose: bool = False, extra_flags: list[str] | None = None) -> Path:
    """Compile every CUDA source for sm_100a and link the shared library."""
    if not force and is_current():
        return LIB
    nvcc = find_nvcc()
    if nvcc is None:
        raise RuntimeError("nvcc not found: cannot build liblocal_cuda.so (there is no CPU fallback)")
    OBJ.mkdir(exist_ok=True)
    flags = NVCC_FLAGS + (extra_flags or [])

    def compile_one(src: Path) -> Path:
        obj = OBJ / (src.stem + ".o")
        cmd = [nvcc, *flags, "-c", str(src), "-o", str(obj)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode != 0:
            sys.stderr.write(f"$ {' '.join(cmd)}\n{r.stdout}{r.stderr}")
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src.name}")
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        objs = list(ex.map(compile_one, sources()))
    cmd = [nvcc, "-shared", "-o", str(LIB), *map(str, objs), "-gencode", "arch=compute_100a,code=sm_100a", "-ldl"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("link of liblocal_cuda.so failed")
    HASH.write_text(source_hash() + "\n")
    return LIB


if __name__ == "__main__":
    print(build_fastcall(force="--force" in sys.argv))
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
