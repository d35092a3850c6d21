"""In-tree build of liblocal_cuda.so for sm_100a with nvcc.

The library is rebuilt when the hash of its sources (csrc/*.cu, csrc/*.h,
include/local_cuda.h) differs from the hash recorded beside the built file,
so a stale binary is never loaded.  Several processes may find one stale at once (the
ranks of a job): one builds while the others wait, and a finished file takes its name
by a rename, so nobody loads half of one.  Each .cu is compiled to an object file in
parallel, then linked.  The CPython extension of fastcall.py (the argument
conversion of the Python mirror) is generated from the header and built beside it;
a machine that cannot build it calls through ctypes (slowcall.py).
"""
from __future__ import annotations

import fcntl
import hashlib
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from contextlib import contextmanager
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


@contextmanager
def _building():
    """One process at a time builds in this tree."""
    OBJ.mkdir(exist_ok=True)
    with open(OBJ / "lock", "w") as f:
        fcntl.flock(f, fcntl.LOCK_EX)
        yield


def _install(new: Path, final: Path, hash_file: Path, digest: str) -> None:
    """The finished file takes its name, and only then does the recorded hash say that it is current."""
    os.replace(new, final)
    new_hash = new.with_suffix(".hash")
    new_hash.write_text(digest + "\n")
    os.replace(new_hash, hash_file)


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


def fastcall_is_current() -> bool:
    return FAST.exists() and FAST_HASH.exists() and FAST_HASH.read_text().strip() == fastcall_hash()


def build_fastcall(force: bool = False) -> Path:
    """Generate and compile the CPython extension for the running interpreter."""
    if not force and fastcall_is_current():
        return FAST
    cc = shutil.which("gcc") or shutil.which("cc")
    if cc is None:
        raise RuntimeError("no C compiler: cannot build the _fastcall extension")
    with _building():
        if not force and fastcall_is_current():   # (built while this process waited)
            return FAST
        digest = fastcall_hash()
        spec = importlib.util.spec_from_file_location("local_ai_b200_fastcall_gen", PKG / "fastcall.py")
        gen = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(gen)
        src, new = OBJ / "_fastcall.c", OBJ / "_fastcall.new"
        src.write_text(gen.generate(ROOT / "include" / "local_cuda.h"))
        cmd = [cc, "-O2", "-std=gnu11", "-shared", "-fPIC", "-fvisibility=hidden", f"-I{sysconfig.get_paths()['include']}",
               f"-I{ROOT / 'include'}", str(src), "-o", str(new)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(f"$ {' '.join(cmd)}\n{r.stdout}{r.stderr}")
            raise RuntimeError("gcc failed on the _fastcall extension")
        _install(new, FAST, FAST_HASH, digest)
    return FAST


def build_library(force: bool = False, verbose: bool = False, extra_flags: list[str] | None = None) -> Path:
    """Compile every CUDA source for sm_100a and link the shared library."""
    if not force and is_current():
        return LIB
    nvcc = find_nvcc()
    if nvcc is None:
        raise RuntimeError("nvcc not found: cannot build liblocal_cuda.so (there is no CPU fallback)")
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

    with _building():
        if not force and is_current():   # (built while this process waited)
            return LIB
        digest = source_hash()
        with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
            objs = list(ex.map(compile_one, sources()))
        new = OBJ / "liblocal_cuda.new"
        cmd = [nvcc, "-shared", "-o", str(new), *map(str, objs), "-gencode", "arch=compute_100a,code=sm_100a", "-ldl"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link of liblocal_cuda.so failed")
        _install(new, LIB, HASH, digest)
    return LIB


if __name__ == "__main__":
    print(build_fastcall(force="--force" in sys.argv))
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
