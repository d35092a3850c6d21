"""Building and loading: the package without a C compiler, and several processes that find a stale build at once."""
import os
import shutil
import subprocess
import sys
import time
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture
def tree(tmp_path, la):
    """A copy of the package with its built library and without the built extension."""
    t = tmp_path / "tree"
    shutil.copytree(ROOT / "local-ai_b200", t / "local-ai_b200", ignore=shutil.ignore_patterns("_fastcall.*", "build", "__pycache__", "liblocal_cuda.so"))
    shutil.copytree(ROOT / "include", t / "include")
    shutil.copy(ROOT / "__graft_entry__.py", t)
    shutil.copy(ROOT / "local-ai_b200" / "liblocal_cuda.so", t / "local-ai_b200")
    return t


def python(tree, code, path):
    return subprocess.Popen([sys.executable, "-c", code], cwd=tree, env=dict(os.environ, PATH=str(path)), stdout=subprocess.PIPE,
                            stderr=subprocess.PIPE, text=True)


SURFACE = """
import __graft_entry__ as g
la = g.load_package()
f = la.kernels._fast
print(type(f).__name__, la.tq_code_bytes(256, 2), la.Kernels.flash_split_count(None, 300))
b = la.CommandBatch.__new__(la.CommandBatch)
b._h = 4096
p = la.PendingCommandBuffer()
assert b._h == 4096 and f.take(b) == 4096 and b._h is None and p._h is None
for call in (lambda: p.wait(), lambda: la.Kernels.gelu_mul_into(None, p, None, None, None, 4), lambda: f.begin(b, None),
             lambda: la.Kernels.matvec_q4_0_group_into(None, b, [None] * 2, 2, None, [p, p], 32, 32), lambda: f.commit(b, p)):
    try:
        call()
        print("accepted")
    except la.Error as e:
        print(e.kind)
for call in (lambda: la.Kernels.gelu_mul_into(None), lambda: la.Kernels.gelu_mul_into(None, "x", None, None, None, 4),
             lambda: la.Kernels.gelu_mul_into(None, p, None, None, None, 4.5)):
    try:
        call()
        print("accepted")
    except TypeError:
        print("TypeError")
"""


def with_and_without_a_compiler(tree, tmp_path, code):
    """What the code prints with nothing to build the extension with, and with it: {"slow": ..., "fast": ...}."""
    nothing = tmp_path / "empty"
    nothing.mkdir()
    out = {}
    for name, path in (("slow", nothing), ("fast", os.environ["PATH"])):
        p = python(tree, code, path)
        stdout, stderr = p.communicate(timeout=300)
        assert p.returncode == 0, stderr[-2000:]
        assert ("calls go through ctypes" in stderr) == (name == "slow")
        out[name] = stdout
    return out


def test_package_without_a_c_compiler(tree, tmp_path):
    """With a built library and nothing to build the extension with, the same calls run through ctypes."""
    out = with_and_without_a_compiler(tree, tmp_path, SURFACE)
    assert out["slow"].split()[0] == "Calls" and out["fast"].split()[0] == "module"
    assert out["slow"].split()[1:] == out["fast"].split()[1:] == ["64", "16"] + ["InvalidArgument"] * 5 + ["TypeError"] * 3


ON_THE_GPU = """
import hashlib
import numpy as np
import __graft_entry__ as g
la = g.load_package()
ctx = la.CudaContext.new(0)
k = la.Kernels.new(ctx)
w, x = la.CudaBuffer.from_slice(ctx, la.synth.q4_0_weights(96, 512, 1)), la.CudaBuffer.from_slice(ctx, la.synth.normal_f16((512,), 2))
outs = [la.CudaBuffer.empty(ctx, 96 * 2) for _ in range(3)]
b = la.CommandBatch.new(ctx)
k.matvec_q4_0_into(b, w, x, outs[0], np.int64(96), 512)
k.matvec_q4_0_group_into(b, [w, w], 2, x, outs[1:], 96, 512)
b.commit_async().wait()
b = la.CommandBatch.capture(ctx)
k.scale_in_place_gpu_into(b, outs[0], 2, 96)
graph = b.end_capture()
graph.launch()
ctx.synchronize()
print(*[hashlib.sha256(o.as_slice(np.uint8)).hexdigest() for o in outs])
"""


@pytest.mark.gpu
def test_calls_through_ctypes_do_the_same_on_the_gpu(tree, tmp_path):
    out = with_and_without_a_compiler(tree, tmp_path, ON_THE_GPU)
    assert out["slow"] == out["fast"] and len(out["slow"].split()) == 3


# a compiler that logs its links, leaves half a file under the output's name for a while, and then does its work
SLOW_COMPILER = """#!/bin/sh
out=; prev=
for a in "$@"; do [ "$prev" = -o ] && out=$a; prev=$a; done
case " $* " in *" -c "*) : > "$out"; exit 0;; esac
echo link >> {log}
printf half > "$out"
sleep 0.7
{work}
"""
BUILD = """
import importlib.util, sys
spec = importlib.util.spec_from_file_location("b", "local-ai_b200/build.py")
b = importlib.util.module_from_spec(spec)
spec.loader.exec_module(b)
print(b.{call}())
"""


@pytest.mark.parametrize("compiler,call,product,work", [
    ("gcc", "build_fastcall", "_fastcall.*.so", '{real} "$@"'), ("nvcc", "build_library", "liblocal_cuda.so", 'printf "whole library" > "$out"')])
def test_processes_that_find_a_stale_build_build_it_once(tree, tmp_path, compiler, call, product, work):
    bin_dir, log = tmp_path / "bin", tmp_path / "log"
    bin_dir.mkdir()
    script = bin_dir / compiler
    script.write_text(SLOW_COMPILER.format(log=log, work=work.format(real=shutil.which(compiler) or "")))
    script.chmod(0o755)
    with open(tree / "include" / "local_cuda.h", "a") as f:
        f.write("/* newer than what is built */\n")
    before = {p: p.read_bytes() for p in (tree / "local-ai_b200").glob(product)}
    ranks = [python(tree, BUILD.format(call=call), f"{bin_dir}:{os.environ['PATH']}") for _ in range(4)]
    seen = set()
    while any(r.poll() is None for r in ranks):
        for p in (tree / "local-ai_b200").glob(product):
            seen.add(p.read_bytes()[:64])
        time.sleep(0.01)
    for r in ranks:
        stdout, stderr = r.communicate()
        assert r.returncode == 0, stderr[-2000:]
    (final,) = (tree / "local-ai_b200").glob(product)
    assert log.read_text() == "link\n"                      # one process built, the others waited
    assert seen <= {final.read_bytes()[:64], *(b[:64] for b in before.values())}   # and nobody could have loaded half a file
    again = python(tree, BUILD.format(call=call), f"{bin_dir}:{os.environ['PATH']}")
    assert again.communicate()[0].strip() and log.read_text() == "link\n"
