"""Builds libftq_b200.so (the CUDA kernels + C ABI) in-tree with nvcc for sm_100a.

    python -m fused_turboquant_b200.build [--force] [--verbose]

The per-head_dim translation units compile in parallel.  No fast-math flag is
ever passed: the encode kernel's bit-exactness depends on IEEE arithmetic.
"""
from __future__ import annotations

import argparse
import concurrent.futures as cf
import os
import re
import shutil
import subprocess
import sys

from ._lib import native_tag

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
OBJ_DIR = os.path.join(PKG_DIR, "build")
LIB_PATH = os.path.join(PKG_DIR, "libftq_b200.so")
# A second library for ONE test (tests/test_gpu_wait_expiry.py): the same objects, except that the
# head_dim-128 decode, chunk attention and slot-format decode units are compiled with FTQ_TEST_WAIT_EXPIRY (one page copy of
# one warp is never issued, one tile of one warp never reported, and the poll limits are small), so that
# a bounded wait runs out and the give-up path (NaN rows, status word, the context stays usable)
# executes.  Never loaded by the package.
TEST_LIB_PATH = os.path.join(PKG_DIR, "libftq_b200_waittest.so")
# The tensor-level host path (csrc/ftq_torch.cpp): a CPython module compiled with the host compiler
# against torch's headers; it gets the C ABI's addresses at import and links nothing of ours.
NATIVE_PATH = os.path.join(PKG_DIR, "_native.so")
TEST_UNITS = [(src, f"{tag}_waittest", [*part, "-DFTQ_D=128", "-DFTQ_ONLY_BITS=4", "-DFTQ_TEST_WAIT_EXPIRY"])
              for src, tag, part in (("ftq_attn_inst.cu", "attn_d128", ()), ("ftq_attn_chunk_inst.cu", "attn_chunk_d128", ()),
                                     ("ftq_tq_v1_inst.cu", "tq_v1_flow_d128", ("-DFTQ_TQ_PART=2",)))]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
]

# (source, object suffix, extra defines)
# (the slowest units first: the pool then finishes them while the short ones fill the gaps)
UNITS = []
for _d in (256, 128, 64):
    UNITS.append(("ftq_tq_v1_inst.cu", f"tq_v1_store_d{_d}", [f"-DFTQ_D={_d}", "-DFTQ_TQ_PART=0"]))
    UNITS.append(("ftq_tq_v1_inst.cu", f"tq_v1_decode_d{_d}", [f"-DFTQ_D={_d}", "-DFTQ_TQ_PART=1"]))
    if _d != 256:   # (not for that size)
        UNITS.append(("ftq_tq_v1_inst.cu", f"tq_v1_flow_d{_d}", [f"-DFTQ_D={_d}", "-DFTQ_TQ_PART=2"]))
for _d in (256, 128, 64):
    UNITS.append(("ftq_attn_inst.cu", f"attn_d{_d}", [f"-DFTQ_D={_d}"]))
    UNITS.append(("ftq_attn_chunk_inst.cu", f"attn_chunk_d{_d}", [f"-DFTQ_D={_d}"]))
    UNITS.append(("ftq_encode_inst.cu", f"encode_d{_d}", [f"-DFTQ_D={_d}"]))
UNITS.append(("ftq_api.cu", "api", []))


def _nvcc() -> str:
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: cannot build libftq_b200.so")


def _run(cmd: list, out: str, what: str) -> str:
    """Run a compiler or linker whose output file is `out`; the file appears complete or not at all (another
    process may have the one before loaded)."""
    part = f"{out}.{os.getpid()}.part"
    r = subprocess.run([*cmd, "-o", part], capture_output=True, text=True)
    if r.returncode != 0:
        if os.path.exists(part):
            os.remove(part)
        raise RuntimeError(f"{what} failed:\n{r.stdout}\n{r.stderr}")
    os.replace(part, out)
    return r.stderr


def _build_native() -> None:
    import sysconfig

    import torch
    src = os.path.join(CSRC, "ftq_torch.cpp")
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    _run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared",
          f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
          f'-DFTQ_BUILT_FOR="{native_tag()}"',
          "-I" + sysconfig.get_paths()["include"], "-I" + os.path.join(root, "include"),
          "-I" + os.path.join(root, "include", "torch", "csrc", "api", "include"),
          "-I" + os.path.join(cuda, "include"), src,
          "-L" + os.path.join(root, "lib"), "-ltorch", "-ltorch_cpu", "-ltorch_python", "-lc10",
          "-lc10_cuda"], NATIVE_PATH, f"g++ for {src}")


def _native_stale() -> bool:
    """Older than its own sources, or compiled against another torch or Python."""
    if _older(NATIVE_PATH, _deps(os.path.join(CSRC, "ftq_torch.cpp"))):
        return True
    with open(NATIVE_PATH, "rb") as f:
        return native_tag().encode() not in f.read()


_INCLUDE = re.compile(r'^\s*#\s*include\s+"([^"]+)"', re.M)


def _deps(path: str, seen=None) -> set:
    """The file and every project header it includes, transitively."""
    seen = set() if seen is None else seen
    path = os.path.normpath(path)
    if path in seen or not os.path.exists(path):
        return seen
    seen.add(path)
    with open(path) as f:
        text = f.read()
    for inc in _INCLUDE.findall(text):
        _deps(os.path.join(os.path.dirname(path), inc), seen)
    return seen


def _older(out: str, deps) -> bool:
    """`out` does not exist or is older than one of `deps`."""
    if not os.path.exists(out):
        return True
    t = os.path.getmtime(out)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile and link what is missing or older than its own sources: the library, the wait-expiry test
    library, the host path."""
    cuda_deps = set().union(*(_deps(os.path.join(CSRC, u[0])) for u in UNITS + TEST_UNITS))
    cuda_stale = force or any(_older(l, cuda_deps) for l in (LIB_PATH, TEST_LIB_PATH))
    if force or _native_stale():
        _build_native()
    if not cuda_stale:
        return LIB_PATH
    nvcc = _nvcc()
    os.makedirs(OBJ_DIR, exist_ok=True)
    extra = ["-Xptxas", "-v"] if verbose else []

    def compile_one(unit):
        src, tag, defs = unit
        obj = os.path.join(OBJ_DIR, f"{tag}.o")
        if not force and not verbose and not _older(obj, _deps(os.path.join(CSRC, src))):
            return obj      # up to date: only units whose sources changed are recompiled
        err = _run([nvcc, *NVCC_FLAGS, *extra, *defs, "-c", os.path.join(CSRC, src)], obj, f"nvcc for {src} {defs}")
        if verbose:
            sys.stderr.write(err)
        return obj

    with cf.ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        objs = list(ex.map(compile_one, UNITS + TEST_UNITS))
    test_objs = {o.replace("_waittest.o", ".o"): o for o in objs[len(UNITS):]}
    objs = objs[:len(UNITS)]
    for lib, members in ((LIB_PATH, objs), (TEST_LIB_PATH, [test_objs.get(o, o) for o in objs])):
        _run([nvcc, "-shared", *members, "-lcudart"], lib, f"link of {lib}")
    return LIB_PATH


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true", help="print ptxas register/spill report")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))
