"""Builds libb200_fattn.so in-tree with nvcc for sm_100a (cross-compiles without a GPU), and, where torch is installed,
_torch_op.so, the torch-facing call path over its C-ABI, with the host compiler."""
from __future__ import annotations

import hashlib
import importlib.util
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libb200_fattn.so")
TORCH_OP = os.path.join(HERE, "_torch_op.so")
STAMP = LIB + ".srchash"   # hash of the sources and flags the library next to it was built from
SOURCES = ["fattn_api.cu", "fattn_mma.cu", "fattn_tc5.cu", "kv_slab.cu", "relpos_table.cu", "segment_sched.cpp", "slice_batch.cpp"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC,-fvisibility=hidden,-Wall", "--expt-relaxed-constexpr",
]
TORCH_OP_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-Wall"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    return "nvcc"


def sources() -> list[str]:
    return [os.path.join(CSRC, s) for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]


def source_hash() -> str:
    """SHA-256 over every file under csrc/, the public header and the compiler flags."""
    h = hashlib.sha256()
    files = sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC)) + [os.path.join(HERE, "..", "include", "b200_fattn.h")]
    for path in files:
        h.update(os.path.basename(path).encode() + b"\0")
        h.update(open(path, "rb").read())
    h.update(" ".join(NVCC_FLAGS + SOURCES + TORCH_OP_FLAGS).encode())
    return h.hexdigest()


def built_hash() -> str | None:
    """The source hash recorded when the library in the tree was linked, or None."""
    try:
        return open(STAMP).read().strip() if os.path.exists(LIB) else None
    except OSError:
        return None


def have_torch() -> bool:
    """Whether torch can be imported; the C library needs none."""
    return importlib.util.find_spec("torch") is not None


def needs_build() -> bool:
    return built_hash() != source_hash() or (have_torch() and not os.path.exists(TORCH_OP))


def _torch_op_command() -> list[str]:
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(shutil.which(_nvcc()) or _nvcc()))
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    return (["g++", *TORCH_OP_FLAGS, f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
            + [x for d in include for x in ("-isystem", d)] + [os.path.join(CSRC, "torch_op.cpp"), "-o", TORCH_OP]
            + ["-L", HERE, "-l:" + os.path.basename(LIB), "-Wl,-rpath,$ORIGIN", "-L", os.path.join(root, "lib"),
               "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda"])


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB
    if shutil.which(_nvcc()) is None and not os.path.exists(_nvcc()):
        raise RuntimeError(
            f"{LIB} is missing or was built from other sources (recorded {built_hash()}, tree {source_hash()}) "
            "and there is no nvcc to rebuild it with")
    if force or built_hash() != source_hash():
        _build_library(verbose)
    if have_torch():
        subprocess.run(_torch_op_command(), check=True)
    elif os.path.exists(TORCH_OP):
        os.remove(TORCH_OP)   # of other sources
    with open(STAMP, "w") as f:
        f.write(source_hash() + "\n")
    return LIB


def _build_library(verbose: bool) -> None:
    objs = []
    procs = []
    os.makedirs(os.path.join(HERE, "build"), exist_ok=True)
    for src in sources():
        obj = os.path.join(HERE, "build", os.path.basename(src) + ".o")
        cmd = [_nvcc(), *NVCC_FLAGS, "-c", src, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            sys.stderr.write(out)
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    link = [_nvcc(), "-shared", "-o", LIB, *objs, "-lcudart", "-Xcompiler", "-fPIC"]
    subprocess.run(link, check=True)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
