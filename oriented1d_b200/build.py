"""In-tree build of libo1d.so (sm_100a only) and of its tensor front end.

``python -m oriented1d_b200.build`` compiles every ``csrc/*.cu`` with nvcc (one object per
file, in parallel) and links them into ``oriented1d_b200/libo1d.so``.  nvcc cross-compiles,
so this works on a machine without a GPU.  The library has no dependency on torch or Python;
``csrc/o1d_torch.cpp``, compiled against the installed torch into ``_o1d_torch.so``, has.
"""
from __future__ import annotations

import glob
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libo1d.so")

EXT = os.path.join(HERE, "_o1d_torch.so")
EXT_SRC = os.path.join(CSRC, "o1d_torch.cpp")
OBJ_DIR = os.path.join(HERE, "_obj")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo", "--expt-relaxed-constexpr",
    "-Xcompiler", "-fPIC",
]


def nvcc() -> str:
    exe = shutil.which("nvcc") or os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; libo1d.so cannot be built")
    return exe


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def source_digest() -> str:
    """Hash of everything the library is compiled from (file names and contents)."""
    import hashlib
    h = hashlib.sha256(" ".join(NVCC_FLAGS).encode())
    deps = sorted(d for d in glob.glob(os.path.join(CSRC, "*")) if d != EXT_SRC) + [os.path.join(HERE, "..", "include", "o1d.h")]
    for d in deps:
        h.update(os.path.basename(d).encode())
        with open(d, "rb") as f:
            h.update(f.read())
    return h.hexdigest()


def stale() -> bool:
    """True when libo1d.so is missing or was built from other sources (content hash kept
    beside the library; file times are not used because copies do not preserve them)."""
    if not os.path.exists(LIB) or not os.path.exists(LIB + ".digest"):
        return True
    with open(LIB + ".digest") as f:
        return f.read().strip() != source_digest()


def _file_digest(src: str) -> str:
    """Hash of one source file together with every header it could include."""
    import hashlib
    h = hashlib.sha256(" ".join(NVCC_FLAGS).encode())
    deps = [src] + sorted(glob.glob(os.path.join(CSRC, "*.cuh"))) + sorted(glob.glob(os.path.join(CSRC, "*.h")))
    deps.append(os.path.join(HERE, "..", "include", "o1d.h"))
    for d in deps:
        h.update(os.path.basename(d).encode())
        with open(d, "rb") as f:
            h.update(f.read())
    return h.hexdigest()


def ext_digest() -> str:
    """Hash of what the tensor front end is compiled from, and of the torch it is compiled for."""
    import hashlib
    import torch
    h = hashlib.sha256(f"{torch.__version__} {sys.version_info[:2]} {torch._C._GLIBCXX_USE_CXX11_ABI}".encode())
    for d in (EXT_SRC, os.path.join(HERE, "..", "include", "o1d.h")):
        with open(d, "rb") as f:
            h.update(f.read())
    return h.hexdigest()


def ext_stale() -> bool:
    if not os.path.exists(EXT) or not os.path.exists(EXT + ".digest"):
        return True
    with open(EXT + ".digest") as f:
        return f.read().strip() != ext_digest()


def build_ext(force: bool = False) -> str:
    """Compile csrc/o1d_torch.cpp (host code only) and link it to libo1d.so beside it."""
    if not (force or ext_stale()):
        return EXT
    import sysconfig
    import torch
    from torch.utils import cpp_extension as ce
    inc = ce.include_paths(device_type="cuda") + [sysconfig.get_paths()["include"]]
    libs = ce.library_paths(device_type="cuda")
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_o1d_torch",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *[f"-isystem{i}" for i in inc], EXT_SRC, "-o", EXT,
           *[f"-L{p}" for p in libs], f"-L{HERE}", "-l:libo1d.so", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch",
           "-ltorch_python", "-Wl,-rpath,$ORIGIN"]
    subprocess.run(cmd, check=True)
    with open(EXT + ".digest", "w") as f:
        f.write(ext_digest())
    return EXT


def _compile_one(src: str, force: bool, verbose: bool) -> str:
    obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
    tag = obj + ".digest"
    digest = _file_digest(src)
    if not force and os.path.exists(obj) and os.path.exists(tag):
        with open(tag) as f:
            if f.read().strip() == digest:
                return obj
    cmd = [nvcc(), *NVCC_FLAGS, "-c", src, "-o", obj]
    if verbose:
        cmd.insert(1, "-Xptxas=-v")
        print(" ".join(cmd))
    subprocess.run(cmd, check=True)
    with open(tag, "w") as f:
        f.write(digest)
    return obj


def build(force: bool = False, verbose: bool = False) -> str:
    if not (force or stale()):
        build_ext()
        return LIB
    from concurrent.futures import ThreadPoolExecutor
    os.makedirs(OBJ_DIR, exist_ok=True)
    srcs = sources()
    with ThreadPoolExecutor(max_workers=min(len(srcs), os.cpu_count() or 1)) as pool:
        objs = list(pool.map(lambda s: _compile_one(s, force, verbose), srcs))
    subprocess.run([nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB, *objs], check=True)
    with open(LIB + ".digest", "w") as f:
        f.write(source_digest())
    build_ext(force)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
