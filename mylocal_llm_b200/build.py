"""In-tree build of ``libb200q.so`` with nvcc for sm_100a.

``python -m mylocal_llm_b200.build`` compiles every ``.cu`` file under ``csrc/`` (in parallel,
one object per file) and links them into ``mylocal_llm_b200/libb200q.so``. The shared object is
kept in the source tree, next to the package, so that it travels with a snapshot of the tree;
it is rebuilt only when a source or header is newer.
"""

import os
import re
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
INCLUDE = PKG.parent / "include"
LIB = PKG / "libb200q.so"
OBJ_DIR = CSRC / "build"
HOST_SRC = CSRC / "host" / "host_ops.cpp"


def _host_lib():
    """The host extension is compiled against one torch: its version is part of the name, so that another torch finds none
    and does not load what it cannot bind."""
    from importlib import metadata
    try:
        tag = re.sub(r"[^0-9A-Za-z.]", "_", metadata.version("torch"))
    except metadata.PackageNotFoundError:
        tag = "none"
    return PKG / f"_b200q_host.{tag}.so"


HOST_LIB = _host_lib()

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xptxas=-v",
]


def _nvcc():
    path = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(path).exists():
        raise RuntimeError("nvcc not found; the b200q kernels cannot be built")
    return path


def _sources():
    return sorted(CSRC.glob("*.cu"))


def _headers():
    return sorted(CSRC.glob("*.cuh")) + sorted(INCLUDE.glob("*.h"))


def needs_build():
    if not LIB.exists():
        return True
    stamp = LIB.stat().st_mtime
    return any(p.stat().st_mtime > stamp for p in _sources() + _headers())


def needs_host_build():
    """The extension module with the native host path: its source or the C ABI header is newer."""
    if not HOST_LIB.exists():
        return True
    stamp = HOST_LIB.stat().st_mtime
    return any(p.stat().st_mtime > stamp for p in [HOST_SRC, *INCLUDE.glob("*.h")])


def build_host(force=False):
    """Compile the host extension (C++ only, against the installed torch); returns its path."""
    if not force and not needs_host_build():
        return HOST_LIB
    import sysconfig
    import torch
    from torch.utils import cpp_extension
    cuda = Path(_nvcc()).resolve().parent.parent / "include"
    tmp = HOST_LIB.with_suffix(f".{os.getpid()}.tmp.so")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-w",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-I", str(INCLUDE),
           *[f"-isystem{path}" for path in [*cpp_extension.include_paths(), sysconfig.get_paths()["include"], str(cuda)]],
           str(HOST_SRC), "-o", str(tmp), *[f"-L{path}" for path in cpp_extension.library_paths()],
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode:
        raise RuntimeError(f"host extension build failed:\n{proc.stderr[-4000:]}")
    os.replace(tmp, HOST_LIB)
    return HOST_LIB


def build(force=False, verbose=False):
    """Compile and link the in-tree ``libb200q.so`` (and the host extension); returns its path."""
    if not force and not needs_build():
        build_host(force)
        return LIB
    nvcc = _nvcc()
    OBJ_DIR.mkdir(parents=True, exist_ok=True)
    header_stamp = max(p.stat().st_mtime for p in _headers())

    def compile_one(src):
        obj = OBJ_DIR / (src.stem + ".o")
        if (not force and obj.exists() and obj.stat().st_mtime >= src.stat().st_mtime
                and obj.stat().st_mtime >= header_stamp):
            return obj, ""
        cmd = [nvcc, *NVCC_FLAGS, "-I", str(INCLUDE), "-c", str(src), "-o", str(obj)]
        proc = subprocess.run(cmd, capture_output=True, text=True)
        if proc.returncode:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{proc.stderr[-4000:]}")
        return obj, proc.stderr

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        host = pool.submit(build_host, force)
        results = list(pool.map(compile_one, _sources()))
        host.result()
    if verbose:
        for obj, log in results:
            if log:
                sys.stderr.write(f"--- {obj.name}\n{log}\n")
    tmp = LIB.with_suffix(f".{os.getpid()}.tmp.so")
    cmd = [nvcc, "-shared", "-o", str(tmp), *[str(o) for o, _ in results]]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode:
        raise RuntimeError(f"link failed:\n{proc.stderr[-4000:]}")
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
