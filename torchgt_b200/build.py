"""In-tree build of the CUDA library and of the host module: ``python -m torchgt_b200.build``.

Compiles every ``csrc/*.cu`` for sm_100a with nvcc (one process per file, in parallel) and links
``torchgt_b200/lib/libtorchgt_b200.so``, the C-ABI library the Python package loads through ``ctypes``; then
every ``csrc/*.cpp`` with the host compiler against PyTorch into ``torchgt_b200/lib/_native.so``, the module that
holds the autograd nodes and issues the launches.  nvcc cross-compiles without a GPU, so this runs on a CPU-only
machine.
"""
from __future__ import annotations

import concurrent.futures
import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
LIB_DIR = PKG_DIR / "lib"
LIB_PATH = LIB_DIR / "libtorchgt_b200.so"
NATIVE_PATH = LIB_DIR / "_native.so"
INCLUDE = PKG_DIR.parent / "include"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-Xcompiler", "-fvisibility=hidden",
    "--expt-relaxed-constexpr",
    "--extended-lambda",
]

CXX_FLAGS = ["-O3", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-Wall", "-Wno-unused-function"]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: the CUDA toolkit is required to build torchgt_b200")
    return exe


def _sources(suffix: str = "cu") -> list[Path]:
    return sorted(CSRC.glob(f"*.{suffix}"))


def _fingerprint(of=("cu", "cuh")) -> str:
    h = hashlib.sha256()
    for p in sorted([f for suffix in of for f in CSRC.glob(f"*.{suffix}")] + list(INCLUDE.glob("*.h"))):
        h.update(p.name.encode())
        h.update(p.read_bytes())
    h.update(" ".join(NVCC_FLAGS if "cu" in of else CXX_FLAGS + [_torch_version()]).encode())
    return h.hexdigest()


def _torch_version() -> str:
    import torch
    return torch.__version__


def _compile_one(nvcc: str, src: Path, obj: Path, verbose: bool) -> str:
    cmd = [nvcc, *NVCC_FLAGS, "-I", str(INCLUDE), "-c", str(src), "-o", str(obj)]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed on {src.name}:\n{r.stdout}\n{r.stderr}")
    return r.stderr


def _torch_dir() -> Path:
    import torch
    return Path(torch.__file__).resolve().parent


def _cuda_home(nvcc: str) -> Path:
    return Path(os.path.realpath(nvcc)).parent.parent


def build_native(force: bool = False) -> Path:
    """Build the host module if its sources (or PyTorch's version) changed; returns its path."""
    LIB_DIR.mkdir(exist_ok=True)
    stamp = LIB_DIR / "native.stamp"
    fp = _fingerprint(("cpp", "h"))
    if not force and NATIVE_PATH.exists() and stamp.exists() and stamp.read_text() == fp:
        return NATIVE_PATH
    torch_dir, cuda = _torch_dir(), _cuda_home(_nvcc())
    cxx = shutil.which("g++") or "c++"
    obj_dir = LIB_DIR / "obj"
    obj_dir.mkdir(exist_ok=True)
    include = [f"-I{torch_dir / 'include'}", f"-I{torch_dir / 'include/torch/csrc/api/include'}", f"-I{cuda / 'include'}",
               f"-I{sysconfig.get_paths()['include']}"]
    srcs = _sources("cpp")
    objs = [obj_dir / (s.stem + ".host.o") for s in srcs]

    def run(cmd, what):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"{what} failed:\n{r.stdout}\n{r.stderr}")

    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        list(ex.map(lambda so: run([cxx, *CXX_FLAGS, *include, "-c", str(so[0]), "-o", str(so[1])], so[0].name),
                    zip(srcs, objs)))
    run([cxx, "-shared", "-o", str(NATIVE_PATH), *map(str, objs), f"-L{LIB_DIR}", "-l:" + LIB_PATH.name,
         f"-L{torch_dir / 'lib'}", "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10",
         f"-L{cuda / 'lib64'}", "-lcudart", "-Wl,-rpath,$ORIGIN", f"-Wl,-rpath,{torch_dir / 'lib'}"], "link of " + NATIVE_PATH.name)
    stamp.write_text(fp)
    return NATIVE_PATH


def build(force: bool = False, verbose: bool = False) -> Path:
    """Build the shared library and the host module if their sources changed; returns the library's path."""
    path = build_library(force, verbose)
    build_native(force)
    return path


def build_library(force: bool = False, verbose: bool = False) -> Path:
    LIB_DIR.mkdir(exist_ok=True)
    stamp = LIB_DIR / "build.stamp"
    fp = _fingerprint()
    if not force and LIB_PATH.exists() and stamp.exists() and stamp.read_text() == fp:
        return LIB_PATH
    nvcc = _nvcc()
    obj_dir = LIB_DIR / "obj"
    obj_dir.mkdir(exist_ok=True)
    srcs = _sources()
    objs = [obj_dir / (s.stem + ".o") for s in srcs]
    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        logs = list(ex.map(lambda so: _compile_one(nvcc, so[0], so[1], verbose), zip(srcs, objs)))
    if verbose:
        for s, log in zip(srcs, logs):
            print(f"==== {s.name}\n{log}")
    cmd = [nvcc, "-shared", "-o", str(LIB_PATH), *map(str, objs),
           "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "static"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    stamp.write_text(fp)
    return LIB_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
