"""In-tree nvcc build of the sm_100a kernel library.

`build()` compiles every `.cu` file under `csrc/` (one object each, in parallel) and links them into
`nano_vllm_jax_b200/libnvj_b200.so` (next to this file, so the built library
travels with a snapshot of the source tree) and is a no-op when the library is
newer than every source.  Beside it, `build_host()` compiles `csrc/host/host_ops.cpp`
(the host side of the hot calls, against torch's C++ headers) into the Python
extension module `_nvj_host.<tag>.so`; `build()` does both.  The pattern follows the reference's build-on-import of
its own CUDA FFI library (nanovllm_jax/kernels/cuda_fp32_ffi.py:121-178) with the
architecture fixed to sm_100a.
"""

from __future__ import annotations

import os
import re
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
INCLUDE = PKG_DIR.parent / "include"
LIB_PATH = PKG_DIR / "libnvj_b200.so"
HOST_SRC = CSRC / "host" / "host_ops.cpp"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]
OBJ_DIR = PKG_DIR / "build"


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _headers() -> list[Path]:
    return list(CSRC.glob("*.cuh")) + list(INCLUDE.glob("*.h"))


def _stale() -> bool:
    if not LIB_PATH.exists():
        return True
    built = LIB_PATH.stat().st_mtime
    return any(p.stat().st_mtime > built for p in sources() + _headers())


def nvcc_path() -> str | None:
    return shutil.which("nvcc") or (
        "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None
    )


def host_path() -> Path:
    """Where the host extension of this Python and this torch lies.  Its C++ interface to both is theirs to change with any
    version, so the file carries the two in its name: after a change of either the old one is not found and a new one is built."""
    import torch
    tag = re.sub(r"[^A-Za-z0-9]+", "_", f"{sys.implementation.cache_tag} torch {torch.__version__}")
    return PKG_DIR / f"_nvj_host.{tag}.so"


def build_host(force: bool = False) -> Path:
    """Compile the host extension module if needed and return its path."""
    target = host_path()
    newest = max(p.stat().st_mtime for p in (HOST_SRC, INCLUDE / "nvj_b200.h"))
    if not force and target.exists() and target.stat().st_mtime > newest:
        return target
    import torch
    torch_dir = Path(torch.__file__).parent
    nvcc = nvcc_path()
    cuda_include = Path(nvcc).resolve().parents[1] / "include" if nvcc else Path("/usr/local/cuda/include")
    part = target.with_suffix(f".{os.getpid()}.part")  # moved into place whole: another process may be loading the old one
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           "-I", str(torch_dir / "include"), "-I", str(torch_dir / "include" / "torch" / "csrc" / "api" / "include"),
           "-I", str(cuda_include), "-I", sysconfig.get_paths()["include"], "-o", str(part), str(HOST_SRC),
           "-L", str(torch_dir / "lib"), "-L", str(cuda_include.parent / "lib64"), "-lcudart", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python"]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError("g++ failed on host_ops.cpp:\n" + proc.stdout + proc.stderr)
    part.replace(target)
    return target


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile the library and the host module if needed and return the library's path.

    Every `.cu` file becomes one object under `build/` (compiled in parallel, recompiled when the
    file or any header is newer than its object); the objects are then linked into the library.
    """
    build_host(force)
    if not force and not _stale():
        return LIB_PATH
    nvcc = nvcc_path()
    if nvcc is None:
        raise RuntimeError("nvcc not found: cannot build libnvj_b200.so")
    OBJ_DIR.mkdir(exist_ok=True)
    newest_header = max((p.stat().st_mtime for p in _headers()), default=0.0)

    def compile_one(src: Path):
        obj = OBJ_DIR / (src.stem + ".o")
        if not force and obj.exists() and obj.stat().st_mtime > max(src.stat().st_mtime, newest_header):
            return obj, ""
        cmd = [nvcc, *NVCC_FLAGS, "-I", str(INCLUDE), "-c", "-o", str(obj), str(src)]
        if verbose:
            cmd += ["-Xptxas", "-v"]
        proc = subprocess.run(cmd, capture_output=True, text=True)
        if proc.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src.name}:\n" + proc.stdout + proc.stderr)
        return obj, proc.stderr

    from concurrent.futures import ThreadPoolExecutor
    with ThreadPoolExecutor(max_workers=max(1, min(8, os.cpu_count() or 1))) as pool:
        results = list(pool.map(compile_one, sources()))
    if verbose:
        for obj, log in results:
            if log:
                print(f"---- {obj.name}\n{log}")
    link = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler", "-fPIC", "-o", str(LIB_PATH)]
    link += [str(obj) for obj, _ in results]
    proc = subprocess.run(link, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError("link failed:\n" + proc.stdout + proc.stderr)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
