"""In-tree build of the C-ABI CUDA library (sm_100a only) and of the native host side of eager calls.

``python -m sparser_faster_llms_b200.build`` compiles every ``csrc/*.cu`` into
``sparser_faster_llms_b200/libb200_sparse_ffn.so`` with plain nvcc: no torch
headers, no pybind, static cudart, so the result is a stable C ABI that loads
with ``ctypes`` on a machine without a GPU driver.

``csrc_host/host_call.cpp`` becomes the extension module ``_host_call`` with the host compiler (Python and torch
headers, no CUDA code).  It reads torch's tensors in place, so its file name carries the torch version, the C++
ABI and Python's own tag, and only the file of the running pair is loaded.  It is optional: where torch, a
compiler or the headers are missing the build warns, and eager calls take their Python path.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
import warnings
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
LIB_NAME = "libb200_sparse_ffn.so"
LIB_PATH = PKG_DIR / LIB_NAME
HOST_SOURCE = PKG_DIR / "csrc_host" / "host_call.cpp"
GENCODE = "arch=compute_100a,code=sm_100a"


def find_nvcc() -> str:
    nvcc = shutil.which("nvcc")
    if nvcc is None:
        cand = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "bin" / "nvcc"
        if cand.exists():
            nvcc = str(cand)
    if nvcc is None:
        raise RuntimeError("nvcc not found: cannot build the sm_100a kernels")
    return nvcc


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def host_path() -> Path:
    """The extension module of the running Python and torch."""
    import torch

    return PKG_DIR / (f"_host_call.torch-{torch.__version__}-abi{int(torch._C._GLIBCXX_USE_CXX11_ABI)}"
                      f"{sysconfig.get_config_var('EXT_SUFFIX')}")


def start_host_build(force: bool = False) -> tuple[Path, subprocess.Popen] | None:
    """Starts the compiler on the extension module if it is missing or older than its source; None if there
    is nothing to do or nothing to do it with."""
    try:
        import torch
    except ImportError:
        warnings.warn("no torch: the native host side of eager calls is not built")
        return None
    path = host_path()
    if not force and path.exists() and HOST_SOURCE.stat().st_mtime <= path.stat().st_mtime:
        return None
    root = Path(torch.__file__).parent
    tmp = path.with_name(path.name + ".tmp")
    try:
        cuda = Path(find_nvcc()).resolve().parent.parent
        include = [sysconfig.get_paths()["include"], root / "include",
                   root / "include" / "torch" / "csrc" / "api" / "include", cuda / "include"]
        cmd = [shutil.which("g++") or "c++", "-O2", "-std=c++17", "-fPIC", "-shared",
               f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
               *(f"-I{p}" for p in include), str(HOST_SOURCE), "-o", str(tmp), f"-L{root / 'lib'}",
               "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
        return tmp, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    except (OSError, RuntimeError) as e:
        warnings.warn(f"the native host side of eager calls is not built: {e}")
        return None


def finish_host_build(started: tuple[Path, subprocess.Popen]) -> None:
    """The module becomes visible when it is renamed."""
    tmp, proc = started
    out, _ = proc.communicate()
    if proc.returncode == 0:
        os.replace(tmp, tmp.with_suffix(""))
        return
    tmp.unlink(missing_ok=True)
    warnings.warn(f"the native host side of eager calls is not built, the compiler failed on {HOST_SOURCE.name}:\n{out}")


def needs_build() -> bool:
    if not LIB_PATH.exists():
        return True
    built = LIB_PATH.stat().st_mtime
    deps = list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + [
        PKG_DIR.parent / "include" / "b200_sparse_ffn.h"]
    return any(p.stat().st_mtime > built for p in deps)


def build_library(force: bool = False, verbose: bool = False, extra_flags=()) -> Path:
    """Compile the library and the host module where missing or older than their sources."""
    host = start_host_build(force)
    try:
        return _build_library(force, verbose, extra_flags)
    finally:
        if host is not None:
            finish_host_build(host)


def _build_library(force: bool, verbose: bool, extra_flags) -> Path:
    if not force and not needs_build():
        return LIB_PATH
    nvcc = find_nvcc()
    objs = []
    obj_dir = PKG_DIR / "build"
    obj_dir.mkdir(exist_ok=True)
    common = [nvcc, "-gencode", GENCODE, "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", *extra_flags]
    if verbose:
        common += ["-Xptxas", "-v"]
    procs = []
    for src in sources():
        obj = obj_dir / (src.stem + ".o")
        objs.append(obj)
        procs.append((src, subprocess.Popen(
            common + ["-c", str(src), "-o", str(obj)],
            stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src, proc in procs:
        out, _ = proc.communicate()
        if verbose and out:
            print(out)
        if proc.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src.name}:\n{out}")
    tmp = LIB_PATH.with_suffix(".so.tmp")
    link = [nvcc, "-gencode", GENCODE, "-shared", "-o", str(tmp), *map(str, objs)]
    res = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc link failed:\n{res.stdout}")
    os.replace(tmp, LIB_PATH)
    return LIB_PATH


if __name__ == "__main__":
    path = build_library(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
