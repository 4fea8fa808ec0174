"""Build recipe for libgbsv.so (the CUDA kernels behind the C ABI).

Each ``csrc/*.cu`` translation unit is compiled for sm_103a only, in
parallel, then linked into ``_build/libgbsv.so`` beside this file; the native
host path (``csrc/host/host.cpp``, against the installed torch) becomes an
extension module beside it.  Nothing is installed into site-packages, so the
libraries that Python loads are the in-tree ones.  A stamp of source hashes
skips the rebuild when nothing changed.
"""
from __future__ import annotations

import concurrent.futures as cf
import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
REPO_DIR = PKG_DIR.parent
CSRC = PKG_DIR / "csrc"
INCLUDE = REPO_DIR / "include"
BUILD_DIR = PKG_DIR / "_build"
LIB_NAME = "libgbsv.so"
HOST_MODULE = "_gbsv_host"
HOST_SOURCE = CSRC / "host" / "host.cpp"
ARCH_FLAGS = ["-gencode", "arch=compute_103a,code=sm_103a"]
NVCC_FLAGS = [
    "-O3", "-std=c++17", "-lineinfo", "--expt-relaxed-constexpr",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-O3",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"),
                 "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found; the CUDA toolkit is required to build "
                       "libgbsv.so")


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cpp"))


def _cxx() -> str:
    return os.environ.get("CXX") or shutil.which("g++") or "g++"


def _stamp() -> str:
    h = hashlib.sha256()
    for p in sorted(list(CSRC.rglob("*")) + list(INCLUDE.glob("*.h"))):
        if p.is_file():
            h.update(p.name.encode())
            h.update(p.read_bytes())
    h.update(" ".join(ARCH_FLAGS + NVCC_FLAGS).encode())
    h.update(os.uname().machine.encode())
    compile_flags, link_flags = _host_flags()
    h.update(" ".join(compile_flags + link_flags).encode())
    h.update(f"{host_tag()} {host_headers()}".encode())
    return h.hexdigest()


def host_tag() -> str:
    """What a built host module goes with: torch's C++ interface and the
    interpreter's."""
    import torch
    return f"torch {torch.__version__}, Python {sys.version}"


def _torch_root() -> Path:
    import torch
    return Path(torch.__file__).resolve().parent


def host_headers() -> bool:
    """Whether the headers that the host module needs are installed (the
    library of kernels needs neither Python's nor torch's)."""
    return (Path(sysconfig.get_paths()["include"]) / "Python.h").exists() and (
        _torch_root() / "include" / "torch" / "csrc" / "autograd" /
        "custom_function.h").exists()


def _host_flags() -> tuple[list[str], list[str]]:
    """(compile flags, link flags) of the host module: torch's headers and
    libraries, the C ABI's library found beside the module."""
    import torch
    root = _torch_root()
    inc = [root / "include",
           root / "include" / "torch" / "csrc" / "api" / "include",
           Path(sysconfig.get_paths()["include"]), INCLUDE]
    abi = int(torch._C._GLIBCXX_USE_CXX11_ABI)
    compile_flags = ["-O2", "-std=c++17", "-fPIC",
                     f"-D_GLIBCXX_USE_CXX11_ABI={abi}",
                     *[f"-isystem{i}" for i in inc]]
    link_flags = [f"-L{BUILD_DIR}", "-lgbsv", "-Wl,-rpath,$ORIGIN",
                  f"-L{root / 'lib'}", "-lc10", "-lc10_cuda", "-ltorch_cpu",
                  "-ltorch_cuda", "-ltorch", "-ltorch_python"]
    return compile_flags, link_flags


def lib_path() -> Path:
    return BUILD_DIR / LIB_NAME


def host_path() -> Path:
    return BUILD_DIR / f"{HOST_MODULE}.so"


def host_tag_path() -> Path:
    return BUILD_DIR / f"{HOST_MODULE}.txt"


def build(verbose: bool = False, force: bool = False,
          extra_flags: list[str] | None = None) -> Path:
    """Compile and link libgbsv.so and, where its headers are installed, the
    host module; return the library's path."""
    BUILD_DIR.mkdir(parents=True, exist_ok=True)
    stamp_file = BUILD_DIR / "stamp.txt"
    stamp = _stamp() + (" ".join(extra_flags) if extra_flags else "")
    out = lib_path()
    with_host = host_headers()
    if (not force and out.exists() and host_path().exists() == with_host
            and stamp_file.exists() and stamp_file.read_text() == stamp):
        return out
    nvcc = _nvcc()
    flags = ARCH_FLAGS + NVCC_FLAGS + (extra_flags or []) + [
        f"-I{INCLUDE}", f"-I{CSRC}"]
    objs = []
    host_compile, host_link = _host_flags()
    host_compile.append(
        f"-isystem{Path(nvcc).resolve().parent.parent / 'include'}")

    def compile_one(src: Path) -> Path:
        obj = BUILD_DIR / (src.stem + ".o")
        if src == HOST_SOURCE:
            cmd = [_cxx(), *host_compile, "-c", str(src), "-o", str(obj)]
        elif src.suffix == ".cpp":  # host-only code
            cmd = [_cxx(), "-O3", "-std=c++17", "-fPIC", f"-I{INCLUDE}",
                   f"-I{CSRC}", "-c", str(src), "-o", str(obj)]
        else:
            cmd = [nvcc, *flags, "-c", str(src), "-o", str(obj)]
        if verbose:
            print(" ".join(cmd), flush=True)
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"compile failed on {src.name}:\n{res.stderr}")
        if verbose and res.stderr:
            print(res.stderr, file=sys.stderr)
        return obj

    srcs = sources() + ([HOST_SOURCE] if with_host else [])
    with cf.ThreadPoolExecutor(max_workers=min(len(srcs), os.cpu_count() or 4)) as ex:
        objs = list(ex.map(compile_one, srcs))
    tmp = out.with_suffix(".so.tmp")

    def link(cmd):
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stderr}")

    lib_objs = objs[:len(sources())]
    link([nvcc, *ARCH_FLAGS, "-shared", "-o", str(tmp),
          f"-Xlinker=-soname={LIB_NAME}", *map(str, lib_objs), "-lcudart"])
    os.replace(tmp, out)
    if with_host:
        tmp = host_path().with_suffix(".so.tmp")
        link([_cxx(), "-shared", "-o", str(tmp), str(objs[-1]), *host_link])
        os.replace(tmp, host_path())
        host_tag_path().write_text(host_tag())
    else:
        host_path().unlink(missing_ok=True)
        print(f"{HOST_MODULE} not built: Python.h or torch's headers are "
              "missing; calls take the Python route", file=sys.stderr)
    stamp_file.write_text(stamp)
    return out


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="-f" in sys.argv))
