"""Builds the sm_100a kernel library in-tree with nvcc.

Every ``csrc/*.cu`` file is compiled with ``-gencode arch=compute_100a,code=sm_100a`` and linked
into ``ultraattn_b200/lib/libultraattn_sm100.so``. The library exposes a plain C ABI (loaded with
ctypes by :mod:`ultraattn_b200._lib`), so its sources see no PyTorch headers and a full rebuild
takes well under a minute. nvcc cross-compiles, so this works on a machine without a GPU.
Beside it, ``csrc/host_ext.cpp``, the native host part of single-device calls, becomes the Python extension
``lib/ua_host.<ABI>.so`` for this interpreter and this PyTorch. It is optional: everything it does is there in Python too,
so without a C++ compiler or Python's headers the library is built alone, with a warning.

The reference ships no native code of its own (it builds NCCL and a flash-attention fork through
``scripts/Makefile:47-96``); this is the equivalent build step of this framework.
"""
from __future__ import annotations

import hashlib
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig
import warnings
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
LIB_DIR = PKG_DIR / "lib"
LIB_PATH = LIB_DIR / "libultraattn_sm100.so"
OBJ_DIR = LIB_DIR / "obj"
HOST_PATH = LIB_DIR / f"ua_host{sysconfig.get_config_var('EXT_SUFFIX') or '.so'}"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    cand = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(cand).exists():
        raise RuntimeError("nvcc not found; set NVCC or add /usr/local/cuda/bin to PATH")
    return cand


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _newest_header_mtime() -> float:
    hdrs = list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h"))
    return max((p.stat().st_mtime for p in hdrs), default=0.0)


STAMP_PATH = LIB_DIR / "build_stamp.txt"


def _digest(files: list, *more: str) -> str:
    """Hash of what a binary is built from (sources, headers, compiler flags). File times do not survive every way of
    copying a tree to another machine; contents do."""
    h = hashlib.sha256("\n".join(more).encode())
    for f in sorted(files):
        h.update(f.name.encode())
        h.update(f.read_bytes())
    return h.hexdigest()


def source_digest() -> str:
    """Hash of everything the kernel library is built from."""
    return _digest([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh"), *CSRC.glob("*.h")], " ".join(NVCC_FLAGS))


def needs_build() -> bool:
    """True when the library is missing or was built from other sources than the present ones."""
    if not LIB_PATH.exists() or not STAMP_PATH.exists():
        return True
    return STAMP_PATH.read_text().strip() != source_digest()


HOST_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-lc10", "-ltorch_cpu", "-ltorch_python"]


def _cxx() -> str:
    return os.environ.get("CXX") or "g++"


def _torch_dir() -> Path:
    return Path(importlib.util.find_spec("torch").origin).parent          # (found, not imported)


def _host_command(out: Path) -> list[str]:
    t = _torch_dir()
    return [_cxx(), f"-I{t / 'include'}", f"-I{t / 'include' / 'torch' / 'csrc' / 'api' / 'include'}",
            f"-I{sysconfig.get_paths()['include']}", str(CSRC / "host_ext.cpp"), "-o", str(out), f"-L{t / 'lib'}", *HOST_FLAGS,
            f"-Wl,-rpath,{t / 'lib'}"]


def _host_stamp() -> Path:
    return HOST_PATH.with_name(HOST_PATH.name + ".stamp")


def host_digest() -> str:
    """Hash of everything the host extension is built from: its sources and flags, the interpreter and the PyTorch."""
    return _digest([CSRC / "host_ext.cpp", *CSRC.glob("*.h"), _torch_dir() / "version.py"], _cxx(), *HOST_FLAGS,
                   str(sysconfig.get_config_var("SOABI")))


def _host_tools() -> str:
    """What a build of the host extension that failed may have lacked (it is tried again when this changes)."""
    return f"{shutil.which(_cxx())} {(Path(sysconfig.get_paths()['include']) / 'Python.h').exists()}"


def host_path() -> Path | None:
    """The host extension, if there is one that belongs to the present sources, interpreter and PyTorch."""
    try:
        ok = HOST_PATH.exists() and _host_stamp().read_text().strip() == host_digest()
    except (OSError, AttributeError):           # (AttributeError: no PyTorch)
        return None
    return HOST_PATH if ok else None


def _host_needs_build() -> bool:
    if host_path() is not None:
        return False
    try:
        return _host_stamp().read_text().strip() != f"failed {host_digest()} {_host_tools()}"
    except OSError:
        return True
    except AttributeError:
        return False


def build_all(force: bool = False, verbose: bool = False) -> Path:
    """Compile (if stale) the kernel library and the host extension; return the path of the library."""
    if not force and not needs_build() and not _host_needs_build():
        return LIB_PATH
    try:
        OBJ_DIR.mkdir(parents=True, exist_ok=True)
        (LIB_DIR / ".build.lock").touch()
    except OSError:
        if force or needs_build():
            raise
        return LIB_PATH                         # (a read-only installation whose library is there)
    # several ranks may arrive here at once on a machine where the library is missing: one builds,
    # the others wait for the lock and then find the library up to date
    import fcntl
    lock = open(LIB_DIR / ".build.lock", "w")
    fcntl.flock(lock, fcntl.LOCK_EX)
    try:
        with ThreadPoolExecutor(max_workers=1) as ex:
            host = ex.submit(_build_host) if force or _host_needs_build() else None
            if force or needs_build():
                _build_locked(_nvcc(), force, verbose)
            if host is not None:
                host.result()
        return LIB_PATH
    finally:
        fcntl.flock(lock, fcntl.LOCK_UN)
        lock.close()


def _build_locked(nvcc: str, force: bool, verbose: bool) -> Path:
    hdr = _newest_header_mtime()

    def compile_one(src: Path) -> Path:
        obj = OBJ_DIR / (src.stem + ".o")
        if (not force and obj.exists() and obj.stat().st_mtime > src.stat().st_mtime
                and obj.stat().st_mtime > hdr):
            return obj
        cmd = [nvcc, *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose and r.stderr:
            sys.stderr.write(r.stderr)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{r.stdout}\n{r.stderr}")
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        objs = list(ex.map(compile_one, sources()))
    tmp = LIB_PATH.with_suffix(".so.tmp")
    cmd = [nvcc, "-shared", "-o", str(tmp), *map(str, objs),
           "-gencode", "arch=compute_100a,code=sm_100a"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    os.replace(tmp, LIB_PATH)          # a reader never sees a half-written library
    STAMP_PATH.write_text(source_digest() + "\n")
    return LIB_PATH


def _build_host() -> None:
    tmp = HOST_PATH.with_name(HOST_PATH.name + ".tmp")
    try:
        digest = host_digest()
        r = subprocess.run(_host_command(tmp), capture_output=True, text=True)
        error = f"{r.stdout}\n{r.stderr}".strip() if r.returncode != 0 else ""
    except AttributeError:
        return                                  # no PyTorch, nothing to build for
    except OSError as e:
        error = str(e)
    if error:
        _host_stamp().write_text(f"failed {digest} {_host_tools()}\n")
        warnings.warn(f"ultraattn_b200: the host extension was not built; calls go through Python instead. {error[-2000:]}")
        return
    os.replace(tmp, HOST_PATH)
    _host_stamp().write_text(digest + "\n")


if __name__ == "__main__":
    path = build_all(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
