"""Builds the native library (``libmaco_b200.so``) in-tree with nvcc for sm_100a.

The reference builds its extension with setuptools for compute_70..90 only
(maco/csrc/setup_sm.py:66-83, maco/csrc/setup.py:108-125); here there is one target, sm_100a, and
the result is a plain shared library with ``extern "C"`` entry points loaded through ctypes, so a
rebuild takes seconds and the library has no libtorch dependency.
"""
from __future__ import annotations

import hashlib
import os
import shlex
import shutil
import subprocess
import sys
import sysconfig
import warnings
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
REPO_DIR = PKG_DIR.parent
CSRC_DIR = REPO_DIR / "csrc"
LIB_DIR = PKG_DIR / "_lib"
LIB_PATH = LIB_DIR / "libmaco_b200.so"
OBJ_DIR = REPO_DIR / "build" / "obj"
FASTCALL_SRC = CSRC_DIR / "py" / "fastcall.c"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr", "--expt-extended-lambda",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("MACO_NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set MACO_NVCC")


def sources() -> list[Path]:
    return sorted(CSRC_DIR.glob("*.cu"))


def _digest(src: Path) -> str:
    h = hashlib.sha256()
    h.update(" ".join(NVCC_FLAGS).encode())
    h.update(src.read_bytes())
    for hdr in sorted(list(CSRC_DIR.glob("*.h")) + list(CSRC_DIR.glob("*.cuh"))):
        h.update(hdr.read_bytes())
    return h.hexdigest()


def _compile_one(src: Path, verbose: bool) -> Path:
    OBJ_DIR.mkdir(parents=True, exist_ok=True)
    obj = OBJ_DIR / (src.stem + ".o")
    stamp = OBJ_DIR / (src.stem + ".sha")
    dig = _digest(src)
    if obj.exists() and stamp.exists() and stamp.read_text() == dig:
        return obj
    cmd = [_nvcc(), *NVCC_FLAGS, "-I", str(CSRC_DIR), "-c", str(src), "-o", str(obj)]
    if verbose:
        print("[maco_b200 build]", " ".join(cmd), file=sys.stderr)
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src.name}:\n{res.stdout}\n{res.stderr}")
    stamp.write_text(dig)
    return obj


def fastcall_path() -> Path:
    """Where the C extension of this source and this interpreter lies. Both are part of the name: CPython loads an untagged extension that
    another minor version built without a word, and runs it with that version's inlined reference counts and tuple layout. Where the package
    lies without its source, the build that came with it."""
    suffix = sysconfig.get_config_var("EXT_SUFFIX")
    if not FASTCALL_SRC.exists():
        came = sorted(LIB_DIR.glob(f"maco_fastcall-*{suffix}"))
        if len(came) == 1:
            return came[0]
    digest = hashlib.sha256(FASTCALL_SRC.read_bytes()).hexdigest()[:12]
    return LIB_DIR / f"maco_fastcall-{digest}{suffix}"


def build_fastcall(force: bool = False) -> "Path | None":
    """The C extension behind the smallest calls (csrc/py/fastcall.c), for this interpreter. None where there is no compiler or no Python
    header, an exception where the compiler fails: those calls then take their general path."""
    include = sysconfig.get_paths()["include"]
    # CC may hold arguments, or a launcher in front of the compiler ("gcc -pthread", "ccache gcc")
    cc = shlex.split(os.environ.get("CC", "")) or [c for c in (shutil.which("gcc") or shutil.which("cc"),) if c]
    if not cc or not os.path.exists(os.path.join(include, "Python.h")):
        return None
    path = fastcall_path()
    if path.exists() and not force:
        return path
    LIB_DIR.mkdir(parents=True, exist_ok=True)
    tmp = path.with_name(f"{path.name}.{os.getpid()}.tmp")
    res = subprocess.run([*cc, "-O2", "-shared", "-fPIC", "-I", include, str(FASTCALL_SRC), "-o", str(tmp)], capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"{shlex.join(cc)} failed for {FASTCALL_SRC.name}:\n{res.stdout}\n{res.stderr}")
    os.replace(tmp, path)
    for old in LIB_DIR.glob("maco_fastcall*"):              # of other states of the source; other interpreters keep theirs
        if old != path and (old.name == "maco_fastcall.so" or old.name.endswith(sysconfig.get_config_var("EXT_SUFFIX"))):
            old.unlink(missing_ok=True)
    return path


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compiles every ``csrc/*.cu`` for sm_100a and links ``maco_b200/_lib/libmaco_b200.so``."""
    srcs = sources()
    if not srcs:
        raise RuntimeError(f"no CUDA sources under {CSRC_DIR}")
    if force and OBJ_DIR.exists():
        shutil.rmtree(OBJ_DIR)
    with ThreadPoolExecutor(max_workers=min(8, len(srcs))) as pool:
        objs = list(pool.map(lambda s: _compile_one(s, verbose), srcs))
    LIB_DIR.mkdir(parents=True, exist_ok=True)
    newest = max(o.stat().st_mtime for o in objs)
    if force or not LIB_PATH.exists() or LIB_PATH.stat().st_mtime < newest:
        cmd = [_nvcc(), "-shared", "-o", str(LIB_PATH), *[str(o) for o in objs], "-Xcompiler", "-fPIC"]
        if verbose:
            print("[maco_b200 build]", " ".join(cmd), file=sys.stderr)
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    try:
        build_fastcall(force)
    except (OSError, RuntimeError, ValueError) as exc:       # the calls it is for take their general path
        warnings.warn(f"the C extension was not built: {exc}")
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
