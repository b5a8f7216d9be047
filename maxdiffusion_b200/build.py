"""Builds the sm_100a kernel library `maxdiffusion_b200/_kernels.so` with nvcc.

The kernels export a plain C ABI (raw pointers + stream) and are loaded through ctypes, so their
build needs neither the PyTorch headers nor a JIT cache: `python -m maxdiffusion_b200.build`
compiles every `csrc/*.cu` in parallel and links one shared object next to the package, and beside it
`_host_ops.so` (csrc/host_ops.cpp, against the headers of the installed PyTorch and Python), which calls
the same entry points with less host time. Without it the ops go through the ctypes wrappers.
"""
from __future__ import annotations

import concurrent.futures
import hashlib
import os
import re
import shutil
import subprocess
import sys
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
SRC_DIR = PKG_DIR / "csrc"
OBJ_DIR = PKG_DIR / "csrc" / "build"
LIB_PATH = PKG_DIR / "_kernels.so"
HOST_PATH = PKG_DIR / "_host_ops.so"  # CPython extension over the kernel library (csrc/host_ops.cpp)

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo", "--use_fast_math",
    "-Xcompiler", "-fPIC", "-Xptxas", "-v",
]
PRECISE = {"softmax_split.cu"}  # built without --use_fast_math


def _flags(src: Path) -> list[str]:
  return [f for f in NVCC_FLAGS if f != "--use_fast_math" or src.name not in PRECISE]


def _nvcc() -> str:
  nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
  if not os.path.exists(nvcc):
    raise RuntimeError("nvcc not found; the sm_100a kernels cannot be built")
  return nvcc


def _digest(path: Path) -> str:
  h = hashlib.sha256()
  h.update(" ".join(_flags(path)).encode())
  h.update(path.read_bytes())
  for hdr in sorted(SRC_DIR.glob("*.cuh")) + sorted(SRC_DIR.glob("*.h")):
    h.update(hdr.read_bytes())
  return h.hexdigest()


def _compile_one(src: Path, verbose: bool) -> Path:
  obj = OBJ_DIR / (src.stem + ".o")
  stamp = OBJ_DIR / (src.stem + ".sha")
  digest = _digest(src)
  if obj.exists() and stamp.exists() and stamp.read_text() == digest:
    return obj
  cmd = [_nvcc(), *_flags(src), "-I", str(SRC_DIR), "-c", str(src), "-o", str(obj)]
  res = subprocess.run(cmd, capture_output=True, text=True)
  log = OBJ_DIR / (src.stem + ".ptxas.log")
  log.write_text(res.stdout + res.stderr)
  if res.returncode != 0:
    raise RuntimeError(f"nvcc failed for {src.name}:\n{res.stdout}\n{res.stderr}")
  if verbose:
    print(f"[build] compiled {src.name}")
  stamp.write_text(digest)
  return obj


def sources() -> list[Path]:
  return sorted(SRC_DIR.glob("*.cu"))


def build(verbose: bool = True, force: bool = False) -> Path:
  """Builds the kernel library and the host extension over it. Returns the library's path."""
  build_kernels(verbose, force)
  build_host_ops(verbose, force)
  return LIB_PATH


def build_kernels(verbose: bool = True, force: bool = False) -> Path:
  """Compiles every kernel for sm_100a and links `_kernels.so`. Returns its path."""
  OBJ_DIR.mkdir(parents=True, exist_ok=True)
  if force:
    for f in OBJ_DIR.glob("*.sha"):
      f.unlink()
  srcs = sources()
  with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as pool:
    objs = list(pool.map(lambda s: _compile_one(s, verbose), srcs))
  newest = max(o.stat().st_mtime for o in objs)
  if force or not LIB_PATH.exists() or LIB_PATH.stat().st_mtime < newest:
    cmd = [_nvcc(), "-shared", "-o", str(LIB_PATH), *[str(o) for o in objs], "-lcudart"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
      raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    if verbose:
      print(f"[build] linked {LIB_PATH}")
  return LIB_PATH


def host_ops_target() -> str:
  """What the extension's binary interface depends on: the versions of PyTorch and of Python."""
  import torch

  return f"PyTorch {torch.__version__}, Python {sys.version.split()[0]}"


def host_ops_built_for(path: Path) -> str | None:
  """The `host_ops_target` that an object was built for, as its text has it (the object is not loaded); None: no such object."""
  if not path.exists():
    return None
  found = re.search(rb"mdb_host_ops built for ([^;\0]+);", path.read_bytes())
  return found.group(1).decode() if found else "something unknown"


def build_host_ops(verbose: bool = True, force: bool = False) -> None:
  """Compiles csrc/host_ops.cpp against the installed PyTorch and links it to `_kernels.so` beside it."""
  import sysconfig

  import torch

  root = Path(torch.__file__).resolve().parent
  cuda = Path(_nvcc()).resolve().parent.parent
  src, obj, stamp = SRC_DIR / "host_ops.cpp", OBJ_DIR / "host_ops.o", OBJ_DIR / "host_ops.sha"
  flags = ["-std=c++17", "-O2", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           f'-DMDB_BUILT_FOR="{host_ops_target()}"']
  digest = hashlib.sha256(" ".join([torch.__version__, sys.version, *flags]).encode() + src.read_bytes()).hexdigest()
  if force or host_ops_built_for(HOST_PATH) != host_ops_target() or not stamp.exists() or stamp.read_text() != digest:
    inc = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", sysconfig.get_paths()["include"], cuda / "include"]
    libs = ["-L", str(PKG_DIR), "-l:_kernels.so", "-Wl,-rpath,$ORIGIN", "-L", str(root / "lib"), "-ltorch_python", "-ltorch_cpu",
            "-ltorch", "-lc10_cuda", "-lc10"]  # PyTorch's libraries are loaded before this one: no run path to them
    for cmd in (["g++", *flags, *[f"-I{i}" for i in inc], "-c", str(src), "-o", str(obj)],
                ["g++", "-shared", str(obj), "-o", str(HOST_PATH), *libs]):
      res = subprocess.run(cmd, capture_output=True, text=True)
      if res.returncode != 0:
        raise RuntimeError(f"{src.name}: {' '.join(cmd[:2])} failed:\n{res.stdout}\n{res.stderr}")
    stamp.write_text(digest)
    if verbose:
      print(f"[build] linked {HOST_PATH}")


if __name__ == "__main__":
  build(verbose=True, force="--force" in sys.argv)
