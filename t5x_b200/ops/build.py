"""Builds the native sm_100a library in-tree.

Every ``csrc/*.cu`` file is compiled with ``nvcc -gencode arch=compute_100a,code=sm_100a``
and linked into ``t5x_b200/lib/libt5x_b200.so``; the result is loaded with ctypes by
:mod:`t5x_b200.ops.native`. nvcc cross-compiles without a GPU present. Beside it stands the Python
extension ``_t5x_host.<key>.so`` (csrc/host). Several processes may build at the same time: a file
lock lets one do it, and finished files are moved into place.
"""
from __future__ import annotations

import concurrent.futures as cf
import contextlib
import fcntl
import hashlib
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
CSRC = os.path.join(ROOT, "csrc")
LIB_DIR = os.path.join(ROOT, "t5x_b200", "lib")
OBJ_DIR = os.path.join(LIB_DIR, "obj")
LIB_PATH = os.path.join(LIB_DIR, "libt5x_b200.so")
HOST_SRC = os.path.join(CSRC, "host", "host_ops.cpp")
HOST_NAME = "_t5x_host"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--use_fast_math", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
  cand = os.environ.get("NVCC") or os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
  return cand if os.path.exists(cand) else "nvcc"


def sources() -> list[str]:
  return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _headers_mtime() -> float:
  return max([os.path.getmtime(os.path.join(CSRC, f)) for f in os.listdir(CSRC)
              if f.endswith((".cuh", ".h"))] + [0.0])


def _compile(src: str, verbose: bool, ptxas_v: bool) -> str:
  obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
  newest = max(os.path.getmtime(src), _headers_mtime())
  if os.path.exists(obj) and os.path.getmtime(obj) >= newest:
    return obj
  cmd = [_nvcc(), *NVCC_FLAGS, "-I", CSRC, "-c", src, "-o", obj]
  if ptxas_v:
    cmd[1:1] = ["-Xptxas", "-v"]
  if verbose:
    print(" ".join(cmd), flush=True)
  r = subprocess.run(cmd, capture_output=True, text=True)
  if r.returncode != 0:
    raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
  if ptxas_v or verbose:
    sys.stderr.write(r.stderr)
  return obj


@contextlib.contextmanager
def _build_lock():
  """One builder at a time, over all processes that share this tree."""
  os.makedirs(OBJ_DIR, exist_ok=True)
  with open(os.path.join(OBJ_DIR, "lock.o"), "w") as f:
    fcntl.flock(f, fcntl.LOCK_EX)
    yield


def _run_to(path: str, cmd: list, verbose: bool) -> None:
  """Runs the command, whose output file is `path`, into a file of this process's own and moves
  that into place."""
  tmp = f"{path}.{os.getpid()}.tmp.so"
  cmd = [tmp if c == path else c for c in cmd]
  if verbose:
    print(" ".join(cmd), flush=True)
  try:
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
      raise RuntimeError(f"{cmd[0]} failed for {path}:\n{r.stdout}\n{r.stderr}")
    os.replace(tmp, path)
  finally:
    if os.path.exists(tmp):
      os.remove(tmp)


def build(verbose: bool = False, force: bool = False, ptxas_v: bool = False) -> str:
  """Compiles what is out of date and links the shared library. Returns its path."""
  with _build_lock():
    srcs = sources()
    wanted = {os.path.basename(s)[:-3] + ".o" for s in srcs}
    relink = not os.path.exists(LIB_PATH)
    for f in os.listdir(OBJ_DIR):
      if f != "lock.o" and (force or f not in wanted):  # also the objects of deleted sources
        os.remove(os.path.join(OBJ_DIR, f))
        relink = True
    with cf.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
      objs = list(ex.map(lambda s: _compile(s, verbose, ptxas_v), srcs))
    if relink or any(os.path.getmtime(o) > os.path.getmtime(LIB_PATH) for o in objs):
      _run_to(LIB_PATH, [_nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o",
                         LIB_PATH, *objs], verbose)
  build_host(verbose, force)
  return LIB_PATH


def host_path() -> str:
  """Where the Python extension for this interpreter, torch and source lies. The name holds a digest
  of everything the binary depends on: its source, the headers with the prototypes of the kernel
  library, and the versions and ABI of Python and torch."""
  import sysconfig
  import torch
  h = hashlib.sha256()
  for f in (HOST_SRC, os.path.join(CSRC, "t5x_b200.h"), os.path.join(CSRC, "t5x_ops.h")):
    with open(f, "rb") as fh:
      h.update(fh.read())
  h.update(repr((torch.__version__, torch.version.cuda, torch._C._GLIBCXX_USE_CXX11_ABI,
                 sysconfig.get_config_var("SOABI"))).encode())
  return os.path.join(LIB_DIR, f"{HOST_NAME}.{h.hexdigest()[:12]}.so")


def build_host(verbose: bool = False, force: bool = False) -> str:
  """Compiles the Python extension that takes tensors to kernel launches unless it is there; it is
  linked with the kernel library beside it."""
  import sysconfig
  import torch
  path = host_path()
  with _build_lock():
    if not force and os.path.exists(path):
      return path
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    includes = [CSRC, os.path.join(root, "include"),
                os.path.join(root, "include", "torch", "csrc", "api", "include"),
                os.path.join(cuda, "include"), sysconfig.get_path("include")]
    _run_to(path, ["g++", "-O2", "-std=c++17", "-fPIC", "-shared",
                   f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                   f"-DTORCH_EXTENSION_NAME={HOST_NAME}", "-DTORCH_API_INCLUDE_EXTENSION_H",
                   *(f"-I{d}" for d in includes), HOST_SRC, "-o", path,
                   f"-L{LIB_DIR}", "-lt5x_b200", f"-L{os.path.join(root, 'lib')}", "-lc10", "-ltorch",
                   "-ltorch_cpu", "-ltorch_python", "-lc10_cuda", "-ltorch_cuda",
                   "-Wl,-rpath,$ORIGIN"], verbose)
    for f in os.listdir(LIB_DIR):  # what earlier sources or versions left
      if f.startswith(HOST_NAME + ".") and f.endswith(".so") and ".tmp." not in f and \
          f != os.path.basename(path):
        os.remove(os.path.join(LIB_DIR, f))
  return path


def load_host():
  """The extension module, built first if it is missing."""
  import importlib.machinery
  import importlib.util
  path = host_path()
  if not os.path.exists(path):
    build_host()
  loader = importlib.machinery.ExtensionFileLoader(HOST_NAME, path)
  spec = importlib.util.spec_from_file_location(HOST_NAME, path, loader=loader)
  module = importlib.util.module_from_spec(spec)
  loader.exec_module(module)
  return module


if __name__ == "__main__":
  print(build(verbose=True, force="--force" in sys.argv, ptxas_v="--ptxas-v" in sys.argv))
