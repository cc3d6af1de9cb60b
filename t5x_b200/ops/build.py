"""Builds the native sm_100a library in-tree.

Every ``csrc/*.cu`` file is compiled with ``nvcc -gencode arch=compute_100a,code=sm_100a``
and linked into ``t5x_b200/lib/libt5x_b200.so``; the result is loaded with ctypes by
:mod:`t5x_b200.ops.native`. nvcc cross-compiles without a GPU present.
"""
from __future__ import annotations

import concurrent.futures as cf
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
HOST_PATH = os.path.join(LIB_DIR, HOST_NAME + ".so")

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


def build(verbose: bool = False, force: bool = False, ptxas_v: bool = False) -> str:
  """Compiles what is out of date and links the shared library. Returns its path."""
  os.makedirs(OBJ_DIR, exist_ok=True)
  srcs = sources()
  if force:
    for f in os.listdir(OBJ_DIR):
      os.remove(os.path.join(OBJ_DIR, f))
  with cf.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
    objs = list(ex.map(lambda s: _compile(s, verbose, ptxas_v), srcs))
  if (not os.path.exists(LIB_PATH)) or any(os.path.getmtime(o) > os.path.getmtime(LIB_PATH) for o in objs):
    cmd = [_nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB_PATH, *objs]
    if verbose:
      print(" ".join(cmd), flush=True)
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
      raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
  build_host(verbose, force)
  return LIB_PATH


def build_host(verbose: bool = False, force: bool = False) -> str:
  """Compiles the Python extension that takes tensors to kernel launches; it is linked with the
  kernel library beside it."""
  if not force and os.path.exists(HOST_PATH) and \
      os.path.getmtime(HOST_PATH) >= os.path.getmtime(HOST_SRC):
    return HOST_PATH
  import sysconfig
  import torch
  root = os.path.dirname(torch.__file__)
  cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
  includes = [os.path.join(root, "include"),
              os.path.join(root, "include", "torch", "csrc", "api", "include"),
              os.path.join(cuda, "include"), sysconfig.get_path("include")]
  cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared",
         f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
         f"-DTORCH_EXTENSION_NAME={HOST_NAME}", "-DTORCH_API_INCLUDE_EXTENSION_H",
         *(f"-I{d}" for d in includes), HOST_SRC, "-o", HOST_PATH + ".tmp",
         f"-L{LIB_DIR}", "-lt5x_b200", f"-L{os.path.join(root, 'lib')}", "-lc10", "-ltorch",
         "-ltorch_cpu", "-ltorch_python", "-lc10_cuda", "-ltorch_cuda", "-Wl,-rpath,$ORIGIN"]
  if verbose:
    print(" ".join(cmd), flush=True)
  r = subprocess.run(cmd, capture_output=True, text=True)
  if r.returncode != 0:
    raise RuntimeError(f"g++ failed for {HOST_SRC}:\n{r.stdout}\n{r.stderr}")
  os.replace(HOST_PATH + ".tmp", HOST_PATH)
  return HOST_PATH


def load_host():
  """The extension module, built first if it is missing."""
  import importlib.machinery
  import importlib.util
  if not os.path.exists(HOST_PATH):
    build_host()
  loader = importlib.machinery.ExtensionFileLoader(HOST_NAME, HOST_PATH)
  spec = importlib.util.spec_from_file_location(HOST_NAME, HOST_PATH, loader=loader)
  module = importlib.util.module_from_spec(spec)
  loader.exec_module(module)
  return module


if __name__ == "__main__":
  print(build(verbose=True, force="--force" in sys.argv, ptxas_v="--ptxas-v" in sys.argv))
