"""Building the native code: several processes at once, what makes a binary stale, no compiler. The
compilers are stand-ins that write their inputs' names slowly, in two parts."""
import os
import subprocess
import sys
import textwrap

import pytest

from t5x_b200.ops import build, native

FAKE = """\
#!/bin/sh
out=""
while [ $# -gt 0 ]; do [ "$1" = "-o" ] && out="$2"; shift; done
echo "$out" >> "$BUILD_LOG"
printf first > "$out"; sleep 0.3; printf second >> "$out"
"""


def _tree(tmp_path):
  csrc, lib, tools = tmp_path / "csrc", tmp_path / "lib", tmp_path / "bin"
  for d in (csrc / "host", lib / "obj", tools):
    d.mkdir(parents=True)
  for f in ("a.cu", "b.cu", "t5x_b200.h", "t5x_ops.h", "host/host_ops.cpp"):
    (csrc / f).write_text(f)
  for t in ("g++", "nvcc"):
    (tools / t).write_text(FAKE)
    (tools / t).chmod(0o755)
  return csrc, lib, tools


def _point(module, csrc, lib):
  module.CSRC, module.LIB_DIR, module.OBJ_DIR = str(csrc), str(lib), str(lib / "obj")
  module.LIB_PATH, module.HOST_SRC = str(lib / "libt5x_b200.so"), str(csrc / "host" / "host_ops.cpp")


@pytest.fixture
def tree(tmp_path, monkeypatch):
  csrc, lib, tools = _tree(tmp_path)
  for name in ("CSRC", "LIB_DIR", "OBJ_DIR", "LIB_PATH", "HOST_SRC"):
    monkeypatch.setattr(build, name, getattr(build, name))
  _point(build, csrc, lib)
  monkeypatch.setenv("PATH", f"{tools}:{os.environ['PATH']}")
  monkeypatch.setenv("NVCC", str(tools / "nvcc"))
  monkeypatch.setenv("BUILD_LOG", str(tmp_path / "log"))
  return csrc, lib


def _log(lib):
  path = lib.parent / "log"
  return path.read_text().split() if path.exists() else []


def test_processes_that_build_at_once_get_one_whole_file(tree):
  csrc, lib = tree
  code = textwrap.dedent(f"""
      import sys; sys.path.insert(0, {build.ROOT!r}); sys.path.insert(0, {os.path.dirname(__file__)!r})
      from pathlib import Path
      from t5x_b200.ops import build
      from test_build import _point
      _point(build, Path({str(csrc)!r}), Path({str(lib)!r}))
      build.build()
      for p in (build.LIB_PATH, build.host_path()):
        assert open(p).read() == "firstsecond", p
  """)
  procs = [subprocess.Popen([sys.executable, "-c", code], stderr=subprocess.PIPE, text=True)
           for _ in range(4)]
  for p in procs:
    err = p.communicate(timeout=120)[1]
    assert p.returncode == 0, err
  assert len(_log(lib)) == 4  # two objects, the library, the extension: each once
  assert not [f for f in os.listdir(lib) if "tmp" in f]


def test_extension_is_rebuilt_when_what_it_depends_on_changes(tree, monkeypatch):
  import torch
  csrc, lib = tree
  first = build.build_host()
  assert build.build_host() == first and len(_log(lib)) == 1
  (csrc / "t5x_ops.h").write_text("int t5x_rmsnorm_fwd(int);")  # an entry's argument list
  second = build.build_host()
  assert second != first and not os.path.exists(first) and os.path.exists(second)
  monkeypatch.setattr(torch, "__version__", "99.0")
  assert build.host_path() != second


def test_library_is_linked_again_without_a_deleted_source(tree):
  csrc, lib = tree
  build.build()
  n = len(_log(lib))
  build.build()
  assert len(_log(lib)) == n
  (csrc / "b.cu").unlink()
  build.build()
  assert len(_log(lib)) == n + 1 and not (lib / "obj" / "b.o").exists()


def test_failed_build_leaves_nothing(tree, monkeypatch):
  csrc, lib = tree
  (lib.parent / "bin" / "g++").write_text("#!/bin/sh\nexit 1\n")
  with pytest.raises(RuntimeError):
    build.build_host()
  assert not [f for f in os.listdir(lib) if f.endswith(".so")]


def test_ops_run_without_the_extension(monkeypatch):
  """No compiler and no binary: one warning, and the general path of the ops."""
  monkeypatch.setattr(native, "_host", None)
  monkeypatch.setattr(native, "lib", lambda: None)
  monkeypatch.delenv("T5X_B200_HOST_OPS", raising=False)

  def missing():
    raise FileNotFoundError("g++")
  monkeypatch.setattr(build, "load_host", missing)
  with pytest.warns(RuntimeWarning, match="ctypes"):
    assert native.host() is None
  assert native.host() is None
