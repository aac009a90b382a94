"""What the two shared objects need to be built and loaded: the C library nvcc alone, the host side the torch in use."""
import os
import subprocess
import sys

import pytest

from tokamax_b200 import _native

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _compiler(tmp_path, name):
  """A stand-in that writes its arguments to the -o file."""
  path = tmp_path / name
  path.write_text('#!/bin/sh\nall="$*"\nwhile [ $# -gt 1 ]; do [ "$1" = -o ] && out="$2"; shift; done\necho "$all" > "$out"\n')
  path.chmod(0o755)
  return str(path)


def test_the_library_builds_and_loads_without_torch_and_without_a_host_compiler(tmp_path):
  program = f"""
import sys
sys.modules["torch"] = None  # `import torch` raises
from tokamax_b200 import _native
built = _native.LIB_PATH
_native._LIB_DIR, _native.LIB_PATH = {str(tmp_path)!r}, {str(tmp_path / "lib.so")!r}
assert _native.build() == _native.LIB_PATH and "splash_torch.cpp" not in open(_native.LIB_PATH).read()
_native.LIB_PATH = built
import tokamax_b200
info, _ = tokamax_b200.process_mask(tokamax_b200.CausalMask((512, 512)), (128, 128))
assert int(info.num_active_blocks[0]) == 10
try:
  _native.host()
except ImportError:
  print("only the host side needs torch")
"""
  env = dict(os.environ, NVCC=_compiler(tmp_path, "nvcc"), CXX="/nonexistent/g++")
  out = subprocess.run([sys.executable, "-c", program], cwd=ROOT, env=env, capture_output=True, text=True)
  assert out.returncode == 0, out.stderr
  assert "only the host side needs torch" in out.stdout


def test_the_host_side_is_rebuilt_for_another_torch(monkeypatch, tmp_path):
  import torch

  monkeypatch.setattr(_native, "_LIB_DIR", str(tmp_path))
  monkeypatch.setenv("CXX", _compiler(tmp_path, "g++"))
  first = _native.build_host()
  assert os.path.exists(first) and _native.build_host() == first
  monkeypatch.setattr(torch, "__version__", "2.99.0")
  assert not os.path.exists(_native.host_path())
  second = _native.build_host()
  assert second != first and os.path.exists(second)


def test_the_host_side_is_not_built_beside_an_older_library_in_use(monkeypatch, tmp_path):
  monkeypatch.setattr(_native, "_LIB_DIR", str(tmp_path))
  monkeypatch.setattr(_native, "LIB_PATH", str(tmp_path / "libsplash_b200.so"))
  monkeypatch.setenv("CXX", _compiler(tmp_path, "g++"))
  monkeypatch.setenv("NVCC", _compiler(tmp_path, "nvcc"))
  (tmp_path / "libsplash_b200.so").write_text("older than the header")
  os.utime(tmp_path / "libsplash_b200.so", (1, 1))
  monkeypatch.setattr(_native, "_lib", object())
  with pytest.raises(RuntimeError, match="already loaded"):
    _native.build_host()
  monkeypatch.setattr(_native, "_lib", None)
  assert os.path.exists(_native.build_host())
  assert "splash_fwd_sm100.cu" in (tmp_path / "libsplash_b200.so").read_text()


def test_the_host_side_loads():
  assert {"bind_library", "forward", "backward"} <= set(dir(_native.host()))


def test_errors_of_the_host_side_are_exceptions():
  # in a process of its own: a module with another C++ runtime than torch's ends it
  program = """
import torch
from tokamax_b200 import _native
host = _native.host()
t, f, rec = torch.zeros(1, 2, 128, 64, dtype=torch.bfloat16), torch.zeros(1, 2, 128), torch.zeros(4, dtype=torch.int32)
huge = t[:, :1, :1].expand(1 << 20, 1 << 20, 1, 64)
forward = lambda q, k, v: host.forward(q, k, v, None, None, None, None, None, rec, 0, 0, 1.0, 0.0, 0.0, 1, 1, 0)
backward = lambda q, d_o: host.backward(q, t, t, t, f, d_o, None, None, None, rec, 0, 0, 0, 1.0, 0.0, True, 1, 1, 0, 0, 0)
for call in (lambda: forward(t, t, t[0]), lambda: backward(t, t[0]), lambda: forward(huge, t, t), lambda: backward(huge, t)):
  try:
    call()
  except RuntimeError as e:
    print("RuntimeError", str(e).splitlines()[0])
"""
  out = subprocess.run([sys.executable, "-c", program], cwd=ROOT, capture_output=True, text=True)
  assert out.returncode == 0, (out.returncode, out.stderr[-500:])
  assert out.stdout.count("RuntimeError") == 4 and out.stdout.count("rank 4") == 2, out.stdout
