"""Building the native code: from several processes, for several interpreters, and without a C++ compiler."""
import os
import subprocess
import sys
import sysconfig
import warnings

import pytest
import torch

from deepgengraph_b200 import _lib
from deepgengraph_b200 import attention as att
from deepgengraph_b200 import build as b

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_processes_that_build_at_once_do_not_share_a_file(tmp_path):
  # a compiler that writes its output in two halves; whatever is in place at any time has to be whole
  cxx = tmp_path / "cxx"
  cxx.write_text('#!/bin/sh\nwhile [ "$1" != "-o" ]; do shift; done\nprintf half > "$2"; sleep 0.5; printf half >> "$2"\n')
  cxx.chmod(0o755)
  target = tmp_path / "out.so"
  code = (f"import sys, time; sys.path.insert(0, {ROOT!r}); from deepgengraph_b200 import build as b; "
          f"b.torch_ext = lambda: {str(target)!r}; time.sleep(float(sys.argv[1])); b.build_torch(force=True); "
          f"assert open({str(target)!r}).read() == 'halfhalf'")
  env = dict(os.environ, CXX=str(cxx))
  runs = [subprocess.Popen([sys.executable, "-c", code, str(0.25 * i)], env=env) for i in range(3)]
  assert [p.wait(timeout=300) for p in runs] == [0, 0, 0]
  assert [f for f in os.listdir(tmp_path) if f.endswith(".tmp")] == []


def test_the_file_name_carries_what_the_binary_depends_on():
  name = os.path.basename(b.torch_ext())
  assert torch.__version__ in name and sysconfig.get_config_var("SOABI") in name


def _no_compiler(*args, **kw):
  raise RuntimeError("no compiler")


@pytest.mark.parametrize("present", ["missing", "of another interpreter"])
def test_operators_run_without_it(tmp_path, monkeypatch, present):
  path = tmp_path / "b200torch.so"
  if present != "missing":
    path.write_bytes(b"\x7fELF of another ABI")
  monkeypatch.setattr(b, "torch_ext", lambda: str(path))
  monkeypatch.setattr(b, "build_torch", _no_compiler)
  host = _lib._Host()
  monkeypatch.setattr(att, "host", host)
  x = torch.zeros(1, 4, 1, 128, dtype=torch.float16)
  with pytest.warns(RuntimeWarning, match="native host path"):
    with pytest.raises(RuntimeError, match="expected CUDA tensors"):   # the Python path, with its own checks
      att.attn_fwd(x, x, x)
  with warnings.catch_warnings():
    warnings.simplefilter("error")   # told once
    assert all(getattr(host, n)() is None for n in host.FUNCTIONS)


def test_the_cuda_library_builds_without_torch():
  code = ("import sys; sys.modules['torch'] = None; sys.path.insert(0, 'deepgengraph_b200'); import build; "
          "build.needs_build = lambda: False; assert build.build().endswith('libb200attn.so')")
  subprocess.run([sys.executable, "-c", code], cwd=ROOT, check=True)
