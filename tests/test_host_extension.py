"""Building the native code: from several processes, for several interpreters."""
import os
import subprocess
import sys
import sysconfig

import torch

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
