"""Builds the native code in-tree, under deepgengraph_b200/csrc/:

  libb200attn.so   the CUDA library (sm_100a only): one translation unit (b200attn.cu) compiled with nvcc; it links only the
                   CUDA runtime (the driver's tensor-map encoder is looked up at run time), so it can be loaded with
                   ctypes from any host language
  b200torch.<torch version>.<ABI tags>.so
                   the torch host path of the public operators (torch_binding.cpp), linked against the library; optional: the
                   operators run without it, with a slower host path
"""
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(CSRC, "libb200attn.so")
SOURCES = ["b200attn.cu"]
HEADER = os.path.join("..", "..", "include", "b200attn.h")
DEPS = ["b200attn.cu", "common.cuh", "elementwise.cuh", "attn_fwd.cuh", "attn_fwd_persist.cuh", "attn_fwd_split.cuh", "attn_pair.h",
        "attn_decode.cuh", "attn_decode_plan.h", "attn_sweep.cuh", "kv_evict.cuh", HEADER]
TORCH_DEPS = ["torch_binding.cpp", HEADER]


def _nvcc():
  for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
    if cand and os.path.exists(cand):
      return cand
  raise RuntimeError("nvcc not found (set NVCC or install the CUDA toolkit)")


def _older(target, deps):
  if not os.path.exists(target):
    return True
  t = os.path.getmtime(target)
  return any(os.path.getmtime(os.path.join(CSRC, d)) > t for d in deps)


def needs_build():
  return _older(LIB, DEPS)


def torch_ext():
  """Path of the torch host path for this interpreter: the name carries what its binary interface depends on, so that another
  torch or Python finds no file and builds its own."""
  import torch
  abi = int(torch._C._GLIBCXX_USE_CXX11_ABI)
  return os.path.join(CSRC, f"b200torch.{torch.__version__}.cxx11abi{abi}.{sysconfig.get_config_var('SOABI')}.so")


def needs_torch_build():
  return _older(torch_ext(), TORCH_DEPS)


def _temporary(target):
  return f"{target}.{os.getpid()}.tmp"   # of this process: several ranks may build at the same time


def _run(cmd, target, verbose):
  """Runs `cmd`, which writes _temporary(target), and puts the result in place in one step."""
  tmp = _temporary(target)
  try:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
      sys.stderr.write(res.stdout + res.stderr)
      raise RuntimeError(f"{os.path.basename(cmd[0])} failed building {os.path.basename(target)}")
    if verbose:
      sys.stderr.write(res.stdout + res.stderr)
    os.replace(tmp, target)
  finally:
    if os.path.exists(tmp):
      os.remove(tmp)


def build(force=False, verbose=False):
  """Compile the CUDA library if it is missing or older than its sources. Returns its path."""
  if not force and not needs_build():
    return LIB
  cmd = [
      _nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
      "-shared", "-Xcompiler", "-fPIC", "--use_fast_math", "-Xptxas", "-v" if verbose else "-O3",
      "-o", _temporary(LIB),
  ] + [os.path.join(CSRC, s) for s in SOURCES] + ["-lcudart"]
  _run(cmd, LIB, verbose)
  return LIB


def build_torch(force=False, verbose=False):
  """The torch host path, after the library it is linked against; needs only a C++ compiler and torch's headers."""
  target = torch_ext()
  if not (force or needs_torch_build()):
    return target
  import torch
  from torch.utils import cpp_extension
  cuda_home = os.path.dirname(os.path.dirname(_nvcc()))
  includes = cpp_extension.include_paths() + [os.path.join(cuda_home, "include"), sysconfig.get_paths()["include"]]
  torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
  cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
         f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
  cmd += ["-isystem" + p for p in includes]
  cmd += ["-o", _temporary(target), os.path.join(CSRC, "torch_binding.cpp"), "-L" + torch_lib, "-L" + CSRC,
          "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10", "-l:libb200attn.so", "-Wl,-rpath,$ORIGIN"]
  _run(cmd, target, verbose)
  return target


if __name__ == "__main__":
  for step in (build, build_torch):
    print(step(force="--force" in sys.argv, verbose="-v" in sys.argv))
