"""ctypes binding of libb200attn.so (the C ABI declared in include/b200attn.h).

The library is built in-tree by deepgengraph_b200/build.py.  There is no fallback: if the
shared object is missing and cannot be built, importing the ops raises.

`host` is the torch host path of the public operators (csrc/torch_binding.cpp): `host.attn_fwd(...)` and so on, each of
which returns None when the call is not the regular case and the Python operator has to take it from there.
"""
import ctypes
import importlib.machinery
import importlib.util
import os
import threading
import warnings

from . import build as _build

_LIB = None

F32, F16, BF16 = 0, 1, 2

STATUS_NAMES = {
    0: "ok", 1: "bad argument", 2: "unsupported dtype", 3: "misaligned pointer or stride",
    4: "unsupported shape", 5: "workspace missing or too small", 6: "CUDA call failed",
    7: "device-side wait expired",
}

_vp, _i, _i64, _f = ctypes.c_void_p, ctypes.c_int, ctypes.c_int64, ctypes.c_float

# name -> (restype, argtypes); mirrors include/b200attn.h one to one
SIGNATURES = {
    "b200_status_string": (ctypes.c_char_p, [_i]),
    "b200_last_cuda_error": (_i, []),
    "b200_abi_version": (_i, []),
    "b200_device_status": (_i, [ctypes.POINTER(_i)]),
    "b200_selftest_bounded_wait": (_i, [_i, _vp, _vp]),
    "b200_rms_norm": (_i, [_vp, _vp, _vp, _f, _i64, _i, _i, _vp]),
    "b200_fused_add_rms_norm": (_i, [_vp, _vp, _vp, _f, _i64, _i, _i, _vp]),
    "b200_silu_and_mul": (_i, [_vp, _vp, _i64, _i, _i, _vp]),
    "b200_gelu_tanh_and_mul": (_i, [_vp, _vp, _i64, _i, _i, _vp]),
    "b200_rotary_embedding_online": (_i, [_vp, _vp, _vp, _i64, _i, _i, _i, _i64, _i64, _f, _i, _vp]),
    "b200_attn_fwd": (_i, [_vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _i, _i, _i, _f, _f, _vp]),
    "b200_attn_fwd_strided": (_i, [_vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _i, _i64, _i64, _i64, _i64, _i64, _i64,
                                   _i, _i, _f, _f, _vp]),
    "b200_attn_score_workspace_bytes": (_i64, [_i, _i, _i, _i]),
    "b200_attn_score": (_i, [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _i64, _i, _i, _i, _i, _i, _i, _i, _i, _f, _f, _vp]),
    "b200_attn_score_gqa": (_i, [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i64, _i, _i, _i, _i, _i, _i, _i, _i, _i, _f, _f,
                                 _vp]),
    "b200_attn_kf_score_seeded": (_i, [_vp, _vp, _vp, ctypes.c_uint64, _vp, _vp, _vp, _i64, _i, _i, _i, _i, _i, _i, _i, _i, _f,
                                       _f, _vp]),
    "b200_kf_noise_fill": (_i, [_vp, ctypes.c_uint64, _i, _i, _i, _i, _vp]),
    "b200_attn_kf_score_gqa": (_i, [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _i64, _i, _i, _i, _i, _i, _i, _i, _i, _f, _f, _vp]),
    "b200_attn_score_static": (_i, [_vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _i, _i, _f, _f, _vp]),
    "b200_attn_corm": (_i, [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _i64, _i, _i, _i, _i, _i, _i, _i, _f, _vp]),
    "b200_avg_pool1d_f32": (_i, [_vp, _vp, _i64, _i, _i, _vp]),
    "b200_kv_evict_topk": (_i, [_vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _vp]),
    "b200_kv_evict_roco": (_i, [_vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _i, _i, _vp]),
    "b200_attn_kf_score": (_i, [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _i64, _i, _i, _i, _i, _i, _i, _i, _f, _f, _vp]),
}


def lib_path():
  return _build.LIB


def load():
  """Loads (building first if needed) the native library and declares its signatures."""
  global _LIB
  if _LIB is not None:
    return _LIB
  path = _build.LIB
  if _build.needs_build():
    try:
      _build.build()
    except Exception as e:  # a present library is still usable where no compiler is installed
      if not os.path.exists(path):
        raise RuntimeError(f"libb200attn.so is missing and could not be built: {e}") from e
  lib = ctypes.CDLL(path)
  for name, (res, args) in SIGNATURES.items():
    fn = getattr(lib, name)  # AttributeError here = header / library mismatch
    fn.restype = res
    fn.argtypes = args
  _LIB = lib
  return lib


class _Host:
  """The functions of the torch host path (b200torch.*.so), loaded -- built first if needed -- on the first use of any of
  them.  Where it can be neither built nor loaded there is one warning, and every function returns None: the operators then
  take their Python path, which needs the CUDA library only."""
  FUNCTIONS = ("attn_fwd", "attn_score", "attn_snapkv", "attn_corm", "attn_kf", "kv_evict", "norm", "act_and_mul", "rotary")
  _lock = threading.Lock()   # of the class: an attribute set in __init__ makes every later look-up of a function 20 ns slower

  def __getattr__(self, name):   # only reached while `name` is not set
    if name not in self.FUNCTIONS:
      raise AttributeError(name)
    load()      # the CUDA library it links against
    with self._lock:
      if name not in self.__dict__:
        try:
          self.__dict__.update(self._load())
        except Exception as e:   # noqa: BLE001 -- no compiler, no headers, no loadable file: whatever it is, the path is optional
          warnings.warn(f"the native host path of deepgengraph_b200 is not available ({type(e).__name__}: {e}); its operators "
                        "take several microseconds more of host time per call", RuntimeWarning, stacklevel=3)
          self.__dict__.update({n: _declined for n in self.FUNCTIONS})
    return self.__dict__[name]

  def _load(self):
    path = _build.torch_ext()
    if _build.needs_torch_build():
      try:
        _build.build_torch()
      except Exception:   # a present file is still usable where no compiler is installed
        if not os.path.exists(path):
          raise
    loader = importlib.machinery.ExtensionFileLoader("b200torch", path)
    mod = importlib.util.module_from_spec(importlib.util.spec_from_loader("b200torch", loader))
    loader.exec_module(mod)
    return {n: getattr(mod, n) for n in self.FUNCTIONS}


def _declined(*args):
  return None


host = _Host()


class B200Error(RuntimeError):
  def __init__(self, status, where):
    self.status = status
    lib = load()
    detail = ""
    if status == 6:
      detail = f" (cudaError {lib.b200_last_cuda_error()})"
    super().__init__(f"{where}: {STATUS_NAMES.get(status, status)}{detail}")


def check(status, where):
  if status != 0:
    raise B200Error(status, where)
