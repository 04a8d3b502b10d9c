"""Calls that reach the native host path of the public operators in other ways than a plain call with regular arguments."""
import math
import threading

import pytest
import torch
import torch.autograd.forward_ad as fwAD
from torch.utils._python_dispatch import TorchDispatchMode

from deepgengraph_b200 import _lib
from deepgengraph_b200 import attention as att
from deepgengraph_b200 import native_ops as ops

pytestmark = pytest.mark.gpu


def _rand(*shape, dtype=torch.bfloat16, seed=0):
  return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(dtype).cuda()


@pytest.mark.parametrize("fn", [att.attn_fwd, att.attn_fwd_with_lse, att.attn_score_fwd, att.attn_kf_fwd, att.attn_snapkv_fwd,
                                att.attn_corm_fwd])
def test_a_scale_that_is_no_number_is_refused(cuda_device, fn):
  q = _rand(1, 64, 2, 128)
  with pytest.raises(_lib.B200Error):
    fn(q, q, q, scale=math.nan)


def test_the_current_stream_is_used(cuda_device):
  q, k, v = _rand(2, 256, 4, 128), _rand(2, 256, 2, 128, seed=1), _rand(2, 256, 2, 128, seed=2)
  want = att.attn_score_fwd(q, k, v, want_sq=True)
  side = torch.cuda.Stream()
  side.wait_stream(torch.cuda.current_stream())
  with torch.cuda.stream(side):
    torch.cuda._sleep(20_000_000)      # about 10 ms: on another stream the operator would read `late` before it is written
    late = torch.zeros_like(q)
    late.copy_(q)
    got = att.attn_score_fwd(late, k, v, want_sq=True)
  side.synchronize()
  assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_threads_with_streams_of_their_own(cuda_device):
  args = [[_rand(1, 150 + 10 * i, 4, 128, seed=3 * i + j) for j in range(3)] for i in range(4)]
  want = [att.attn_score_fwd(*a) for a in args]
  torch.cuda.synchronize()
  bad = []

  def work(i):
    with torch.cuda.stream(torch.cuda.Stream()):
      for _ in range(20):
        got = att.attn_score_fwd(*args[i])
        torch.cuda.current_stream().synchronize()
        if not all(torch.equal(a, b) for a, b in zip(got, want[i])):
          bad.append(i)

  threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
  for t in threads:
    t.start()
  for t in threads:
    t.join()
  assert not bad


def test_batched_tensors_of_vmap_are_declined(cuda_device):
  q, k, v = _rand(2, 1, 64, 2, 128), _rand(1, 64, 2, 128, seed=1), _rand(1, 64, 2, 128, seed=2)
  taken = []

  def call(x):
    taken.append(_lib.host.attn_fwd(x, k, v, True, -1, 0.0, None, False))
    return att.attn_fwd(x, k, v)

  with pytest.raises(RuntimeError):    # the Python path: such a tensor has no address
    torch.vmap(call)(q)
  assert taken == [None]


def test_a_dispatch_mode_sees_the_python_path(cuda_device):
  q, k, v = _rand(1, 64, 2, 128), _rand(1, 64, 2, 128, seed=1), _rand(1, 64, 2, 128, seed=2)
  want = att.attn_fwd(q, k, v)
  seen = []

  class Mode(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
      seen.append(str(func))
      return func(*args, **(kwargs or {}))

  with Mode():
    assert _lib.host.attn_fwd(q, k, v, True, -1, 0.0, None, False) is None
    got = att.attn_fwd(q, k, v)
  assert any("empty" in f for f in seen) and torch.equal(got, want)


@pytest.mark.parametrize("kind", ["requires_grad", "dual"])
def test_tensors_under_differentiation_give_plain_results(cuda_device, kind):
  q, k, v = _rand(1, 64, 2, 128), _rand(1, 64, 2, 128, seed=1), _rand(1, 64, 2, 128, seed=2)
  want = att.attn_fwd(q, k, v)
  with fwAD.dual_level():
    x = fwAD.make_dual(q, torch.ones_like(q)) if kind == "dual" else q.clone().requires_grad_()
    got, python = att.attn_fwd(x, k, v), att._attn_fwd_impl(x, k, v, True, -1, 0.0, None)
    for out in (got, python):
      assert not out.requires_grad and fwAD.unpack_dual(out).tangent is None and torch.equal(out, want)


@pytest.mark.parametrize("kv_heads", [4, 2])
def test_keyformer_with_a_noise_tensor_matches_the_python_path(cuda_device, kv_heads):
  q, k, v = _rand(2, 200, 4, 128), _rand(2, 200, kv_heads, 128, seed=1), _rand(2, 200, kv_heads, 128, seed=2)
  noise = _rand(2, 4, 200, 200, dtype=torch.float32, seed=3).abs() + 1e-3
  got = _lib.host.attn_kf(q, k, v, noise, 0, 1.5, True, None)
  assert all(torch.equal(a, b) for a, b in zip(got, att._attn_kf_impl(q, k, v, noise, 1.5, True, None)))


def _same(got, want, what):
  bad = (got != want).flatten().nonzero().flatten()
  assert bad.numel() == 0, f"{what}: {bad.numel()} of {want.numel()} elements differ, flat indices {bad[0].item()} to {bad[-1].item()}"


def test_library_launches_with_other_kernels_between_them(cuda_device):
  # every launch may start while its predecessor drains: neither side of a foreign kernel may be overtaken
  T, H, D = 700, 8, 128
  x, w = _rand(T, H * D, dtype=torch.float16), _rand(H * D, dtype=torch.float16, seed=1)
  proj = _rand(H * D, 3 * H * D, dtype=torch.float16, seed=2) * 0.03
  pos = torch.arange(T, device="cuda", dtype=torch.int32)

  def chain(between):
    h = torch.empty_like(x)
    ops.rms_norm(h, x, w, 1e-6)
    between()
    qkv = h @ proj
    between()
    q, k, v = qkv[:, :H * D], qkv[:, H * D:2 * H * D], qkv[:, 2 * H * D:]
    ops.rotary_embedding_online(pos, q, k, D, 10000.0)
    between()
    out, score, score_sq = att.attn_score_fwd(*(t.unflatten(-1, (H, D))[None].contiguous() for t in (q, k, v)), want_sq=True)
    between()
    last = att.attn_fwd(out[:, -4:].contiguous(), q.unflatten(-1, (H, D))[None], v.unflatten(-1, (H, D))[None])
    cache = att.kv_evict_roco(score, score_sq, out, out, T, 100, 16)
    act = torch.empty(T, 3 * H * D // 2, device="cuda", dtype=torch.float16)
    ops.silu_and_mul(act, qkv)
    return {"h": h, "qkv": qkv, "out": out, "score": score, "score_sq": score_sq, "last": last, "cache": cache, "act": act}

  want = chain(torch.cuda.synchronize)
  for n in range(20):
    got = chain(lambda: None)
    wrong = [name for name in want if not torch.equal(got[name], want[name])]
    for name in wrong:
      _same(got[name], want[name], f"pass {n}: {wrong}, {name}")
    del got   # the next pass takes the same memory


@pytest.mark.parametrize("kind", ["scores", "capped_scores", "keyformer"])
def test_launches_behind_ordinary_kernels_on_the_same_buffers(cuda_device, kind):
  # q, k, v and the noise are rewritten, and the output buffer is read and overwritten, by ordinary kernels right before the call
  B, S, H, D = 2, 700, 4, 128
  lib, stream = _lib.load(), torch.cuda.current_stream().cuda_stream
  sets = [[_rand(B, S, H, D, seed=10 * i + j) for j in range(3)] + [_rand(B, H, S, S, dtype=torch.float32, seed=10 * i + 3).abs() + 1e-3]
          for i in range(2)]
  ins = [torch.empty_like(t) for t in sets[0]]
  ws = torch.empty(lib.b200_attn_score_workspace_bytes(B, S, S, H), dtype=torch.uint8, device="cuda")
  out, score, seen = torch.empty_like(ins[0]), torch.empty(B, H, S, device="cuda"), torch.zeros_like(ins[0])

  def call(src, between):
    for a, b in zip(ins, src):
      a.copy_(b)
    seen.add_(out)
    out.fill_(7.0)
    score.fill_(7.0)
    between()
    args = [t.data_ptr() for t in ins]
    if kind == "keyformer":
      st = lib.b200_attn_kf_score(*args, out.data_ptr(), score.data_ptr(), ws.data_ptr(), ws.numel(), B, S, S, H, D, _lib.BF16, 1, 1.5,
                                  D ** -0.5, stream)
    else:
      st = lib.b200_attn_score(*args[:3], out.data_ptr(), score.data_ptr(), None, ws.data_ptr(), ws.numel(), B, S, S, H, D, _lib.BF16, 1, 0,
                               50.0 if kind == "capped_scores" else 0.0, D ** -0.5, stream)
    assert st == 0
    between()
    return out.clone(), score.clone()

  want = [call(src, torch.cuda.synchronize) for src in sets]
  got = [call(sets[n % 2], lambda: None) for n in range(40)]
  for n, pair in enumerate(got):
    for what, a, b in zip(("out", "score"), pair, want[n % 2]):
      _same(a, b, f"pass {n}: {what}")
