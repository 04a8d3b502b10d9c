"""Failure detection without a GPU fault: a device-side wait that nothing will ever satisfy runs out after its
limit, the kernel returns normally, the host reads the recorded status, and the device keeps working."""
import ctypes

import pytest
import torch

from deepgengraph_b200 import _lib
from deepgengraph_b200 import attention as att

pytestmark = pytest.mark.gpu


def test_expired_wait_is_reported_and_the_device_stays_usable(cuda_device):
  lib = _lib.load()
  word = ctypes.c_int(0)
  assert lib.b200_device_status(ctypes.byref(word)) == 0 and word.value == 0
  gave_up = torch.zeros(1, dtype=torch.int32, device=cuda_device)
  assert lib.b200_selftest_bounded_wait(50, gave_up.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
  st = lib.b200_device_status(ctypes.byref(word))          # synchronises
  assert st == 7 and (word.value & 0xff) == 17             # B200_ERR_DEVICE_TIMEOUT, code WAIT_SELFTEST
  assert gave_up.item() == 1
  # the word was cleared by the read, and kernels run normally afterwards
  assert lib.b200_device_status(ctypes.byref(word)) == 0 and word.value == 0
  q = torch.randn(1, 256, 2, 128, device=cuda_device, dtype=torch.bfloat16)
  out = att.attn_fwd(q, q, q)
  assert torch.isfinite(out.float()).all()
  assert lib.b200_device_status(ctypes.byref(word)) == 0 and word.value == 0


def test_launches_drain_while_the_status_word_is_set(cuda_device):
  # a kernel that follows an expired wait returns at once (its output stays untouched) until the host has read
  # and cleared the status word
  lib = _lib.load()
  word = ctypes.c_int(0)
  lib.b200_selftest_bounded_wait(20, None, torch.cuda.current_stream().cuda_stream)
  torch.cuda.synchronize()
  q = torch.randn(1, 256, 2, 128, device=cuda_device, dtype=torch.bfloat16)
  out = torch.full_like(q, 7.0)
  st = lib.b200_attn_fwd(q.data_ptr(), q.data_ptr(), q.data_ptr(), out.data_ptr(), None, 1, 256, 256, 2, 2, 128,
                         _lib.BF16, 1, 0, 0.0, 0.088, torch.cuda.current_stream().cuda_stream)
  assert st == 0
  torch.cuda.synchronize()
  assert torch.all(out == 7.0)
  assert lib.b200_device_status(ctypes.byref(word)) == 7
  ok = att.attn_fwd(q, q, q)
  assert torch.isfinite(ok.float()).all() and not torch.all(ok == 7.0)
  assert lib.b200_device_status(ctypes.byref(word)) == 0


def _score_calls(B, S, H, Hk, kinds):
  g = torch.Generator().manual_seed(S)
  q, k, v = (torch.randn(B, S, h, 128, generator=g).to(torch.bfloat16).cuda() for h in (H, Hk, Hk))
  noise = torch.rand(B, H, S, S, device="cuda") + 0.1 if "keyformer" in kinds else None
  lib, scale, stream = _lib.load(), 128 ** -0.5, torch.cuda.current_stream().cuda_stream
  ws = torch.zeros(lib.b200_attn_score_workspace_bytes(B, S, S, H), dtype=torch.uint8, device="cuda")
  outputs = [torch.empty_like(q), torch.empty(B, Hk, S, device="cuda"), torch.empty(B, Hk, S, device="cuda")]
  out, score, score_sq = (t.data_ptr() for t in outputs)
  head, tail = (q.data_ptr(), k.data_ptr(), v.data_ptr()), (ws.data_ptr(), ws.numel(), B, S, S, H)

  def scores(sq, cap):
    return lib.b200_attn_score_gqa(*head, out, score, sq, None, *tail, Hk, 128, _lib.BF16, 1, 0, cap, scale, stream)

  calls = {
      "sums": lambda: scores(None, 0.0), "squares": lambda: scores(score_sq, 0.0), "capped": lambda: scores(score_sq, 50.0),
      "keyformer": lambda: lib.b200_attn_kf_score_gqa(*head, noise.data_ptr(), out, score, *tail, Hk, 128, _lib.BF16, 1, 1.5, scale, stream),
      "seeded": lambda: lib.b200_attn_kf_score_seeded(*head, 5, out, score, *tail, Hk, 128, _lib.BF16, 1, 1.5, scale, stream),
  }
  inputs = (q, k, v, noise, ws)   # (the calls hold addresses only)
  return [(kind, calls[kind], outputs, inputs) for kind in kinds]


def _set_status_word():
  _lib.load().b200_selftest_bounded_wait(20, None, torch.cuda.current_stream().cuda_stream)
  torch.cuda.synchronize()


@pytest.mark.parametrize("S", [128, 1500])   # fewer and more blocks than the sweep's ring has stages
@pytest.mark.parametrize("H,Hk,kinds", [(4, 4, ("sums", "squares", "capped", "keyformer", "seeded")), (4, 2, ("squares", "capped"))])
def test_score_launches_drain_while_the_status_word_is_set(cuda_device, S, H, Hk, kinds):
  word = ctypes.c_int(0)
  for kind, call, outputs, _inputs in _score_calls(2, S, H, Hk, kinds):   # (one partial sum per key: the sweep writes the result itself)
    def run():
      for t in outputs:
        t.fill_(7.0)
      assert call() == 0
      torch.cuda.synchronize()
      return [t.clone() for t in outputs]
    want = run()
    _set_status_word()
    assert all(torch.all(t == 7.0) for t in run()), kind
    assert _lib.load().b200_device_status(ctypes.byref(word)) == 7 and (word.value & 0xff) == 17   # no other wait ran out
    assert all(torch.equal(a, b) for a, b in zip(run(), want)), kind
    assert _lib.load().b200_device_status(ctypes.byref(word)) == 0


def test_every_wave_of_a_score_launch_drains_at_once(cuda_device):
  # The producer of the plain column sums starts to load before it knows of the status word and has to be told to stop; with a soft-cap
  # nothing starts before.  14 waves of CTAs: 10 us for each would be 140 us more (measured: 27 us more).
  times = {}
  for kind, call, *_tensors in _score_calls(16, 512, 64, 64, ("sums", "capped")):
    assert call() == 0
    _set_status_word()
    start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    for _ in range(5):
      start.record()
      assert call() == 0
      end.record()
      torch.cuda.synchronize()
      times[kind] = min(times.get(kind, 1e9), start.elapsed_time(end) * 1e3)
    _lib.load().b200_device_status(ctypes.byref(ctypes.c_int(0)))
  assert times["sums"] < times["capped"] + 140, times
