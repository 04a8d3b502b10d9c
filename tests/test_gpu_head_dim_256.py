"""Attention at head_dim 256 (csrc/attn_fwd_split.cuh): blocks of 128 keys whose halves go to two softmax warpgroups.  Edges of
tiles, blocks and halves, windows that leave a half or a whole first block without a visible key, maxima that grow (rescales decided by
one half only), NaN-free rows, both passes of the soft-cap, streams, graphs and the drained launch."""
import ctypes
import math

import pytest
import torch

from deepgengraph_b200 import _lib
from deepgengraph_b200 import attention as att
from oracle import reference_math as rm

pytestmark = pytest.mark.gpu


def _qkv(b, sq, skv, h, hk, dtype, seed, head_dim=256):
  g = torch.Generator().manual_seed(seed)
  return [torch.randn(b, s, n, head_dim, generator=g).to(dtype) for s, n in ((sq, h), (skv, hk), (skv, hk))]


def _check(q, k, v, device, window=-1, softcap=0.0):
  ref = rm.attention_ref(q, k, v, causal=True, window=window, softcap=softcap, want=("out", "lse2"))
  out, lse = att.attn_fwd_with_lse(q.to(device), k.to(device), v.to(device), causal=True, window=window, softcap=softcap)
  torch.testing.assert_close(out.float().cpu(), ref["out"], rtol=2e-2, atol=2e-2)
  torch.testing.assert_close(lse.cpu(), ref["lse2"], rtol=1e-3, atol=1e-3)


@pytest.mark.parametrize("q_len,extra", [(17, 0), (63, 1), (64, 64), (65, 63), (127, 1), (128, 0), (128, 128), (129, 127), (257, 64),
                                         (300, 333), (33, 1000)])
@pytest.mark.parametrize("softcap", [0.0, 30.0])
def test_edges_of_tiles_and_halves(cuda_device, q_len, extra, softcap):
  q, k, v = _qkv(1, q_len, q_len + extra, 2, 1, torch.bfloat16, q_len + extra)
  _check(q, k, v, cuda_device, softcap=softcap)


@pytest.mark.parametrize("window", [1, 2, 63, 64, 65, 128, 129, 300])
def test_windows(cuda_device, window):
  q, k, v = _qkv(1, 400, 467, 2, 2, torch.float16, window)
  _check(q, k, v, cuda_device, window=window)


@pytest.mark.parametrize("grow", [slice(0, 64), slice(64, 128), slice(0, 128)])
def test_maximum_that_grows_in_one_half(cuda_device, grow):
  q, k, v = _qkv(2, 700, 700, 2, 2, torch.bfloat16, 5)
  scale = torch.ones(700)
  for block in range(6):
    scale[128 * block:128 * block + 128][grow] = 0.3 + 1.5 * block
  _check(q, (k.float() * scale[None, :, None, None]).to(torch.bfloat16), v, cuda_device)


def test_more_tiles_than_sms(cuda_device):
  q, k, v = _qkv(3, 2000, 2000, 4, 2, torch.bfloat16, 9)
  ref = rm.attention_ref(q, k, v, causal=True, head_chunk=2)["out"]
  got = [att.attn_fwd(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device)) for _ in range(2)]
  assert torch.equal(got[0], got[1])
  torch.testing.assert_close(got[0].float().cpu(), ref, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("q_len,extra", [(17, 0), (40, 24), (64, 1), (64, 128), (150, 42), (192, 0), (193, 0), (320, 0), (65, 256)])
@pytest.mark.parametrize("softcap", [0.0, 30.0])
def test_half_blocks(cuda_device, q_len, extra, softcap):
  # a tile's last block has 64 keys (in the first, second or a later place) or, one key further, 128
  q, k, v = _qkv(2, q_len, q_len + extra, 2, 1, torch.float16, q_len + extra)
  _check(q, k, v, cuda_device, softcap=softcap)


def test_a_half_block_can_move_the_maximum(cuda_device):
  # the last 64 keys are the largest: the warpgroup that has none of them rescales its half of the output all the same
  q, k, v = _qkv(1, 64, 320, 2, 2, torch.bfloat16, 3)
  k[:, 256:] *= 6.0
  _check(q, k, v, cuda_device)


def test_tiles_of_one_block_repeat_their_bits(cuda_device):
  # every tile hands its maxima and its sums through the same words, one right after the other
  q, k, v = (t.to(cuda_device) for t in _qkv(8, 128, 128, 40, 40, torch.bfloat16, 11))
  want, want_lse = att.attn_fwd_with_lse(q, k, v, causal=True)
  ref = rm.attention_ref(q.cpu(), k.cpu(), v.cpu(), causal=True, want=("out", "lse2"))
  torch.testing.assert_close(want.float().cpu(), ref["out"], rtol=2e-2, atol=2e-2)
  torch.testing.assert_close(want_lse.cpu(), ref["lse2"], rtol=1e-3, atol=1e-3)
  for _ in range(50):
    out, lse = att.attn_fwd_with_lse(q, k, v, causal=True)
    assert torch.equal(out, want) and torch.equal(lse, want_lse)


@pytest.mark.parametrize("q_len,kv_len", [(17, 40), (64, 65), (130, 193), (130, 321), (333, 500)])
@pytest.mark.parametrize("softcap", [0.0, 30.0])
def test_without_the_causal_mask(cuda_device, q_len, kv_len, softcap):
  q, k, v = _qkv(2, q_len, kv_len, 4, 2, torch.bfloat16, q_len)
  ref = rm.attention_ref(q, k, v, causal=False, softcap=softcap, want=("out", "lse2"))
  out, lse = att.attn_fwd_with_lse(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device), causal=False, softcap=softcap)
  torch.testing.assert_close(out.float().cpu(), ref["out"], rtol=2e-2, atol=2e-2)
  torch.testing.assert_close(lse.cpu(), ref["lse2"], rtol=1e-3, atol=1e-3)


def _check_capped(q, k, v, device, softcap, window=-1):
  """Logits beyond the cap, so that warps take the pass with tanh.approx.  Its relative error is 2^-11: a capped logit is off by
  d = softcap * 2^-11 at most, the base-2 log-sum-exp by d * log2(e), and an output by d * sum_j p_j |v_j - out|, at most d times
  the square root of (sum_j p_j v_j^2 - out^2).  The other terms are those of `_check`."""
  kw = dict(causal=True, window=window, softcap=softcap)
  ref = rm.attention_ref(q, k, v, want=("out", "lse2"), **kw)
  spread = (rm.attention_ref(q, k, v.float() ** 2, **kw)["out"] - ref["out"] ** 2).clamp_min(0).sqrt()
  out, lse = att.attn_fwd_with_lse(q.to(device), k.to(device), v.to(device), **kw)
  d = softcap * 2.0 ** -11
  assert ((out.float().cpu() - ref["out"]).abs() <= d * spread + 2e-2 + 2e-2 * ref["out"].abs()).all()
  assert ((lse.cpu() - ref["lse2"]).abs() <= d * math.log2(math.e) + 1e-3 + 1e-3 * ref["lse2"].abs()).all()


@pytest.mark.parametrize("window", [-1, 1, 64, 65, 129, 300])
def test_logits_beyond_the_cap(cuda_device, window):
  q, k, v = _qkv(1, 400, 467, 2, 2, torch.bfloat16, 30 + window)
  _check_capped(30 * q, k, v, cuda_device, 30.0, window=window)


@pytest.mark.parametrize("grow", [slice(0, 64), slice(64, 128), slice(0, 128)])
def test_maximum_that_grows_under_a_cap(cuda_device, grow):
  q, k, v = _qkv(2, 700, 700, 2, 2, torch.bfloat16, 6)
  scale = torch.ones(700)
  for block in range(6):
    scale[128 * block:128 * block + 128][grow] = 0.3 + 3.0 * block
  _check_capped(q, (k.float() * scale[None, :, None, None]).to(torch.bfloat16), v, cuda_device, 30.0)


@pytest.mark.parametrize("head_dim", [128, 256])
def test_logits_all_below_minus_the_cap(cuda_device, head_dim):
  # the largest value is harmless: only the magnitude keeps a warp off the pass that is exact between -cap and cap
  q, k, v = _qkv(1, 300, 300, 2, 2, torch.bfloat16, 7, head_dim)
  q, k = 12 * q.abs(), -k.abs()
  logits = torch.einsum("bqhd,bkhd->bhqk", q.float(), k.float()) * head_dim ** -0.5
  assert logits.max() < -30.0
  _check_capped(q, k, v, cuda_device, 30.0)


def test_two_streams(cuda_device):
  q, k, v = (t.to(cuda_device) for t in _qkv(2, 1200, 1200, 16, 16, torch.bfloat16, 23))
  want = att.attn_fwd(q, k, v)
  torch.cuda.synchronize()
  streams, outs = [torch.cuda.Stream(device=cuda_device) for _ in range(2)], []
  for _ in range(4):
    for st in streams:
      with torch.cuda.stream(st):
        outs.append(att.attn_fwd(q, k, v))
  torch.cuda.synchronize()
  assert all(torch.equal(o, want) for o in outs)


def test_graph_replay(cuda_device):
  q, k, v = (t.to(cuda_device) for t in _qkv(2, 1200, 1200, 16, 8, torch.bfloat16, 24))
  want = att.attn_fwd(q, k, v, window=500)
  side = torch.cuda.Stream(device=cuda_device)
  side.wait_stream(torch.cuda.current_stream(cuda_device))
  with torch.cuda.stream(side):
    att.attn_fwd(q, k, v, window=500)
  torch.cuda.current_stream(cuda_device).wait_stream(side)
  graph = torch.cuda.CUDAGraph()
  with torch.cuda.graph(graph):
    outs = [att.attn_fwd(q, k, v, window=500) for _ in range(3)]
  for _ in range(3):
    for o in outs:
      o.fill_(float("nan"))
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in outs)


def test_a_launch_drains_while_the_status_word_is_set(cuda_device):
  lib, word = _lib.load(), ctypes.c_int(0)
  stream = torch.cuda.current_stream().cuda_stream
  lib.b200_selftest_bounded_wait(20, None, stream)
  torch.cuda.synchronize()
  q = torch.randn(1, 256, 2, 256, device=cuda_device, dtype=torch.bfloat16)
  out = torch.full_like(q, 7.0)
  assert lib.b200_attn_fwd(q.data_ptr(), q.data_ptr(), q.data_ptr(), out.data_ptr(), None, 1, 256, 256, 2, 2, 256, _lib.BF16, 1, 0, 0.0,
                           0.0625, stream) == 0
  torch.cuda.synchronize()
  assert torch.all(out == 7.0)
  assert lib.b200_device_status(ctypes.byref(word)) == 7
  ref = rm.attention_ref(q.cpu(), q.cpu(), q.cpu(), causal=True)["out"]
  torch.testing.assert_close(att.attn_fwd(q, q, q).float().cpu(), ref, rtol=2e-2, atol=2e-2)
  assert lib.b200_device_status(ctypes.byref(word)) == 0
