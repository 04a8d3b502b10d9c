"""Tensor maps are kept by layout and take the address of every call: the same layout on other buffers, more layouts than the
table holds, views of one buffer, several threads."""
import threading

import pytest
import torch

from deepgengraph_b200 import attention as att
from oracle import reference_math as rm

pytestmark = pytest.mark.gpu


def _qkv(seq, seed, heads=2):
  g = torch.Generator().manual_seed(seed)
  return [torch.randn(1, seq, heads, 128, generator=g).to(torch.bfloat16) for _ in range(3)]


def _close(got, q, k, v):
  ref = rm.attention_ref(q, k, v, want=("out", "colsum"))
  torch.testing.assert_close(got[0].float().cpu(), ref["out"], rtol=2e-2, atol=2e-2)
  torch.testing.assert_close(got[1].cpu(), ref["colsum"], rtol=1e-3, atol=1e-5)


def test_one_layout_on_many_buffers(cuda_device):
  inputs = [_qkv(150, s) for s in range(6)]
  on_gpu = [[t.to(cuda_device) for t in i] for i in inputs]
  results = [att.attn_score_fwd(*i) for i in on_gpu for _ in range(2)]
  for n, got in enumerate(results):
    _close(got, *inputs[n // 2])


def test_more_layouts_than_are_kept(cuda_device):
  first = {}
  for sweep in range(2):
    for seq in range(20, 20 + 3 * 90, 3):
      q, k, v = (t.to(cuda_device) for t in _qkv(seq, seq))
      out, score = att.attn_score_fwd(q, k, v)
      if sweep == 0:
        first[seq] = (out, score)
      else:
        assert torch.equal(out, first[seq][0]) and torch.equal(score, first[seq][1])
  _close(first[101], *_qkv(101, 101))


def test_views_that_share_layout_and_buffer(cuda_device):
  qkv = torch.randn(1, 140, 9, 128, generator=torch.Generator().manual_seed(3)).to(torch.bfloat16)
  d = qkv.to(cuda_device)
  for h in range(3):
    views = [qkv[:, :, 3 * i + h:3 * i + h + 1] for i in range(3)]
    got = att.attn_fwd(*(d[:, :, 3 * i + h:3 * i + h + 1] for i in range(3)))
    ref = rm.attention_ref(*views, want=("out",))["out"]
    torch.testing.assert_close(got.float().cpu(), ref, rtol=2e-2, atol=2e-2)


def test_threads(cuda_device):
  inputs = [_qkv(150, s) for s in range(4)]
  results = [None] * 4

  def work(i):
    mine = [t.to(cuda_device) for t in inputs[i]]
    for _ in range(10):
      results[i] = att.attn_score_fwd(*mine)
    torch.cuda.synchronize()

  threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
  for t in threads:
    t.start()
  for t in threads:
    t.join()
  for i in range(4):
    _close(results[i], *inputs[i])
