"""Attention for a few query rows (csrc/attn_decode.cuh): keys and values that are not finite, launches inside a captured graph,
and what a unit's result keeps when the problem is cut up."""
import pytest
import torch

from deepgengraph_b200 import attention as att
from deepgengraph_b200 import sharding as sh
from oracle import reference_math as rm

pytestmark = pytest.mark.gpu


def _rand(*shape, seed=0, dtype=torch.bfloat16):
  return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(dtype)


@pytest.mark.parametrize("what", ["logit -inf", "value inf", "key nan", "value nan"])
@pytest.mark.parametrize("Skv,kv_heads,at", [(40, 2, 3), (3000, 2, 2999), (700, 4, 350)])
def test_values_that_are_not_finite(cuda_device, what, Skv, kv_heads, at):
  q, k, v = _rand(1, 2, 4, 128).abs(), _rand(1, Skv, kv_heads, 128, seed=1), _rand(1, Skv, kv_heads, 128, seed=2)
  if what == "logit -inf":
    k[0, at, 0] = -3e38
  elif what == "value inf":
    v[0, at, 0, 5] = float("inf")
  elif what == "key nan":
    k[0, at, 0, 7] = float("nan")
  else:
    v[0, at, 0, 5] = float("nan")
  ref = rm.attention_ref(q, k, v, want=("out",))["out"]
  out = att.attn_fwd(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device)).float().cpu()
  if at == Skv - 1:   # query 0 does not see the last key: it is finite in the oracle only (the kernel computes 0 * value)
    ref, out = ref[:, 1:], out[:, 1:]
  # the bound of the finite case: P and the output rounded to bf16, a weighted mean of N(0, 1) values
  torch.testing.assert_close(out, ref, rtol=0, atol=2 * 2 ** -9 * 4.5, equal_nan=True)


def test_inside_a_captured_graph(cuda_device):
  q, cache = _rand(2, 1, 8, 128).to(cuda_device), _rand(2, 2, 900, 2, 128, seed=1).to(cuda_device)
  want = att.attn_fwd(q, cache[:, 0], cache[:, 1])
  graph = torch.cuda.CUDAGraph()
  with torch.cuda.graph(graph):
    out = att.attn_fwd(q, cache[:, 0], cache[:, 1])
    again = att.attn_fwd(out, cache[:, 0], cache[:, 1])
  for _ in range(3):
    out.zero_()
    graph.replay()
    assert torch.equal(out, want)
  assert torch.equal(again, att.attn_fwd(want, cache[:, 0], cache[:, 1]))
  new = _rand(2, 1, 8, 128, seed=5).to(cuda_device)
  q.copy_(new)
  graph.replay()
  assert torch.equal(out, att.attn_fwd(new, cache[:, 0], cache[:, 1]))


@pytest.mark.parametrize("q_len,kv_len,kv_heads", [(1040, 1536, 2), (260, 700, 2), (130, 130, 2)])
def test_row_shards_with_a_short_tail_have_the_bits_of_the_full_problem(cuda_device, q_len, kv_len, kv_heads):
  q, k, v = (t.to(cuda_device) for t in (_rand(1, q_len, 4, 128), _rand(1, kv_len, kv_heads, 128, seed=1),
                                         _rand(1, kv_len, kv_heads, 128, seed=2)))
  full, got = att.attn_fwd(q, k, v), torch.full_like(q, float("nan"))
  world = 9 * kv_heads
  for rank in range(world):
    for pc, out in sh.run_row_sharded(att.attn_fwd, q, k, v, world, rank):
      got[pc.b, pc.r0:pc.r1, pc.hk * 2:pc.hk * 2 + 2] = out[0]
  assert torch.equal(got, full)


def test_head_shards_agree_to_the_rounding_of_the_probabilities(cuda_device):
  # the split of a unit's keys, and with it the last bits, follows the number of units in the launch: 64 here, 8 in a shard.
  # A probability is rounded to bf16 against another running maximum, the output once: both within 2^-9 of a mean of N(0, 1)
  # values whose weights add up to 1
  q, k, v = (t.to(cuda_device) for t in (_rand(8, 1, 32, 128), _rand(8, 4096, 8, 128, seed=1), _rand(8, 4096, 8, 128, seed=2)))
  full, full_lse = att.attn_fwd_with_lse(q, k, v)
  for rank in range(8):
    for piece, (out, lse) in sh.run_sharded(att.attn_fwd_with_lse, q, k, v, 8, rank, dense=False):
      rows = slice(piece.hk_lo * 4, piece.hk_hi * 4)
      torch.testing.assert_close(out[0].float(), full[piece.b, :, rows].float(), rtol=0, atol=2 * 2 ** -9 * 4.5)
      torch.testing.assert_close(lse[0], full_lse[piece.b, rows], rtol=0, atol=2e-5)


def test_a_very_large_batch_goes_to_the_kernel_of_its_shards(cuda_device):
  # 90000 units in one launch and 300 in another, both of one CTA per unit: the same kernel, the same bits
  q, k, v = (t.to(cuda_device) for t in (_rand(300, 1, 300, 128), _rand(300, 40, 300, 128, seed=1), _rand(300, 40, 300, 128, seed=2)))
  full = att.attn_fwd(q, k, v)
  for b in (0, 299):
    assert torch.equal(full[b:b + 1], att.attn_fwd(q[b:b + 1], k[b:b + 1], v[b:b + 1]))
