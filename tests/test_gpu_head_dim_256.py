"""Attention at head_dim 256 (csrc/attn_fwd_split.cuh): blocks of 128 keys whose halves go to two softmax warpgroups.  Edges of
tiles, blocks and halves, windows that leave a half or a whole first block without a visible key, maxima that grow (rescales decided by
one half only), and NaN-free rows."""
import pytest
import torch

from deepgengraph_b200 import attention as att
from oracle import reference_math as rm

pytestmark = pytest.mark.gpu


def _qkv(b, sq, skv, h, hk, dtype, seed):
  g = torch.Generator().manual_seed(seed)
  return [torch.randn(b, s, n, 256, generator=g).to(dtype) for s, n in ((sq, h), (skv, hk), (skv, hk))]


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
