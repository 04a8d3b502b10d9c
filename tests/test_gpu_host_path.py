"""The native host path of the public operators (csrc/torch_binding.cpp) against the Python implementations it stands in for:
the same bits where it takes a call, and None -- the Python path with its checks -- where it does not."""
import pytest
import torch

from deepgengraph_b200 import _lib
from deepgengraph_b200 import attention as att
from deepgengraph_b200 import native_ops as ops

pytestmark = pytest.mark.gpu


def _rand(*shape, dtype=torch.bfloat16, seed=0):
  return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(dtype).cuda()


@pytest.mark.parametrize("layout", ["dense", "qkv", "cache"])
def test_attention_calls_match_the_python_path(cuda_device, layout):
  B, S, H, Hk, D = 2, 200, 4, 2, 128
  if layout == "qkv":
    qkv = _rand(B, S, (H + 2 * Hk) * D)
    q, k, v = (t.unflatten(-1, (-1, D)) for t in qkv.split([H * D, Hk * D, Hk * D], dim=-1))
  else:
    cache = _rand(B, 2, S, Hk, D)
    q, k, v = _rand(B, S, H, D, seed=1), cache[:, 0], cache[:, 1]
    if layout == "dense":
      k, v = k.contiguous(), v.contiguous()
  got = _lib.host.attn_fwd(q, k, v, True, 70, 30.0, None, True)
  want = att._attn_fwd_impl(q, k, v, True, 70, 30.0, None, want_lse=True)
  assert all(torch.equal(a, b) for a, b in zip(got, want))
  if layout != "dense":     # the score variants take dense tensors only
    assert _lib.host.attn_score(q, k, v, True, True, -1, 0.0, None) is None
    return
  got = _lib.host.attn_score(q, k, v, True, True, -1, 0.0, None)
  assert all(torch.equal(a, b) for a, b in zip(got, att._attn_score_impl(q, k, v, True, True, -1, 0.0, None)))
  for mine, theirs in ((_lib.host.attn_snapkv(q, k, v, 5, True, None), att._attn_snapkv_impl(q, k, v, 5, True, None)),
                       (_lib.host.attn_corm(q, k, v, True, None), att._attn_corm_impl(q, k, v, True, None)),
                       (_lib.host.attn_kf(q, k, v, None, 2**64 - 3, 1.5, True, None),
                        att._attn_kf_seeded_impl(q, k, v, 2**64 - 3, 1.5, True, None))):
    assert all(torch.equal(a, b) and a.dtype == b.dtype for a, b in zip(mine, theirs))


def test_irregular_calls_are_left_to_the_python_path(cuda_device):
  q = _rand(1, 64, 2, 128)
  host = _lib.host
  assert host.attn_fwd(q, q.cpu(), q, True, -1, 0.0, None, False) is None
  assert host.attn_fwd(q, q.half(), q, True, -1, 0.0, None, False) is None
  assert host.attn_fwd(q, q[:, :, :1], q, True, -1, 0.0, None, False) is None
  assert host.attn_fwd(q[:0], q[:0], q[:0], True, -1, 0.0, None, False) is None
  assert host.attn_fwd(q, q, q, True, 2**40, 0.0, None, False) is None
  assert host.attn_fwd(q, q, q, 1, -1, 0.0, None, False) is None
  assert host.norm(q, q, None, q, 1e-6) is None                       # weight of another size
  assert host.act_and_mul(q, q, False) is None
  assert host.rotary(torch.zeros(64, device="cuda"), q[0].flatten(1), q[0].flatten(1), 128, 1e4) is None
  assert host.kv_evict(_rand(1, 2, 64, dtype=torch.float32), None, q, q, 1, 65, 0, True) is None
  with pytest.raises(ValueError):
    ops.silu_and_mul(q, q)
  with pytest.raises(ValueError):
    ops.rms_norm(q, q, q, 1e-6)
