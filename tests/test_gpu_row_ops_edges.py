"""RMSNorm and the rotary embedding around the sizes where their launches change: rows of up to 128 / 256 / 512 / 1024 16-byte
vectors and beyond, up to and above 1024 rows, heads of a token shared out over several warps.  Tolerances: one rounding of
the tensor's type for 16 bits (the oracle rounds where the kernels round), sums of at most 8200 terms for fp32."""
import pytest
import torch

from deepgengraph_b200 import native_ops as ops
from oracle import reference_math as rm

pytestmark = pytest.mark.gpu
TOL = {torch.float32: dict(rtol=1e-5, atol=1e-5), torch.float16: dict(rtol=2e-3, atol=2e-3)}


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("vectors", [1, 128, 129, 256, 257, 512, 513, 1024, 1025])
@pytest.mark.parametrize("tokens", [1, 1025])
def test_norms(cuda_device, dtype, vectors, tokens):
  hidden = vectors * (16 // torch.empty(0, dtype=dtype).element_size())
  g = torch.Generator().manual_seed(vectors)
  x, r = (torch.randn(tokens, hidden, generator=g).to(dtype) for _ in range(2))
  w = (1 + 0.1 * torch.randn(hidden, generator=g)).to(dtype)
  out = torch.full_like(x, float("nan"), device=cuda_device)
  ops.rms_norm(out, x.to(cuda_device), w.to(cuda_device), 1e-6)
  torch.testing.assert_close(out.float().cpu(), rm.rms_norm_ref(x, w, 1e-6).float(), **TOL[dtype])
  ref_x, ref_r = rm.fused_add_rms_norm_ref(x, r, w, 1e-5)
  xd, rd = x.to(cuda_device), r.to(cuda_device)
  ops.fused_add_rms_norm(xd, rd, w.to(cuda_device), 1e-5)
  torch.testing.assert_close(rd.float().cpu(), ref_r.float(), **TOL[dtype])
  torch.testing.assert_close(xd.float().cpu(), ref_x.float(), **TOL[dtype])


@pytest.mark.parametrize("tokens,heads,kv_heads,head_dim", [(1, 1, 1, 64), (1, 40, 10, 128), (3, 33, 31, 128), (300, 16, 8, 256),
                                                            (1000, 17, 1, 128)])
def test_rotary_with_shared_out_heads(cuda_device, tokens, heads, kv_heads, head_dim):
  # every share of a token's heads gives what the token gives in a launch of many tokens, where a warp takes it whole
  g = torch.Generator().manual_seed(tokens)
  many = 148 * 16 + 1
  qkv = torch.randn(many, (heads + kv_heads) * head_dim, generator=g).to(torch.float16).to(cuda_device)
  pos = torch.randint(0, 8192, (many,), generator=g, dtype=torch.int32).to(cuda_device)
  few = qkv[:tokens].clone()
  split = heads * head_dim
  ops.rotary_embedding_online(pos, qkv[:, :split], qkv[:, split:], head_dim, 10000.0)
  ops.rotary_embedding_online(pos[:tokens], few[:, :split], few[:, split:], head_dim, 10000.0)
  assert torch.equal(few, qkv[:tokens])
