"""Attention for a few query rows (csrc/attn_decode.cuh) against the oracle: row counts around the 16-row tile, key counts
around the 16-key tiles and the split over CTAs, grouped heads, cache views, windows, soft-cap."""
import pytest
import torch

from deepgengraph_b200 import attention as att
from oracle import reference_math as rm

pytestmark = pytest.mark.gpu
# P and the output are rounded to the input type (unit round-off 2^-9 and 2^-11): a weighted mean of N(0, 1) values differs by
# at most 2 x the round-off x max |v| (4.5 at these sizes)
TOL = {torch.bfloat16: dict(rtol=0, atol=2 * 2 ** -9 * 4.5), torch.float16: dict(rtol=0, atol=2 * 2 ** -11 * 4.5)}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,Sq,Skv,H,Hk,D,opt", [
    (1, 1, 1, 1, 1, 128, {}),
    (2, 1, 17, 4, 4, 128, {}),                               # one key past a tile
    (1, 16, 16, 2, 2, 128, {}),                              # 16 rows, the most that one tile takes
    (3, 4, 500, 12, 3, 128, {}),                             # 4 queries x 4 heads = 16 rows, ragged keys
    (1, 3, 1031, 10, 2, 128, {"window": 33}),                # 15 rows; tiles before the window are skipped
    (1, 1, 4099, 8, 2, 128, {}),                             # 2 units: clusters of 16 CTAs
    (1, 2, 2048, 16, 8, 128, {"softcap": 20.0}),             # 8 units: clusters of 8
    (160, 1, 130, 1, 1, 128, {}),                            # more units than SMs: one CTA per unit
    (2, 1, 700, 8, 4, 256, {"softcap": 30.0}),
    (1, 5, 333, 3, 1, 256, {"causal": False}),
    (1, 4, 640, 4, 1, 256, {"window": 1}),
])
def test_matches_oracle(cuda_device, B, Sq, Skv, H, Hk, D, opt, dtype):
  g = torch.Generator().manual_seed(Skv + H)
  q = torch.randn(B, Sq, H, D, generator=g).to(dtype)
  cache = torch.randn(B, 2, Skv, Hk, D, generator=g).to(dtype)
  ref = rm.attention_ref(q, cache[:, 0], cache[:, 1], want=("out", "lse2"), **opt)
  dev = cache.to(cuda_device)
  out, lse = att.attn_fwd_with_lse(q.to(cuda_device), dev[:, 0], dev[:, 1], **opt)
  torch.testing.assert_close(out.float().cpu(), ref["out"], **TOL[dtype])
  torch.testing.assert_close(lse.cpu(), ref["lse2"], rtol=1e-4, atol=1e-4)
  dense = att.attn_fwd(q.to(cuda_device), dev[:, 0].contiguous(), dev[:, 1].contiguous(), **opt)
  assert torch.equal(dense, out)


def test_rows_that_grow_by_large_factors(cuda_device):
  # every key tile raises the row maximum: the rescale of the partial outputs runs in every step and in both merges
  q = torch.randn(1, 2, 4, 128, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16)
  k = torch.randn(1, 900, 2, 128, generator=torch.Generator().manual_seed(2))
  k = (k * torch.linspace(0.1, 8.0, 900)[None, :, None, None]).to(torch.bfloat16)
  v = torch.randn(1, 900, 2, 128, generator=torch.Generator().manual_seed(3)).to(torch.bfloat16)
  ref = rm.attention_ref(q, k, v, want=("out",))["out"]
  out = att.attn_fwd(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device))
  torch.testing.assert_close(out.float().cpu(), ref, **TOL[torch.bfloat16])
