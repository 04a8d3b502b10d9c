"""RMSNorm in fp32: how far the scale that a row is multiplied by is from its value in 64 bits."""
import pytest
import torch

from deepgengraph_b200 import native_ops as ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,limit", [(2560, 4.83e-8), (3584, 5.09e-8)])
def test_row_scale(cuda_device, hidden, limit):
  # The limits are what one warp per row gives, whose 32 lanes are added pairwise.  Most of it (4.6e-8 and 4.9e-8) is the
  # approximate reciprocal root; a block's eight warps added one after the other round near the total seven times instead of
  # three: 4.98e-8 and 5.25e-8.  Mean over 32768 rows: good to 0.5 %.
  g = torch.Generator(device=cuda_device).manual_seed(11)
  err = []
  for _ in range(4):
    x = torch.randn((8192, hidden), generator=g, device=cuda_device)
    out = torch.empty_like(x)
    ops.rms_norm(out, x, torch.ones(hidden, device=cuda_device), 1e-6)
    want = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-6)
    err.append((out.double() * want).sum(-1) / want.square().sum(-1) - 1)
  rms = torch.cat(err).square().mean().sqrt().item()
  assert rms < limit, f"relative error of the row scale {rms:.3e}"
