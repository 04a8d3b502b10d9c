"""Calls that reach the native host path of the public operators in other ways than a plain call with regular arguments."""
import math

import pytest
import torch

from deepgengraph_b200 import _lib
from deepgengraph_b200 import attention as att

pytestmark = pytest.mark.gpu


def _rand(*shape, dtype=torch.bfloat16, seed=0):
  return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(dtype).cuda()


@pytest.mark.parametrize("fn", [att.attn_fwd, att.attn_fwd_with_lse, att.attn_score_fwd, att.attn_kf_fwd, att.attn_snapkv_fwd,
                                att.attn_corm_fwd])
def test_a_scale_that_is_no_number_is_refused(cuda_device, fn):
  q = _rand(1, 64, 2, 128)
  with pytest.raises(_lib.B200Error):
    fn(q, q, q, scale=math.nan)
