"""Where the forward kernel's bulk stores are cut off (a warp stores 32 rows, a tile has 128) and where the rings of the KeyFormer
sweeps wrap (one stage of the streamed operand, three of noise, 64-wide blocks)."""
import pytest
import torch

from deepgengraph_b200 import _lib
from deepgengraph_b200 import attention as att
from oracle import reference_math as rm

pytestmark = pytest.mark.gpu


def _rand(*shape, seed, dtype):
  return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(dtype)


@pytest.mark.parametrize("q_len", [17, 31, 32, 33, 64, 97, 127, 128, 129, 160, 161, 255, 257])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_rows_of_the_last_tile(cuda_device, q_len, dtype):
  B, H = 2, 3
  q, k, v = (_rand(B, q_len, H, 128, seed=q_len + i, dtype=dtype).to(cuda_device) for i in range(3))
  guard = 64 * 128 * H   # as many elements as the rows of half a tile
  flat = torch.full((q.numel() + guard,), float("nan"), dtype=dtype, device=cuda_device)
  st = _lib.load().b200_attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), flat.data_ptr(), None, B, q_len, q_len, H, H, 128,
                                 _lib.BF16 if dtype == torch.bfloat16 else _lib.F16, 1, 0, 0.0, 128 ** -0.5,
                                 torch.cuda.current_stream(cuda_device).cuda_stream)
  assert st == 0
  assert torch.isnan(flat[q.numel():].float()).all()   # nothing behind the last row; batch 0's tail would land in batch 1
  ref = rm.attention_ref(q.cpu(), k.cpu(), v.cpu(), want=("out",))["out"]
  # P and the output are rounded to the type once each; the result is a weighted mean of N(0, 1) values, of magnitude below 5
  eps = 2 ** -9 if dtype == torch.bfloat16 else 2 ** -12
  torch.testing.assert_close(flat[:q.numel()].view_as(q).float().cpu(), ref, rtol=0, atol=2 * eps * 5)


@pytest.mark.parametrize("seq", [4, 64, 68, 128, 132, 192, 196, 256, 260, 388])
def test_keyformer_ring_depths(cuda_device, seq):
  q, k, v = (_rand(1, seq, 2, 128, seed=seq + i, dtype=torch.bfloat16) for i in range(3))
  noise = -torch.rand(1, 2, seq, seq, generator=torch.Generator().manual_seed(seq)).clamp_min(1e-10).log()
  ref = rm.attention_ref(q, k, v, exp_rand=noise, tau=1.5, want=("kf",))["kf"]
  _, score = att.attn_kf_fwd(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device), noise.to(cuda_device), tau=1.5)
  # sums of at most 388 fp32 probabilities, exponents good to 2^-20
  torch.testing.assert_close(score.cpu(), ref, rtol=1e-3, atol=1e-5)


@pytest.mark.parametrize("q_len,kv_len,heads,kv_heads", [(1, 200, 2, 2), (127, 129, 2, 2), (4096, 4100, 1, 1), (4097, 4100, 1, 1),
                                                         (300, 300, 4, 2), (4100, 4100, 2, 1)])
def test_sums_written_to_the_result_or_reduced(cuda_device, q_len, kv_len, heads, kv_heads):
  # one partial sum per key (up to 4096 queries, one query head per K/V head or the sweep over the group's mean), or several
  q = _rand(1, q_len, heads, 128, seed=q_len, dtype=torch.bfloat16).to(cuda_device)
  k, v = (_rand(1, kv_len, kv_heads, 128, seed=kv_len + i, dtype=torch.bfloat16).to(cuda_device) for i in range(2))
  ref = rm.attention_ref(q, k, v, want=("out", "colsum", "colsum_sq"))
  _, score, score_sq = att.attn_score_fwd(q, k, v, want_sq=True)
  _, alone = att.attn_score_fwd(q, k, v)
  # fp32 sums of at most 4100 probabilities, exponents good to 2^-20
  torch.testing.assert_close(score, ref["colsum"], rtol=1e-3, atol=1e-5)
  torch.testing.assert_close(score_sq, ref["colsum_sq"], rtol=1e-3, atol=1e-5)
  torch.testing.assert_close(alone, ref["colsum"], rtol=1e-3, atol=1e-5)


@pytest.mark.parametrize("q_len,kv_len", [(2048, 2048), (2049, 2052)])
def test_keyformer_sums_of_one_and_two_chunks(cuda_device, q_len, kv_len):
  q = _rand(1, q_len, 1, 128, seed=1, dtype=torch.float16).to(cuda_device)
  k, v = (_rand(1, kv_len, 1, 128, seed=2 + i, dtype=torch.float16).to(cuda_device) for i in range(2))
  noise = -torch.rand(1, 1, q_len, kv_len, generator=torch.Generator().manual_seed(5)).clamp_min(1e-10).log().to(cuda_device)
  ref = rm.attention_ref(q, k, v, exp_rand=noise, tau=1.0, want=("kf",))["kf"]
  _, score = att.attn_kf_fwd(q, k, v, noise, tau=1.0)
  torch.testing.assert_close(score, ref, rtol=1e-3, atol=1e-5)
