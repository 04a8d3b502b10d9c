"""The eviction kernels around the sizes where their work is cut differently: keys per thread (2, 4, ... 32 of 512 threads),
the longest sequence whose keys stay in registers and the first one beyond it, rows of scores that are not 16-byte aligned,
many equal scores.  Index work: bit-exact; equal scores are taken in key order."""
import pytest
import torch

from deepgengraph_b200 import attention as att

pytestmark = pytest.mark.gpu


def _pick(rank_by, n):
  return torch.argsort(rank_by, dim=-1, descending=True, stable=True)[..., :n]


@pytest.mark.parametrize("seq,budget", [(1, 1), (31, 7), (511, 511), (1024, 1), (1025, 300), (2049, 64), (4095, 2000), (4097, 512),
                                        (8193, 4097), (16384, 12288), (16385, 100)])
@pytest.mark.parametrize("levels", [0, 5])
def test_selection_and_rows(cuda_device, seq, budget, levels):
  B, H, D = 2, 3, 64
  g = torch.Generator().manual_seed(seq + levels)
  score = torch.randn(B, H, seq, generator=g)
  if levels:
    score = torch.round(score * levels) / levels + 0.0   # a handful of distinct values, none of them -0.0
  k, v = (torch.randn(B, seq, H, D, generator=g).to(torch.bfloat16) for _ in range(2))
  want = _pick(score, budget).sort(dim=-1)[0]
  cache, idx = att.kv_evict_topk(score.to(cuda_device), k.to(cuda_device), v.to(cuda_device), budget, return_indices=True)
  assert torch.equal(idx.cpu().long(), want)
  rows = want.permute(0, 2, 1)[..., None].expand(B, budget, H, D)
  assert torch.equal(cache.cpu(), torch.stack([k.gather(1, rows), v.gather(1, rows)], dim=1))


@pytest.mark.parametrize("seq,budget,recent", [(2, 1, 1), (513, 0, 513), (1023, 500, 0), (3001, 900, 130), (16384, 9000, 77),
                                               (16385, 40, 16)])
@pytest.mark.parametrize("levels", [0, 4])
def test_two_stage_selection(cuda_device, seq, budget, recent, levels):
  B, H, D, q_len = 1, 2, 32, 64.0
  g = torch.Generator().manual_seed(seq)
  score = torch.rand(B, H, seq, generator=g) * 8
  if levels:
    score = torch.round(score * levels) / levels
  score_sq = score * score / q_len * (1.0 + torch.rand(B, H, seq, generator=g).round(decimals=1 if levels else 6))
  k, v = (torch.randn(B, seq, H, D, generator=g) for _ in range(2))
  mean = score / q_len
  std = torch.sqrt(score_sq / q_len - mean * mean)
  std = torch.where(torch.isnan(std), torch.full_like(std, float("inf")), std)   # NaN ranks above everything
  taken = torch.zeros(B, H, seq, dtype=torch.bool).scatter_(-1, _pick(std, recent), True)
  taken.scatter_(-1, _pick(torch.where(taken, torch.full_like(mean, -1.0), mean), budget), True)
  want = taken.nonzero()[:, 2].view(B, H, budget + recent)
  cache, idx = att.kv_evict_roco(score.to(cuda_device), score_sq.to(cuda_device), k.to(cuda_device), v.to(cuda_device),
                                 int(q_len), budget, recent, return_indices=True)
  assert torch.equal(idx.cpu().long(), want)
  rows = want.permute(0, 2, 1)[..., None].expand(B, budget + recent, H, D)
  assert torch.equal(cache.cpu(), torch.stack([k.gather(1, rows), v.gather(1, rows)], dim=1))
