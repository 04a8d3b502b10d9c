"""The launch of an eviction holds as many CTAs as are resident at once: each of them repeats the selection, so a second wave
would double it."""
import pytest
import torch

from deepgengraph_b200 import attention as att

pytestmark = pytest.mark.gpu


def _best_ms(fn, launches=20, batches=8):
  start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
  times = []
  for _ in range(batches):
    start.record()
    for _ in range(launches):
      fn()
    end.record()
    end.synchronize()
    times.append(start.elapsed_time(end))
  return min(times[1:])


@pytest.mark.parametrize("seq", [5000, 12000, 16384])
def test_more_heads_do_not_start_a_second_wave(cuda_device, seq):
  # 8 heads leave half of the chip idle, 32 fill it: the selections run side by side and only the gather grows.  Measured 1.41,
  # 1.08 and 1.16 times the time; with a second wave 1.98, 2.03 and 2.06.
  def time_of(heads):
    g = torch.Generator(device=cuda_device).manual_seed(seq)
    p = torch.randn((1, heads, 64, seq), generator=g, device=cuda_device).mul_(2.0).softmax(-1)
    score, score_sq = p.sum(2), p.square().sum(2)
    k, v = (torch.randn((1, seq, heads, 128), generator=g, device=cuda_device).to(torch.bfloat16) for _ in range(2))
    return _best_ms(lambda: att.kv_evict_roco(score, score_sq, k, v, 64, seq // 8, 32))

  few, many = time_of(8), time_of(32)
  assert many < 1.7 * few, f"8 heads {few * 50:.1f} us, 32 heads {many * 50:.1f} us a launch"
