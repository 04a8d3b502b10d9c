"""Bounded waits in roles that a whole warp takes (csrc/attn_fwd.cuh, attn_fwd_persist.cuh, attn_sweep.cuh).  Such a wait ends lane by
lane: one lane may see the abort flag where another sees the barrier's phase.  If the first then left its role, the next step that
takes the whole warp would wait for it without limit, so every wait has one outcome for the warp.  Checked on the source text, since
going wrong could hang a GPU.  (The head_dim 256 kernel: test_split_issuer.py, test_pair_protocol.py.)"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deepgengraph_b200", "csrc")
LANE_WAIT = re.compile(r"\bmbar_wait\(")


def _source(name):
  return open(os.path.join(CSRC, name)).read()


@pytest.mark.parametrize("name", ["attn_fwd.cuh", "attn_fwd_persist.cuh"])
def test_forward_kernels_wait_lane_by_lane_only_in_the_producer(name):
  text = _source(name)
  producer, issuer = text.index("- TMA producer"), text.index("- MMA issuer")
  assert producer < issuer
  outside = [text.count("\n", 0, m.start()) + 1 for m in LANE_WAIT.finditer(text) if not producer < m.start() < issuer]
  assert not outside, f"{name}: lines {outside}"


def test_the_sweeps_vote_on_every_wait():
  text = _source("attn_sweep.cuh")
  roles = text[text.index("- MMA issuer"):]
  # behind these two nothing takes the whole warp: the lanes meet again in the block's last barrier
  roles = re.sub(r"mbar_wait\(&c\.bars\[Cfg::BAR_(COMBINE|DRAIN)\]", "", roles)
  roles = re.sub(r"if \(!__all_sync\(0xffffffffu, mbar_wait\([^;]*?\)\)\)\s*return;", "", roles)
  roles = re.sub(r"bool ok = mbar_wait\([^;]*;\s*(if constexpr \([^;]*\)\s*)?ok = ok && mbar_wait\([^;]*;\s*"
                 r"if \(!__all_sync\(0xffffffffu, ok\)\) return;", "", roles)
  assert not LANE_WAIT.search(roles), roles[LANE_WAIT.search(roles).start() - 80:][:200]


def test_a_warp_wait_votes_on_both_ways_out():
  text = _source("common.cuh")
  body = text[text.index("bool mbar_wait_warp("):]
  body = body[:body.index("\n}\n")]
  assert re.findall(r"return ([^;]*);", body) == ["true", "__all_sync(0xffffffffu, mbar_wait_slow(bar, parity, abort_flag, code))"]
  assert "if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;" in body
