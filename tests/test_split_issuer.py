"""The MMA issuer of the head_dim 256 attention kernel (csrc/attn_fwd_split.cuh) after a wait that ran out.  Its waits end lane by lane, so
one lane may give up where another goes on; a lane that left the loop would then be waited for, without limit, by the next step that
takes the whole warp.  Checked on the source text, since going wrong could hang a GPU."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deepgengraph_b200", "csrc")
WHOLE_WARP = r"__all_sync|__any_sync|__syncwarp|wait_warp|elect_one|__shfl"


def _issuer():
  text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "attn_fwd_split.cuh")).read())
  body = text[text.index("void split_issuer("):]
  body = body[:body.index("Cfg::BAR_DRAIN")]
  tiles = body.index("for (int k = 0; ok; ++k) {")
  return body[:tiles], body[tiles:]


def test_lanes_agree_before_the_next_step_of_the_whole_warp():
  _, loop = _issuer()
  first_lane_wait = re.search(r"ok = c\.wait\(", loop).start()
  vote = "ok = __all_sync(0xffffffffu, ok);"
  assert vote in loop[first_lane_wait:]
  between, after = loop[first_lane_wait:].split(vote, 1)
  assert not re.search(WHOLE_WARP, between), "a step of the whole warp between a lane's wait and the vote"
  assert "return" not in between          # a lane that gave up skips to the vote: it may leave the block loops, not the tile loop
  assert between.count("{") == between.count("}")
  assert re.match(r"\s*g0 \+= nb;\s*\}", after)


def test_the_issue_helpers_take_no_step_of_the_whole_warp():
  helpers, _ = _issuer()
  helpers = helpers[helpers.index("auto wait_full = "):]
  assert not re.search(WHOLE_WARP, helpers)


def test_an_expired_wait_for_v_is_reported_as_one_for_v():
  text = open(os.path.join(CSRC, "attn_fwd_split.cuh")).read()
  assert "is_v ? WAIT_V_EMPTY : WAIT_K_EMPTY" in text                                        # the producer's one wait
  full = dict(re.findall(r"wait_full\((ring_i(?: \+ part)?), (\w+)\)", text))                # the issuer's two
  assert full == {"ring_i": "WAIT_K_FULL", "ring_i + part": "WAIT_V_FULL"}
