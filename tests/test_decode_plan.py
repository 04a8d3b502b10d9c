"""The split of a few-rows attention launch over clusters (csrc/attn_decode_plan.h), compiled for the host."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deepgengraph_b200", "csrc")
PROGRAM = """
#include "attn_decode_plan.h"
extern "C" int cluster(long long units, int n_tiles, int sms, int placeable) {
  return b200::decode_cluster_that_fits(b200::decode_split(units, n_tiles, sms).ctas, units, placeable);
}
"""


@pytest.fixture(scope="module")
def cluster(tmp_path_factory):
  d = tmp_path_factory.mktemp("plan")
  (d / "plan.cpp").write_text(PROGRAM)
  subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "plan.so"),
                  str(d / "plan.cpp")], check=True)
  fn = ctypes.CDLL(str(d / "plan.so")).cluster
  fn.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_int, ctypes.c_int]
  return fn


@pytest.mark.parametrize("units,placeable,want", [(2, 7, 16), (4, 4, 16), (4, 3, 8), (1, 0, 8), (2, 0, 8), (8, 0, 8)])
def test_clusters_that_the_device_cannot_place_are_not_launched(cluster, units, placeable, want):
  assert cluster(units, 1024, 148, placeable) == want


def test_the_launch_stays_within_one_cta_per_sm(cluster):
  for sms in (16, 132, 148):
    for units in (1, 2, 3, 4, 5, 8, 10, 33, 64, 74, 75, 148, 149, 1000):
      for n_tiles in (1, 8, 9, 31, 32, 171, 512, 1 << 27):
        c = cluster(units, n_tiles, sms, 4)
        assert c in (1, 2, 4, 8, 16) and (c == 1 or c * units <= sms)
