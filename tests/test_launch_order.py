"""Every launch of the library may start while its predecessor in the stream still runs (csrc/common.cuh, launch_kernel).  What a
kernel may do before it has waited for that predecessor is checked on the source text, since going wrong could hang a GPU."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deepgengraph_b200", "csrc")
PLAIN_LAUNCHES = {"kf_noise_fill_kernel", "bounded_wait_selftest_kernel"}   # <<< >>>: these start after their predecessor's end


def _kernels():
  for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    for m in re.finditer(r"__global__ void\b(?:\s*__launch_bounds__\((?:[^()]|\([^()]*\))*\))?\s*(\w+)\s*\(", text):
      start = text.index("{", text.index(")", m.end()))
      depth, end = 0, start
      while True:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
        if depth == 0:
          break
      yield m.group(1), text[start:end]


KERNELS = dict(_kernels())


def test_the_kernels_are_found():
  assert {"attn_fwd_kernel", "attn_fwd_persist_kernel", "attn_fwd_split_kernel", "attn_decode_kernel", "attn_sweep_kernel", "kv_evict_regs_kernel",
          "rms_norm_block_kernel", "rotary_online_kernel"} | PLAIN_LAUNCHES <= set(KERNELS)


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_nothing_is_taken_before_the_wait(name):
  body = KERNELS[name]
  if name in PLAIN_LAUNCHES:
    return
  assert "pdl_wait()" in body
  # Tensor memory: a predecessor that let this launch start early may still have to allocate its own.  The status word: what the
  # predecessor wrote is visible only after the wait.
  waits, depth = [], 0    # where the whole block waits: not inside a branch
  for m in re.finditer(r"[{}]|pdl_wait\(\)", body):
    if m.group() == "pdl_wait()":
      waits += [m.start()] if depth == 1 else []
    else:
      depth += 1 if m.group() == "{" else -1
  assert waits
  for taken in re.finditer(r"tmem_alloc\(|(?<!prefetch_l2\(&)g_device_status", body):
    assert waits[0] < taken.start(), f"{taken.group()} before pdl_wait()"


def test_only_the_plain_launches_are_plain():
  launched = set()
  for path in glob.glob(os.path.join(CSRC, "*.cu*")):
    launched |= set(re.findall(r"(\w+)(?:<[^<>;]*>)?<<<", open(path).read()))
  assert launched == PLAIN_LAUNCHES


BULK_COPY = re.compile(r"\btma_(?:load|store)_\dd\(|cp\.async\.bulk\.(?!commit|wait)")
FENCE = "fence_proxy_async_global();"


def _functions_with_bulk_copies():
  for path in sorted(glob.glob(os.path.join(CSRC, "attn_*.cuh"))):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    for m in re.finditer(r"__device__ __forceinline__ void (\w+)\([^;{]*\{", text):
      depth, end = 1, m.end()
      while depth:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
      if BULK_COPY.search(text, m.end(), end):
        yield m.group(1), text[m.end():end]
  yield from ((name, body) for name, body in KERNELS.items() if BULK_COPY.search(body))


def test_bulk_copies_follow_a_proxy_fence():
  # Earlier kernels read and wrote with ordinary loads and stores; a copy through the async proxy is ordered behind them by a fence of
  # the thread that issues it, after its pdl_wait.
  found = dict(_functions_with_bulk_copies())
  helpers = {"split_load_q", "split_load_k", "row_store_bulk"}   # called by the roles below
  assert set(found) == helpers | {"fwd_producer", "sweep_producer", "split_producer", "attn_fwd_persist_kernel"}
  for name in ("fwd_producer", "sweep_producer"):                # roles that begin behind the wait, one thread each
    assert found[name].index(FENCE) < BULK_COPY.search(found[name]).start(), name
    assert found[name][:found[name].index(FENCE)].count("{") == found[name][:found[name].index(FENCE)].count("}"), name
  # head_dim 256: the producer thread's first loads come before its role
  assert re.search(r"pdl_wait\(\);\s*if \(producer\) \{\s*fence_proxy_async_global\(\);\s*split_first_loads\(", KERNELS["attn_fwd_split_kernel"])
  # head_dim 128: the producer, with and without loads before its role, and the threads that store
  body = KERNELS["attn_fwd_persist_kernel"]
  wait = body.index("pdl_wait();")
  assert BULK_COPY.search(body).start() > wait
  early, = re.findall(r"if \((Cfg::STAGED && warp == PRODUCER_WARP && lane == 0)\) \{\s*fence_proxy_async_global\(\);\s*load_q\(first_tile\);", body)
  softmax, rest = body[wait:].split("if (warp < PRODUCER_WARP) {")[1].split("} else if (warp == PRODUCER_WARP) {")
  assert "if (Cfg::STAGED && lane == 0) " + FENCE in softmax[:softmax.index("for (int k = 0;;")]
  producer = rest[:rest.index("for (int k = 0; ok;")]
  assert re.search(r"if \(lane == 0\) \{\s*if \(!Cfg::STAGED\) fence_proxy_async_global\(\);", producer)


def test_dynamic_shared_memory_has_one_alignment_per_name():
  # the compiler gives all declarations of a name the alignment of one of them; kernels that do not round up rely on their own
  found = {}
  for path in glob.glob(os.path.join(CSRC, "*.cuh")):
    for align, name in re.findall(r"extern __shared__ (?:__align__\((\d+)\) )?\w+ (\w+)\[\]", open(path).read()):
      found.setdefault(name, set()).add(align)
  assert found["sweep_smem"] == found["persist_smem"] == {"1024"}
  assert all(len(aligns) == 1 for aligns in found.values()), found
