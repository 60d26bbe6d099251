"""What orders a barrier's initialisation before its use, and a signal or a read across a cluster before its owner leaves
(csrc/common.cuh).  A missing order is a race that a run need not show, so the sources are read."""

import re

import pytest
from test_chained_launches import FILES, _kernels, _source

BLOCK_SYNC = re.compile(r"__syncthreads(?:_\w+)?\(|__syncwarp\(|cluster_sync_all\(")


@pytest.mark.parametrize("name", FILES)
def test_barriers_are_initialised_before_another_lane_uses_them(name):
  """Thread 0 initialises; the lane that `one_lane` or `elect_one` picks need not be lane 0."""
  for kernel, body in _kernels(_source(name)).items():
    inits = [m.end() for m in re.finditer(r"if \(threadIdx\.x == 0\) \{", body) if "mbar_init" in body[m.end():m.end() + 200]]
    for at in inits:
      used = re.search(r"\bone_lane\(|\belect_one\(", body[at:])
      if used:
        assert BLOCK_SYNC.search(body[at:at + used.start()]), f"{kernel} uses its barriers before they are seen"


def _without_loops(body, head):
  """``body`` without the loops that begin with ``head``."""
  while (start := body.find(head)) >= 0:
    at, depth = body.index("{", body.index(")", start)), 0
    while True:
      depth += {"{": 1, "}": -1}.get(body[at], 0)
      at += 1
      if not depth:
        break
    body = body[:start] + body[at:]
  return body


@pytest.mark.parametrize("barrier", ["acc_empty", "empty", "ring_free"])
def test_a_pair_waits_for_the_last_signals_of_its_neighbours(barrier):
  """In the tile loop these barriers are waited for ahead of a reuse; the signals after the last one have a wait of their own,
  so that none reaches shared memory whose CTA has left."""
  body = _kernels(_source("gemm_sm100.cu"))["gemm_kernel"]
  assert "cluster_leave()" in body
  rest = _without_loops(body, "for (int t = cta;")
  assert re.search(r"mbar_wait(?:_warp|_cluster)?\(&?%s\b" % barrier, rest), f"nobody waits for the last arrival on {barrier}"


def test_loads_of_a_neighbours_memory_feed_a_store():
  """Threads without a result load nothing: nothing would wait for such a load before the neighbour leaves."""
  body = _kernels(_source("moe.cu"))["logit_dw_kernel"]
  tail = body[body.rindex("cluster_sync_all()"):]
  assert 0 < tail.find("if (n0 + n < N && c0 + c < K) {") < tail.index("ld.shared::cluster")


@pytest.mark.parametrize("name", FILES)
def test_shared_arrays_read_as_vectors_are_aligned_for_them(name):
  """A __shared__ array has its element's alignment unless it says more."""
  for kernel, body in _kernels(_source(name)).items():
    for decl in re.finditer(r"__shared__ ((?:__align__\(\d+\) )?)(float|int|__nv_bfloat16|unsigned|uint8_t) (\w+)\[", body):
      if not decl.group(1):
        as_vector = re.search(r"reinterpret_cast<(?:const )?(?:float|int|uint|double)[24]\*>\(&?%s\b" % decl.group(3), body)
        assert as_vector is None, f"{kernel}: {decl.group(3)} is read as {as_vector.group()}"


@pytest.mark.parametrize("name", FILES)
def test_warps_part_from_a_cluster_together(name):
  """The cluster barrier is the aligned one: all lanes of a warp arrive at once, also those that have left a loop early."""
  for kernel, body in _kernels(_source(name)).items():
    for m in re.finditer(r"(?:if \([^()]*\) )?cluster_leave\(\);", body):
      assert re.search(r"__sync(?:threads|warp)\(\);\s*$", body[:m.start()]), f"{kernel} may part in pieces"
