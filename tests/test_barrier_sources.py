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
