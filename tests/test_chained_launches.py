"""Every kernel that is launched chained waits for the kernel before it ahead of its first access to global memory
(csrc/common.cuh).  A missing wait is a race that a run need not show, so the sources are read."""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csrc")
FILES = sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu")))
# loads and copies as the kernels write them; prefetches are none
ACCESS = re.compile(r"tma_load_|bulk_load\(|__ldg\(|ld\.(?:global|acquire)|cp\.async\.(?!bulk\.prefetch)|fetch_keys\(|seg_range128\("
                    r"|\bp\.\w+\[|\*reinterpret_cast<const")


def _source(name):
  src = open(os.path.join(CSRC, name)).read()
  return re.sub(r"//[^\n]*|__launch_bounds__\([^)]*\)", "", src)


def _kernels(src):
  """name -> body of every __global__ function."""
  out = {}
  for m in re.finditer(r"__global__[^;{]*?\b(\w+)\s*\((?=[^;{]*\)\s*\{)", src):
    start = src.index("{", m.end())
    depth, at = 1, start + 1
    while depth:
      depth += {"{": 1, "}": -1}.get(src[at], 0)
      at += 1
    out[m.group(1)] = src[start:at]
  return out


@pytest.mark.parametrize("name", FILES)
def test_chained_kernels_wait_before_they_read(name):
  src = _source(name)
  kernels = _kernels(src)
  chained = set()
  for call in re.findall(r"\bchain(?:_clusters)?\(\s*([^,]*),", src) + re.findall(r"cudaLaunchKernelEx\(&cfg,\s*([^,]*),", src):
    chained |= set(re.findall(r"\w+_kernel\b", call))
  chained |= {k for k, body in kernels.items() if "chain_" in body}
  for k in sorted(chained):
    waits = list(re.finditer(r"if \(!chain_(?:wait|begin)\(\)\) return;", kernels[k]))
    assert waits, f"{k} does not wait"
    found = ACCESS.search(kernels[k][:waits[0].start()])
    assert found is None, f"{k} uses global memory ({found.group()}) before its wait"


def test_kernels_are_found():
  assert "gemm_kernel" in _kernels(_source("gemm_sm100.cu"))
  assert {"mla_prep_kernel", "mla_fold_kernel", "mla_split_kernel", "mla_merge_kernel"} <= set(_kernels(_source("mla_decode.cu")))
