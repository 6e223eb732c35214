"""CPU: what ptxas reports of the matrix kernels whose shared-memory carve-out leaves local memory no L1."""
import re
import shutil
import subprocess
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import pytest

from mtlqwen_b200 import build


def compiled(name, directory):
  """{(type, integers of the template): (stack frame, spill stores)} of the kernels of one source."""
  nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
  report = subprocess.run([nvcc, *build.ARCH, *build.FLAGS, "-Xptxas=-v", "-I", str(build.PACKAGE.parent / "include"), "-x", "cu", "-cubin", str(build.CSRC / name),
                           "-o", str(directory / (name + ".out"))], capture_output=True, text=True, check=True).stderr
  found = re.findall(r"Function properties for (\S+)\s+(\d+) bytes stack frame, (\d+) bytes spill stores", report)
  return {(match[1], tuple(int(v) for v in re.findall(r"Li(\d+)E", match[2]))): (int(stack), int(spills))
          for symbol, stack, spills in found if (match := re.search(r"kernelINS0_\d(\w+?)E((?:Li\d+E)+)", symbol))}


@pytest.fixture(scope="module")
def reports(tmp_path_factory):
  directory = tmp_path_factory.mktemp("ptxas")
  with ThreadPoolExecutor() as pool:
    return dict(zip(("gemv.cu", "gemv_wide.cu"), pool.map(lambda name: compiled(name, directory), ("gemv.cu", "gemv_wide.cu"))))


def test_gemv_keeps_no_array_in_local_memory(reports):
  """A frame beyond the spills (rounded to eight bytes) is an array that is chosen from at run time."""
  kernels = reports["gemv.cu"]
  assert len(kernels) >= 12
  for kernel, (stack, spills) in kernels.items():
    assert stack <= (spills + 7) // 8 * 8, kernel


def test_q6k_of_few_rows_is_decoded_without_spills(reports):
  kernels = {tiles: spills for (qtype, tiles), (_, spills) in reports["gemv_wide.cu"].items() if qtype == "Q6K"}
  assert sorted(kernels) == [(2, ), (3, ), (4, ), (5, )] and not any(kernels.values()), kernels


def test_the_norm_of_long_queries_leaves_short_ones_their_registers(tmp_path):
  """The launch of the token-by-token delta rule also normalises the outputs of the chunked one: without that it spills 52 bytes, with the norm inlined 68."""
  nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
  report = subprocess.run([nvcc, *build.ARCH, *build.FLAGS, "-Xptxas=-v", "-I", str(build.PACKAGE.parent / "include"), "-x", "cu", "-cubin", str(build.CSRC / "gdn.cu"),
                           "-o", str(tmp_path / "gdn.out")], capture_output=True, text=True, check=True).stderr
  spills = re.findall(r"Function properties for \S*delta_rule_kernelILb0E\S*\s+\d+ bytes stack frame, (\d+) bytes spill stores", report)
  assert len(spills) == 1 and int(spills[0]) <= 52
