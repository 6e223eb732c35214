"""CPU: warps that read and write tensor memory together leave their loops together when a bounded wait runs out, and hand nothing on after it."""
import re

import pytest

from mtlqwen_b200 import build


def role(name, begin, end):
  source = (build.CSRC / name).read_text()
  return source[source.index(begin):source.index(end, source.index(begin))]


@pytest.mark.parametrize("name,begin,end", [("umma.cu", "// ---------------- dequant:", "  fence_before_sync();\n  __syncthreads();\n  if (warp == kIssueWarp)"),
                                            ("attention.cu", "// ---------------- workers:", "  if (!ok && lane == 0) {")])
def test_waits_are_the_whole_warps(name, begin, end):
  text = role(name, begin, end)
  assert re.search(r"tmem_(load|store)|store_rows", text)
  waits = [line for line in text.splitlines() if "mbar_wait_bounded(" in line]
  assert waits and all(re.search(r"__all_sync\(0xffffffffu, (ok && )?mbar_wait_bounded\(", line) for line in waits), waits


def test_no_operand_is_stored_or_announced_after_a_wait_that_ran_out():
  text = role("umma.cu", "// ---------------- dequant:", "// ---- epilogue:")
  stores = [match.start() for match in re.finditer(r"tmem_store32\(", text)]
  assert stores and all(re.search(r"if \(ok\)\s*$", text[:at]) for at in stores)
  announced = text.index("mbar_arrive(&ctl.aReady")
  assert re.search(r"if \(!ok\)\s+break;", text[max(stores):announced])
