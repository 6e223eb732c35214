"""GPU: the RMS norm that the tensor-core GEMM's operand layout does itself has the bits of the norm's own launch."""
import numpy as np
import pytest

from mtlqwen_b200 import device as D
from mtlqwen_b200.testing import synth

pytestmark = pytest.mark.gpu
K = 4096


# both sides of a step of the MMA's width, a whole launch, and two slices of rows
@pytest.mark.parametrize("m", [9, 16, 17, 128, 137])
@pytest.mark.parametrize("store", [False, True])
# K slices with a reduction, a group, a pair
@pytest.mark.parametrize("widths,pair", [((4096,), False), ((8192, 4096), False), ((12288,), True)])
def test_same_bits_as_apart(dev, m, store, widths, pair):
  x, gain = synth.activations(m, K, 81), (1 + 0.1 * synth.activations(1, K, 82)[0]).astype(np.float32)
  if m > 100:
    x[100] *= 1.0e-9
  base = synth.weight(D.Q4_K, 128, K, 83).reshape(128, -1)
  weights = [dev.array(np.tile(base, (n // 128, 1))) for n in widths]
  hidden, rows, scratch, weight = dev.array(x), dev.empty((m, K)), dev.array(np.zeros((m, K), np.float32)), dev.array(gain)

  def run(source):
    results = [dev.empty((m, n)) for n in widths]
    if pair:
      dev.gate_up(D.Q4_K, weights[0], weights[0], widths[0], K, source, m, results[0])
    elif len(widths) == 1:
      dev.linear(D.Q4_K, weights[0], widths[0], K, source, m, results[0])
    else:
      dev.linear_group(D.Q4_K, weights, widths, K, source, m, results)
    dev.commit()
    return [result.download().tobytes() for result in results]

  dev.rms_norm(hidden, weight, m, K, rows)
  want = run(rows)
  dev.norm_supply(weight, scratch, store)
  before = dev.launch_count
  assert run(hidden) == want
  assert dev.launch_count - before == ((3 if widths == (4096,) else 2) * (2 if m > 128 else 1))  # none for the norm
  if store:
    assert scratch.download().tobytes() == rows.download().tobytes()


class Part:
  """A buffer from one of its floats on."""

  def __init__(self, buffer, offset):
    self.ptr = buffer.ptr + 4 * offset


# More than one launch of 128 rows: the norm of the later ones must not meet what the earlier ones have stored, nor these a residual that is not there yet.
@pytest.mark.parametrize("m", [137, 257])
@pytest.mark.parametrize("alias", ["results over activations", "rows over activations", "everything over activations", "residual in its rows", "residual a row on",
                                   "residual of wider rows", "results over weights"])
def test_what_lies_over_what(dev, m, alias):
  n = 8192 if alias == "residual of wider rows" else K
  x, gain = synth.activations(m, K, 84), (1 + 0.1 * synth.activations(1, K, 85)[0]).astype(np.float32)
  base = synth.weight(D.Q4_K, 128, K, 86).reshape(128, -1)
  w, fill = dev.array(np.tile(base, (n // 128, 1))), synth.activations(1, (m + 1) * n, 87)[0]
  shift = {"residual in its rows": 0, "residual a row on": K, "residual of wider rows": 0}.get(alias)

  rows, want = dev.array(fill), dev.empty((m, n))  # the norm of all rows first, nothing over anything else
  dev.rms_norm(dev.array(x), dev.array(gain), m, K, rows)
  dev.linear(D.Q4_K, w, n, K, rows, m, want, None if shift is None else Part(rows, shift))
  dev.commit()

  hidden, scratch, results, weight, stored = dev.array(x), dev.array(fill), dev.empty(m * n), dev.array(gain), True
  if alias == "results over activations":
    results = hidden
  elif alias == "rows over activations":
    scratch, stored = hidden, False
  elif alias == "everything over activations":
    results = scratch = hidden
  elif alias == "results over weights":
    results = dev.array(np.concatenate([np.zeros(3 * n, np.float32), gain, np.zeros((m - 3) * n - K, np.float32)]))
    weight = Part(results, 3 * n)
  dev.norm_supply(weight, scratch, stored)
  dev.linear(D.Q4_K, w, n, K, hidden, m, results, None if shift is None else Part(scratch, shift))
  dev.commit()
  assert results.download().tobytes() == want.download().tobytes()
  if scratch is not results:
    assert scratch.download().reshape(-1)[:m * K].tobytes() == rows.download().reshape(-1)[:m * K].tobytes()
