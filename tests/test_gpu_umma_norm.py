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
