"""GPU: the preparation of the gated delta rule spreads its rows by their number; the bits do not depend on it."""
import numpy as np
import pytest

from mtlqwen_b200 import device as D
from test_gpu_gdn import LAYER, View, layer_weights

pytestmark = pytest.mark.gpu


# both sides of every line, with queries that begin and end inside the rows of a thread
@pytest.mark.parametrize("lengths", [[24], [3, 22], [47, 1], [5, 2, 42], [1, 190, 1], [100, 3, 90], [9, 1, 2, 200, 3, 5]])
def test_every_spread_has_the_same_bits(dev, lengths):
  rng = np.random.default_rng(41)
  rows, nq = sum(lengths), len(lengths)
  w = {name: dev.array(value) for name, value in layer_weights(rng).items()}
  x, mixed = dev.array(rng.standard_normal((rows, 4096)).astype(np.float32)), rng.standard_normal((rows, 8192)).astype(np.float32)
  previous = dev.array(rng.standard_normal((nq, LAYER // 4)).astype(np.float32))

  def run(offset):  # inputs off 16 bytes take the spread of one row and one head
    next_ = dev.empty((nq, LAYER // 4))
    queries, start = [], 0
    for i, count in enumerate(lengths):
      q = D.Query()
      q.previous, q.next = previous.ptr + i * LAYER, next_.ptr + i * LAYER
      q.start, q.count, q.position, q.slot, q.state = start, count, 77, i, D.UNBOUND
      queries.append(q)
      start += count
    out = [dev.empty((rows, 2048)), dev.empty((rows, 2048)), dev.empty((rows, 4096)), dev.empty((rows, 32)), dev.empty((rows, 32))]
    dev.gdn_prepare(x, View(dev, mixed, offset=offset), w["w_beta"], w["w_alpha"], w["ssm_a"], w["ssm_dt"], w["conv"], dev.queries(queries), nq, rows, 0, LAYER,
                    *out)
    dev.commit()
    return [buffer.download().tobytes() for buffer in (*out, next_)]

  assert run(0) == run(1)
