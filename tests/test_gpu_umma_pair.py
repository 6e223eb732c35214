"""GPU: the gate / up pair of the tensor-core GEMM, whose two accumulators take all of a CTA's buffers."""
import numpy as np
import pytest

import oracle
from mtlqwen_b200 import device as D
from mtlqwen_b200.testing import synth

pytestmark = pytest.mark.gpu


# one tile; more tiles than SMs, so that a CTA waits for its epilogue before the next; the fewest rows, both sides of a step of 16, all
@pytest.mark.parametrize("n,k", [(128, 2048), (19072, 2048), (384, 4096)])
@pytest.mark.parametrize("m", [9, 16, 17, 96, 97, 128])
def test_gate_up(dev, n, k, m):
  gate, up, x = synth.weight(D.Q4_K, n, k, 61), synth.weight(D.Q4_K, n, k, 62), synth.activations(m, k, 63)
  y = dev.empty((m, n))
  dev.gate_up(D.Q4_K, dev.array(gate), dev.array(up), n, k, dev.array(x), m, y)
  want = oracle.gate_up(gate, up, D.Q4_K, n, k, x).astype(np.float64)
  rows = np.linalg.norm(y.download() - want, axis=1) / np.linalg.norm(want, axis=1)
  assert rows.max() <= 1.5e-3  # the fp16 operands' 5e-4 of either factor
