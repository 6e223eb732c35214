"""GPU: the rings of the tensor-core GEMM, whose slots follow the row count, and its two accumulators, against fp64."""
import numpy as np
import pytest

from mtlqwen_b200 import device as D
from mtlqwen_b200.testing import synth

pytestmark = pytest.mark.gpu


# every width of the MMA from both sides: the last row count of one ring geometry and the first of the next
@pytest.mark.parametrize("m", [9, 16, 17, 32, 33, 48, 49, 64, 65, 80, 81, 96, 97, 112, 113, 128])
# K slices of fewer super-blocks than a ring has slots, one item of more, and two items for one CTA
@pytest.mark.parametrize("n,k", [(128, 2048), (256, 6144), (19072, 2048)])
def test_ring_geometries(dev, n, k, m):
  rows = 256  # the matrix repeats these, so that the reference stays small
  base = synth.weight(D.Q4_K, rows, k, 71).reshape(rows, -1)
  w, x, res = np.tile(base, (-(-n // rows), 1))[:n], synth.activations(m, k, 72), synth.activations(m, n, 73)
  y, dense = dev.empty((m, n)), dev.empty((rows, k))
  weights = dev.array(w)
  dev.dequant(D.Q4_K, weights, rows * k // 256 if n >= rows else n * k // 256, dense)
  dev.linear(D.Q4_K, weights, n, k, dev.array(x), m, y, dev.array(res))
  dev.commit()
  live = min(n, rows)
  product = x.astype(np.float64) @ dense.download()[:live].astype(np.float64).T
  want = np.tile(product, (1, -(-n // live)))[:, :n] + res
  # weights and activations are rounded to fp16 (2^-12 of either on average, at most 2^-11): 4.5e-4 of the product, which is at most the sum
  error = np.linalg.norm(y.download() - want, axis=1) / np.linalg.norm(want - res, axis=1)
  assert error.max() <= 1e-3
