"""GPU: both ways in which the tensor-core GEMM dequantises Q4_K, on either side of the scales where they part."""
import numpy as np
import pytest

from mtlqwen_b200 import device as D
from mtlqwen_b200.testing import synth

pytestmark = pytest.mark.gpu


def set_scales(blocks, rng, value):
  """d so that the largest product d * sc of a block is about `value`, either sign."""
  largest = 63.0
  d = (value / largest * rng.choice([-1.0, 1.0], blocks.shape[0])).astype(np.float16)
  blocks[:, 0:2] = d.view(np.uint8).reshape(-1, 2)
  blocks[:, 2:4] = (d.astype(np.float32) * 7.5).astype(np.float16).view(np.uint8).reshape(-1, 2)
  return blocks


# subnormal products, ordinary ones, the line at 2^-6 from both sides, scales far above it, and rows of both kinds in one warp
@pytest.mark.parametrize("value", [3e-6, 4e-3, 0.0155, 0.0157, 0.3, 40.0, None])
@pytest.mark.parametrize("pair", [False, True])
def test_scales(dev, value, pair):
  n, k, m = 256, 2048, 24
  rng = np.random.default_rng(81)
  weights = []
  for seed in range(2 if pair else 1):
    blocks = synth.weight(D.Q4_K, n, k, 82 + seed).reshape(-1, 144)
    blocks = blocks.copy()
    if value is None:
      for row in range(n):
        set_scales(blocks[row * k // 256:(row + 1) * k // 256], rng, 0.004 if row % 3 else 0.5)
    else:
      set_scales(blocks, rng, value)
    weights.append(blocks)
  x = synth.activations(m, k, 84)
  y, dense = dev.empty((m, n)), dev.empty((n, k))
  buffers, products = [dev.array(w) for w in weights], []
  for w in buffers:
    dev.dequant(D.Q4_K, w, n * k // 256, dense)
    # the operands as the kernel has them: fp16 weights and activations, products summed without error
    products.append(x.astype(np.float16).astype(np.float64) @ dense.download().astype(np.float64).T)
  if pair:
    dev.gate_up(D.Q4_K, buffers[0], buffers[1], n, k, dev.array(x), m, y)
    with np.errstate(over="ignore"):
      want = products[0] / (1 + np.exp(-products[0])) * products[1]
  else:
    dev.linear(D.Q4_K, buffers[0], n, k, dev.array(x), m, y)
    want = products[0]
  dev.commit()
  # A weight is d*sc*q - dmin*m with d*sc and dmin*m rounded to fp16 first: relative 2^-11 of terms that are up to 15/7.5 of the weights'
  # spread, or half a step of 2^-24 where they are subnormal (products of 3e-6: 0.01 of them).
  bound = 3e-2 if value == 3e-6 else 1.5e-3
  error = np.linalg.norm(y.download() - want, axis=1) / np.linalg.norm(want, axis=1)
  assert error.max() <= bound * (2 if pair else 1)
