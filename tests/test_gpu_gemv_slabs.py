"""GPU: the fp16 GEMV where its division of a CTA changes: gate / up pairs, and rows of one slab (K up to 2048) with a single group of
consumer warps, on one tile, on as many as there are SMs, and on several a CTA."""
import numpy as np
import pytest

import oracle
from mtlqwen_b200 import device as D
from mtlqwen_b200.testing import synth

pytestmark = pytest.mark.gpu
TYPES = [D.Q5_K, D.Q8_0, D.IQ4_XS]


def worst_row(got, want):
  return float((np.abs(got - want.astype(np.float64)).max(axis=1) / np.abs(want).max(axis=1)).max())


# Bounds as in test_gpu_formats: exact quants times hi + lo activations, fp32 sums of up to 4096 terms.
@pytest.mark.parametrize("qtype", TYPES)
@pytest.mark.parametrize("n,k,m", [(16, 512, 8), (2368, 2048, 1), (2384, 2048, 8), (4752, 2048, 3), (16, 2304, 2), (2384, 2560, 8), (7120, 4096, 7)])
def test_pairs(dev, qtype, n, k, m):
  gate, up, x = synth.weight(qtype, n, k, 41), synth.weight(qtype, n, k, 42), synth.activations(m, k, 43)
  y = dev.empty((m, n))
  dev.gate_up(qtype, dev.array(gate), dev.array(up), n, k, dev.array(x), m, y)
  assert worst_row(y.download(), oracle.gate_up(gate, up, qtype, n, k, x)) < 1e-5


@pytest.mark.parametrize("qtype", [*TYPES, D.Q6_K])
@pytest.mark.parametrize("n,k,m", [(16, 1536, 8), (2368, 2048, 8), (2384, 2048, 1), (7120, 2048, 5), (4752, 2304, 8)])
def test_rows_of_one_slab(dev, qtype, n, k, m):
  if qtype == D.Q6_K and k % 2048:
    pytest.skip("Q6_K takes rows of whole 2048-value spans")
  w, x, residual = synth.weight(qtype, n, k, 44), synth.activations(m, k, 45), synth.activations(m, n, 46)
  y = dev.array(residual)
  dev.linear(qtype, dev.array(w), n, k, dev.array(x), m, y, y)
  assert worst_row(y.download(), oracle.linear(w, qtype, n, k, x, residual)) < 1e-5


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("xsplit", [1, 2])
@pytest.mark.parametrize("n,k,m", [(2384, 2048, 8), (2384, 2304, 3)])
def test_q4k_without_the_integer_kernel(dev, n, k, m, xsplit, pair):
  first, second, x = synth.weight(D.Q4_K, n, k, 47), synth.weight(D.Q4_K, n, k, 48), synth.activations(m, k, 49)
  y = dev.empty((m, n))
  dev.lib.infdev_set_integer_decode(dev.ctx, 0)
  dev.lib.infdev_set_xsplit(dev.ctx, xsplit)
  try:
    if pair:
      dev.gate_up(D.Q4_K, dev.array(first), dev.array(second), n, k, dev.array(x), m, y)
    else:
      dev.linear(D.Q4_K, dev.array(first), n, k, dev.array(x), m, y)
  finally:
    dev.lib.infdev_set_integer_decode(dev.ctx, 1)
    dev.lib.infdev_set_xsplit(dev.ctx, 2)
  want = oracle.gate_up(first, second, D.Q4_K, n, k, x) if pair else oracle.linear(first, D.Q4_K, n, k, x)
  assert worst_row(y.download(), want) < (1e-5 if xsplit == 2 else 3e-3)  # fp16 activations: 2^-11 of each term
