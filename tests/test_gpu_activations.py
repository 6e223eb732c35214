"""GPU: the integer Q4_K GEMV quantising and normalising its fp32 activations itself."""
import numpy as np
import pytest

import oracle
from mtlqwen_b200 import device as D
from mtlqwen_b200.testing import synth

pytestmark = pytest.mark.gpu


def linear(dev, w, n, k, x, image=None, norm=None):
  m, y = x.shape[0], dev.empty((x.shape[0], n))
  if image is not None:
    dev.image_supply(image)
  if norm is not None:
    dev.norm_supply(*norm)
  dev.linear(D.Q4_K, w, n, k, dev.array(x), m, y)
  return y.download()


def awkward(m, k):
  """Blocks of zeros, of values whose levels overflow fp32, an infinity and a NaN, each in one super-block of one row."""
  x = synth.activations(m, k, 21)
  for row, (block, value) in enumerate(((0, 0.0), (k // 256 - 1, 1e-36), (k // 512, 1e37))):
    if row < m:
      x[row, 256 * block:256 * (block + 1)] *= np.float32(value)
  x[m - 1, k // 2 + 3] = np.inf
  x[m // 2, 17] = np.nan
  return x


# one row, two, and the eight-column form; one super-block, a chunk that ends in half a slab, several chunks
@pytest.mark.parametrize("m", [1, 2, 3, 8])
@pytest.mark.parametrize("n,k", [(16, 256), (48, 2304), (2416, 4096), (160, 5120), (64, 12288)])
@pytest.mark.parametrize("make", [lambda m, k: synth.activations(m, k, 22), awkward])
def test_same_bits_as_from_an_image(dev, m, n, k, make):
  w, x = dev.array(synth.weight(D.Q4_K, n, k, 23)), make(m, k)
  image = dev.empty(dev.image_bytes(m, k), np.uint8)
  dev.quantize(dev.array(x), m, k, image)
  assert linear(dev, w, n, k, x).tobytes() == linear(dev, w, n, k, x, image).tobytes()


@pytest.mark.parametrize("m", [1, 2, 5, 8, 9])
@pytest.mark.parametrize("n", [48, 4096])
def test_norm_on_the_way_in(dev, m, n):
  k = 4096
  weights = synth.weight(D.Q4_K, n, k, 24)
  w, x = dev.array(weights), synth.activations(m, k, 25) * np.float32(3)
  gain = (1 + 0.1 * synth.activations(1, k, 26)[0]).astype(np.float32)
  normalised, scratch = dev.array(np.zeros((m, k), np.float32)), dev.empty((m, k))
  y = linear(dev, w, n, k, x, norm=(dev.array(gain), normalised, True))
  want = oracle.rms_norm(x, gain)
  assert np.abs(normalised.download() - want).max() <= 1e-6 * np.abs(want).max()  # three roundings and a reciprocal root of a sum
  apart = dev.empty((m, k))
  dev.rms_norm(dev.array(x), dev.array(gain), m, k, apart)
  assert normalised.download().tobytes() == apart.download().tobytes()
  assert linear(dev, w, n, k, apart.download()).tobytes() == y.tobytes()
  error = np.linalg.norm(y - oracle.linear(weights, D.Q4_K, n, k, want)) / np.linalg.norm(y)
  assert error <= (1e-4 if m <= 8 else 1e-3)  # the levels of an activation block; fp16 operands above eight rows
  # a row does not depend on the others, nor on whether the normalised rows are stored
  if m <= 8:
    for row in range(m):
      assert linear(dev, w, n, k, x[row:row + 1], norm=(dev.array(gain), scratch, False)).tobytes() == y[row:row + 1].tobytes()
  # the request is gone after one call
  plain = linear(dev, w, n, k, x)
  assert np.linalg.norm(plain - oracle.linear(weights, D.Q4_K, n, k, x)) <= 1e-3 * np.linalg.norm(plain)


def test_norm_needs_a_row_of_4096_and_no_image(dev):
  gain, scratch = dev.array(np.ones(4096, np.float32)), dev.empty((1, 4096))
  w, x = dev.array(synth.weight(D.Q4_K, 16, 4096, 27)), synth.activations(1, 4096, 28)
  with pytest.raises(RuntimeError, match="4096"):
    linear(dev, w, 16, 2048, x[:, :2048], norm=(gain, scratch))
  image = dev.empty(dev.image_bytes(1, 4096), np.uint8)
  dev.quantize(dev.array(x), 1, 4096, image)
  with pytest.raises(RuntimeError, match="no image"):
    linear(dev, w, 16, 4096, x, image, (gain, scratch))


def in_place(dev, w, n, k, x, norm=None, normalised=None, residual=False):
  """The result over the activations (n = k)."""
  buffer = dev.array(x)
  if norm is not None:
    dev.norm_supply(norm, buffer if normalised is None else normalised, True)
  dev.linear(D.Q4_K, w, n, k, buffer, x.shape[0], buffer, buffer if residual else None)
  return buffer.download()


# more tiles than SMs, fewer, and several K chunks, which read the activations again behind the first stores
@pytest.mark.parametrize("m", [1, 2, 3, 8])
@pytest.mark.parametrize("k", [1024, 4096, 8192])
def test_result_over_its_activations(dev, m, k):
  w, x = dev.array(synth.weight(D.Q4_K, k, k, 31)), synth.activations(m, k, 32)
  assert in_place(dev, w, k, k, x).tobytes() == linear(dev, w, k, k, x).tobytes()


@pytest.mark.parametrize("m", [1, 2, 8, 9])
def test_norm_over_its_activations_and_results(dev, m):
  k = 4096
  w, x = dev.array(synth.weight(D.Q4_K, k, k, 33)), synth.activations(m, k, 34)
  gain, scratch = dev.array((1 + 0.1 * synth.activations(1, k, 35)[0]).astype(np.float32)), dev.empty((m, k))
  want = linear(dev, w, k, k, x, norm=(gain, scratch, True))
  assert in_place(dev, w, k, k, x, gain).tobytes() == want.tobytes()  # norm, activations and result in one buffer
  assert in_place(dev, w, k, k, x, gain, scratch).tobytes() == want.tobytes()  # result over the activations
  assert in_place(dev, w, k, k, x, gain, scratch, True).tobytes() == (want + x).astype(np.float32).tobytes()
  y = dev.empty((m, k))
  dev.norm_supply(gain, y)  # norm where the result goes
  dev.linear(D.Q4_K, w, k, k, dev.array(x), m, y)
  assert y.download().tobytes() == want.tobytes()
  buffer = dev.array(x)
  dev.norm_supply(gain, buffer, True)  # norm over the activations
  dev.linear(D.Q4_K, w, k, k, buffer, m, y)
  assert y.download().tobytes() == want.tobytes() and buffer.download().tobytes() == scratch.download().tobytes()


def test_norm_across_its_activations_is_refused(dev):
  k, m = 4096, 2
  w, gain = dev.array(synth.weight(D.Q4_K, 16, k, 36)), dev.array(np.ones(k, np.float32))
  buffer = dev.array(synth.activations(m + 1, k, 37))
  dev.norm_supply(gain, type("View", (), {"ptr": buffer.ptr + 4 * k}))
  with pytest.raises(RuntimeError, match="across"):
    dev.linear(D.Q4_K, w, 16, k, buffer, m, dev.empty((m, 16)))


@pytest.mark.parametrize("qtype,n,m", [(D.Q6_K, 24, 1), (D.Q4_K, 24, 9), (D.Q4_K, 24, 1)])
def test_a_refused_call_leaves_the_normalised_rows_alone(dev, qtype, n, m):
  k = 4096
  w, gain, scratch = dev.empty(n * k, np.uint8), dev.array(np.ones(k, np.float32)), dev.array(np.zeros((m, k), np.float32))
  dev.norm_supply(gain, scratch, True)
  with pytest.raises(RuntimeError, match="multiple of 16"):
    dev.linear(qtype, w, n, k, dev.array(synth.activations(m, k, 38)), m, dev.empty((m, n)))
  assert not scratch.download().any()
