"""GPU: the sums under the norms have one order of additions, whichever kernel forms them.

A sum cannot be read from outside, but a scale can: a second row of powers of two, whose squares add up to the first row's
expected sum without any rounding, has the scale that the first one must have."""
import numpy as np
import pytest

from mtlqwen_b200 import device as D
from mtlqwen_b200.testing import synth

pytestmark = pytest.mark.gpu


def fma(a, b, c):
  return (a.astype(np.float64) * b + c).astype(np.float32)


def butterfly(values):
  """Sum over the last axis as the lanes of a warp form it: partners 16, 8, 4, 2, 1 apart."""
  while values.shape[-1] > 1:
    half = values.shape[-1] // 2
    values = values[..., :half] + values[..., half:]
  return values[..., 0]


def in_turn(values):
  total = values[..., 0]
  for i in range(1, values.shape[-1]):
    total = total + values[..., i]
  return total


def row_sums(x):
  """Rows of 4096: a lane's eight values in two chains, a warp's lanes, the sixteen warps in turn."""
  v = x.reshape(len(x), 16, 32, 2, 4)
  chain = v[..., 1] * v[..., 1]
  for i in (0, 2, 3):
    chain = fma(v[..., i], v[..., i], chain)
  return in_turn(butterfly(chain[..., 0] + chain[..., 1]))


def head_sums(x):
  """Heads of 256: the squares of 32 dims as of the lanes of a warp, the eight groups in turn."""
  return in_turn(butterfly((x * x).reshape(*x.shape[:-1], 8, 32)))


def powers_of_two(total, width, first):
  """A row whose squares add up to `total` exactly, in any order; None where the last of its 24 bits would take half of itself twice."""
  mantissa, exponent = np.frexp(np.float64(total))
  row, at, bits = np.zeros(width, np.float32), first, int(mantissa * 2**24)
  if bits & 1 and exponent % 2:
    return None
  for bit in reversed(range(24)):
    power = int(exponent) - 24 + bit
    if bits >> bit & 1:
      for _ in range(1 + power % 2):
        row[at] = 2.0**(power // 2)
        at += 1
  return row


def check(x, sums, run, first):
  """run(x) from column `first` on is what it must be if the squares of x's rows add up to `sums`."""
  twins = [powers_of_two(s, x.shape[-1], first) for s in sums]
  known = [i for i, twin in enumerate(twins) if twin is not None]
  assert len(known) >= len(x) // 3
  twins = np.stack([twin if twin is not None else np.ones(x.shape[-1], np.float32) for twin in twins])
  scales = run(twins)[:, first] / twins[:, first]
  assert run(x)[known, first:].tobytes() == (x * scales[:, None])[known, first:].tobytes()


@pytest.mark.parametrize("deviation", [1.0, 1e-3, 300.0])
def test_rms_norm(dev, deviation):
  x, ones = synth.activations(64, 4096, 71) * np.float32(deviation), dev.array(np.ones(4096, np.float32))

  def run(rows):
    y = dev.empty(rows.shape)
    dev.rms_norm(dev.array(rows), ones, len(rows), 4096, y)
    return y.download()

  check(x, row_sums(x), run, 0)


@pytest.mark.parametrize("deviation", [1.0, 1e-2, 30.0])
@pytest.mark.parametrize("offset", [0, 1])  # floats by which the operands miss a 16-byte boundary
def test_heads_of_queries(dev, deviation, offset):
  rows, block_tokens = 8, 16
  x = synth.activations(rows * 16, 256, 72) * np.float32(deviation)
  ones, rope = dev.array(np.ones(256, np.float32)), dev.rope_table(rows)
  k, cache, table = dev.array(np.zeros((rows, 4, 256), np.float32)), [dev.empty((1, 4, block_tokens, 256), np.uint16) for _ in range(2)], dev.array(np.zeros(1, np.int32))
  info = D.Query()
  info.start, info.count, info.position, info.slot, info.state = 0, rows, 0, 0, D.UNBOUND

  def run(heads):
    qg = np.zeros((rows, 16, 512), np.float32)
    qg[:, :, :256] = heads.reshape(rows, 16, 256)
    buffer = dev.array(np.concatenate([np.zeros(offset, np.float32), qg.reshape(-1)]))
    q = dev.empty((rows, 16, 256))
    dev.attention_prepare(type("View", (), {"ptr": buffer.ptr + 4 * offset}), k, k, ones, ones, rope, dev.queries([info]), 1, rows, table, 1, block_tokens, q,
                          *cache)
    return q.download().reshape(-1, 256)

  check(x, head_sums(x), run, 64)
