"""GPU: the chunked gated delta rule with a head's value columns on one CTA or on two, by the number of chunked queries."""
import numpy as np
import pytest

from mtlqwen_b200 import device as D
from test_gpu_gdn import LAYER

pytestmark = pytest.mark.gpu
STATE = 32 * 128 * 128


class Pass:
  def __init__(self, dev, lengths, seed=51):
    rng = np.random.default_rng(seed)
    rows, self.dev, self.lengths = sum(lengths), dev, lengths
    draw = lambda *shape: rng.standard_normal(shape).astype(np.float32)
    self.host = {"q": draw(rows, 16, 128), "k": draw(rows, 16, 128), "v": draw(rows, 32, 128), "z": draw(rows, 32, 128),
                 "g": -np.abs(draw(rows, 32)), "beta": 1 / (1 + np.exp(-draw(rows, 32)))}
    self.previous, self.norm = (0.1 * draw(len(lengths), STATE)).astype(np.float32), dev.array(1 + 0.01 * draw(128))

  def run(self, chosen, speculative=(), in_place=False):
    """[(outputs, state) of each chosen query], in one pass of these alone."""
    dev, queries, start, at = self.dev, [], 0, np.concatenate([[0], np.cumsum(self.lengths)])
    pick = np.concatenate([np.arange(at[i], at[i + 1]) for i in chosen])
    buffers = {name: dev.array(np.ascontiguousarray(value[pick])) for name, value in self.host.items()}
    records = sum(self.lengths[i] if i in speculative else 1 for i in chosen)
    previous, next_, record, places = dev.array(self.previous[list(chosen)]), dev.empty((records, STATE)), 0, []
    for slot, i in enumerate(chosen):
      q = D.Query()
      q.previous, q.next = previous.ptr + slot * STATE * 4, next_.ptr + record * STATE * 4
      q.start, q.count, q.position, q.slot, q.state = start, self.lengths[i], 77, slot, (record if i in speculative else D.UNBOUND)
      queries.append(q)
      places.append((start, record))
      start += self.lengths[i]
      record += self.lengths[i] if i in speculative else 1
    out = buffers["z"] if in_place else dev.empty((start, 32, 128))
    dev.delta_rule(buffers["q"], buffers["k"], buffers["v"], buffers["g"], buffers["beta"], buffers["z"], self.norm, dev.queries(queries), len(chosen), 0,
                   STATE * 4, out, prefill=True)
    dev.commit()
    outputs, states = out.download().reshape(start, 32, 128), next_.download()
    return [(outputs[s:s + self.lengths[i]], states[r]) for i, (s, r) in zip(chosen, places)]


@pytest.fixture()
def mixed(dev):
  assert LAYER > STATE * 4
  return Pass(dev, [40, 100, 17, 1, 5, 20, 16, 15])


def same(a, b):
  return a[0].tobytes() == b[0].tobytes() and a[1].tobytes() == b[1].tobytes()


def test_one_cta_or_two_have_the_same_bits(mixed):
  """One and two chunked queries are split (64 heads' halves on up to 148 SMs), three are not; short ones do not count."""
  alone = {i: mixed.run([i])[0] for i in range(8)}
  for chosen in ([0, 1], [3, 0, 4], [0, 1, 2], [7, 1, 3, 2, 4], [0, 1, 2, 3, 4, 5, 6, 7]):
    for i, got in zip(chosen, mixed.run(chosen)):
      assert same(got, alone[i]), (chosen, i)


def test_speculative_queries_are_not_counted_however_long(mixed):
  """Longer than the chunked ones, they must not take the places of their halves."""
  alone = {i: mixed.run([i])[0] for i in (2, 6)}
  for chosen in ([1, 0, 2, 6], [2, 1, 6]):
    got = dict(zip(chosen, mixed.run(chosen, speculative=(0, 1))))
    assert same(got[2], alone[2]) and same(got[6], alone[6])


def test_outputs_over_the_gates(mixed):
  for i in (0, 1, 3):
    (apart, state), (over, other) = mixed.run([i])[0], mixed.run([i], in_place=True)[0]
    # the norm's sum of 128 squares in another order: 7 roundings of it, half as many of its root, and the three products'
    assert np.linalg.norm(apart - over) <= 7 * 2.0 ** -24 * np.linalg.norm(apart) and state.tobytes() == other.tobytes()


@pytest.mark.parametrize("chosen", [[0], [1], [6], [0, 1], [0, 1, 2], [3, 0, 4, 5, 7]])  # whole and short last chunks, one CTA a head and two, short queries beside
def test_outputs_over_the_gates_have_the_same_bits(mixed, chosen):
  """The norm in the chain and the one behind it add the squares in one order."""
  for i, apart, over in zip(chosen, mixed.run(chosen), mixed.run(chosen, in_place=True)):
    assert same(apart, over), i


def test_the_norm_on_one_cta_or_on_eight_has_the_same_bits(dev):
  """28 queries leave a head of each one CTA for its norms; a query alone has eight of 64 rows at a time, the longest here one row more than they
  take at once."""
  lengths = [513, 64, 65, 1] + [16] * 24
  everything = Pass(dev, lengths, seed=52)
  together = everything.run(range(len(lengths)))
  for i in range(5):
    assert same(everything.run([i])[0], together[i]), lengths[i]


def test_as_many_queries_as_a_grid_has_rows(dev):
  """65535 queries, all of them the same row and record, beside each of which nothing more fits into the grid."""
  rng, count = np.random.default_rng(53), 65535
  draw = lambda *shape: dev.array(rng.standard_normal(shape).astype(np.float32))
  q, k, v, z, g, beta, norm, previous, next_ = draw(1, 16, 128), draw(1, 16, 128), draw(1, 32, 128), draw(1, 32, 128), dev.array(np.full((1, 32), -0.1, np.float32)), \
    dev.array(np.full((1, 32), 0.5, np.float32)), draw(128), draw(1, STATE), dev.empty((1, STATE))
  query = D.Query()
  query.previous, query.next, query.start, query.count, query.position, query.slot, query.state = previous.ptr, next_.ptr, 0, 1, 77, 0, D.UNBOUND
  results = []
  for queries in ([query], [query] * count):
    out = dev.empty((1, 32, 128))
    dev.delta_rule(q, k, v, g, beta, z, norm, dev.queries(queries), len(queries), 0, STATE * 4, out, prefill=True)
    dev.commit()
    results.append((out.download().tobytes(), next_.download().tobytes()))
  assert results[0] == results[1]
