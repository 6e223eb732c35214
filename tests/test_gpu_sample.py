"""GPU: on-device sampling against the CPU oracle (greedy, top-k/top-p/temperature, plain temperature)."""
import numpy as np
import pytest

import oracle
from mtlqwen_b200 import device as D

pytestmark = pytest.mark.gpu
VOCAB = 248320


def make_queries(params, seed=1234, position=41):
  queries, logit = [], 0
  for slot, (temperature, top_p, top_k, samples) in enumerate(params):
    q = D.Query()
    q.start, q.count, q.position, q.slot, q.state = logit, samples, position, slot, D.UNBOUND
    q.logit, q.samples, q.temperature, q.topP, q.topK, q.seed = logit, samples, temperature, top_p, top_k, seed + slot
    queries.append(q)
    logit += samples
  return queries, logit


def expected(logits, queries):
  out = []
  for q in queries:
    for s in range(q.samples):
      u = oracle.uniform(q.seed, q.position + q.count - q.samples + s + 1)
      out.append(oracle.sample(logits[q.logit + s], q.temperature, q.topP, q.topK, u)[0])
  return out


def test_greedy_matches_first_index_argmax(dev):
  rng = np.random.default_rng(0)
  logits = (1.3 * rng.standard_normal((8, VOCAB))).astype(np.float32)
  logits[3, 1000] = logits[3, 2000] = 9.5  # a tie: the first index wins
  queries, count = make_queries([(0.0, 1.0, 0, 1)] * 8)
  tokens = dev.empty(count, np.int32)
  dev.sample(dev.array(logits), VOCAB, dev.queries(queries), len(queries), count, 0, tokens)
  got = tokens.download().tolist()
  assert got == expected(logits, queries)
  assert got[3] == 1000


def test_top_k_top_p_temperature_config5(dev):
  """BASELINE config 5 sampling: temperature 0.7, top-p 0.9, top-k 40, seeded per-slot RNG."""
  rng = np.random.default_rng(1)
  logits = (1.3 * rng.standard_normal((40, VOCAB))).astype(np.float32)
  queries, count = make_queries([(0.7, 0.9, 40, 5)] * 8)
  tokens = dev.empty(count, np.int32)
  dev.sample(dev.array(logits), VOCAB, dev.queries(queries), len(queries), count, 0, tokens)
  assert tokens.download().tolist() == expected(logits, queries)


def test_mixed_sampling_parameters(dev):
  rng = np.random.default_rng(2)
  logits = (2.0 * rng.standard_normal((8, VOCAB))).astype(np.float32)
  params = [(1.0, 1.0, 1, 1), (0.0, 1.0, 0, 1), (1.5, 0.5, 64, 1), (0.3, 0.95, 200, 1), (1.0, 1.0, 0, 1), (0.7, 0.0, 40, 1), (2.0, 1.0, 8, 1),
            (1.0, 0.9, 0, 1)]
  queries, count = make_queries(params)
  tokens = dev.empty(count, np.int32)
  dev.sample(dev.array(logits), VOCAB, dev.queries(queries), len(queries), count, 0, tokens)
  got, want = tokens.download().tolist(), expected(logits, queries)
  # top_k = 1 is greedy whatever the temperature (test_mixed_batch_sampling_matches_greedy of the reference)
  assert got[0] == int(np.argmax(logits[0]))
  for i, (g, w) in enumerate(zip(got, want)):
    if params[i][2] == 0 and params[i][0] > 0:
      # full-vocabulary sampling sums 248k terms in a different order than the serial oracle: accept the
      # neighbour when the target falls within rounding of a boundary
      assert abs(g - w) <= 1, (i, g, w)
    else:
      assert g == w, (i, g, w)


def test_ties_at_the_top_k_cut_keep_the_earliest_indices(dev):
  logits = np.full((1, VOCAB), -5.0, np.float32)
  logits[0, [10, 20, 30]] = [3.0, 2.0, 1.0]
  queries, count = make_queries([(1.0, 1.0, 8, 1)])
  tokens = dev.empty(count, np.int32)
  dev.sample(dev.array(logits), VOCAB, dev.queries(queries), 1, count, 0, tokens)
  assert tokens.download().tolist() == expected(logits, queries)


@pytest.mark.parametrize("vocab", [64, 1003, 4096, 16388])
def test_small_and_odd_vocabularies(dev, vocab):
  """Fewer logits than the cluster has threads, a length that no vector load fits, and parts of uneven size."""
  rng = np.random.default_rng(vocab)
  logits = (2.0 * rng.standard_normal((6, vocab))).astype(np.float32)
  logits[1, [vocab - 1, vocab - 2]] = 12.0  # a tie in the last part
  queries, count = make_queries([(0.0, 1.0, 0, 1), (0.0, 1.0, 0, 1), (0.7, 0.9, 40, 1), (1.2, 1.0, 64, 1), (0.9, 0.8, 1, 1), (0.5, 0.0, 3, 1)])
  tokens = dev.empty(count, np.int32)
  dev.sample(dev.array(logits), vocab, dev.queries(queries), len(queries), count, 0, tokens)
  assert tokens.download().tolist() == expected(logits, queries)


def test_more_ties_than_the_collection_holds(dev):
  """3000 logits share the largest value but one: the row takes the radix select, and the earliest of them are kept."""
  logits = np.full((2, VOCAB), -5.0, np.float32)
  logits[:, 5000:8000], logits[:, 100000] = 2.0, 3.0
  queries, count = make_queries([(0.7, 1.0, 40, 1), (1.0, 0.95, 64, 1)])
  tokens = dev.empty(count, np.int32)
  dev.sample(dev.array(logits), VOCAB, dev.queries(queries), len(queries), count, 0, tokens)
  assert tokens.download().tolist() == expected(logits, queries)


@pytest.mark.parametrize("rows,vocab", [(18, 16384), (19, 16384), (37, 8200), (40, 8192), (75, 4096), (150, 4099), (3, 4095), (2, 130)])
def test_every_number_of_ctas_for_a_row(dev, rows, vocab):
  """Rows share the SMs: eight CTAs for a row of a few, four, two, one of many, and no more than the vocabulary keeps busy."""
  rng = np.random.default_rng(rows)
  logits = (2.0 * rng.standard_normal((rows, vocab))).astype(np.float32)
  params = [(0.0, 1.0, 0, 1), (0.7, 0.9, 40, 1), (1.3, 1.0, 64, 1), (1.0, 0.8, 1, 1), (0.9, 1.0, 0, 1)]
  queries, count = make_queries([params[i % len(params)] for i in range(rows)])
  tokens = dev.empty(count, np.int32)
  dev.sample(dev.array(logits), vocab, dev.queries(queries), len(queries), count, 0, tokens)
  assert tokens.download().tolist() == expected(logits, queries)


@pytest.mark.parametrize("masked", [-np.inf, np.finfo(np.float32).min, -1.0e9])
@pytest.mark.parametrize("temperature", [0.7, 1.0, 1.5])
@pytest.mark.parametrize("live", [0, 3, 200])
def test_masked_rows(dev, masked, temperature, live):
  """A mask leaves few logits, or none: the threshold is the masked value itself (or its overflow), and the earliest equal ones
  fill the set up."""
  rng = np.random.default_rng(live)
  vocab = 20000
  logits = np.full((5, vocab), masked, np.float32)
  for row in logits:
    where = rng.choice(vocab, live, replace=False)
    row[where] = rng.standard_normal(live)
  queries, count = make_queries([(temperature, 1.0, 40, 1), (temperature, 0.9, 64, 1), (temperature, 0.0, 8, 1), (temperature, 1.0, 1, 1), (0.0, 1.0, 0, 1)])
  tokens = dev.empty(count, np.int32)
  dev.sample(dev.array(logits), vocab, dev.queries(queries), len(queries), count, 0, tokens)
  assert tokens.download().tolist() == expected(logits, queries)


@pytest.mark.parametrize("step", [0.5, 1.0, 4.0])
def test_coarse_logits_tie_everywhere(dev, step):
  rng = np.random.default_rng(9)
  logits = (step * np.round(1.5 * rng.standard_normal((6, VOCAB)) / step)).astype(np.float32)
  queries, count = make_queries([(0.7, 0.9, 40, 1), (1.0, 1.0, 64, 1), (1.9, 1.0, 5, 1), (0.3, 1.0, 1, 1), (3.0, 1.0, 64, 1), (0.0, 1.0, 0, 1)])
  tokens = dev.empty(count, np.int32)
  dev.sample(dev.array(logits), VOCAB, dev.queries(queries), len(queries), count, 0, tokens)
  assert tokens.download().tolist() == expected(logits, queries)


@pytest.mark.parametrize("value", [np.nan, -np.nan])
def test_nan_logits_beside_more_ties_than_the_collection_holds(dev, value):
  """A NaN takes part in no comparison: the row samples as if it were not there, also where ties send it through the radix select."""
  logits = np.full((1, VOCAB), -5.0, np.float32)
  logits[0, 5000:8000], logits[0, 100000] = 2.0, 3.0
  clean = logits.copy()
  clean[0, [3, 700, 6001]], logits[0, [3, 700, 6001]] = -1.0e30, value
  for seed in range(8):
    queries, count = make_queries([(1.5, 1.0, 40, 1)])
    queries[0].seed = seed
    tokens = dev.empty(count, np.int32)
    dev.sample(dev.array(logits), VOCAB, dev.queries(queries), len(queries), count, 0, tokens)
    assert tokens.download().tolist() == expected(clean, queries)


# ---- draft verification on the device against the host loop of the reference ----
def host_acceptance(samples, speculative, sampled, proposals, draft_width, stops):
  """runtime/engine.cpp:205-216 for one query: returns (accepted, emitted, stopped)."""
  accepted, emitted, stopped = 0, 0, False
  for i in range(samples):
    if stopped:
      break
    token = sampled[i]
    emitted += 1
    stopped = token in stops
    if not speculative or i == draft_width or token != proposals[i]:
      break
    accepted += 1
  return accepted, emitted, int(stopped)


def test_verify_drafts_and_commit_states_follow_the_reference_loop(dev):
  """Six queries in one pass, draft width 4: full acceptance (stops at s == width), mismatch at proposal 0, a stop
  token inside an accepted draft (it is emitted, counted when it matches, and ends the query), a plain decode
  row, a prefill chunk without a sample, and a mismatch in the middle. The accepted candidate state row of each
  speculative query must land in the slot's next state record."""
  width, stride = 4, 64
  cases = [  # (speculative, sampled rows, proposals, stop tokens)
    (True, [11, 12, 13, 14, 15], [11, 12, 13, 14], []),
    (True, [21, 22, 23, 24, 25], [99, 22, 23, 24], []),
    (True, [31, 32, 33, 34, 35], [31, 32, 33, 34], [32]),
    (False, [41], [0, 0, 0, 0], [41]),
    (False, [], [0, 0, 0, 0], []),
    (True, [51, 52, 53, 54, 55], [51, 52, 77, 54], [7, 8, 9]),
  ]
  state_bytes = 4096
  queries, sampled, logit, candidate = [], [], 0, 0
  proposed = np.zeros((width + 1, 8), np.int32)
  stops, counts = np.zeros((8, stride), np.int32), np.zeros(8, np.uint32)
  for slot, (speculative, rows, proposals, stop) in enumerate(cases):
    q = D.Query()
    q.slot, q.position, q.count, q.samples, q.logit = slot, 100 + slot, max(len(rows), 1) if rows else 7, len(rows), logit
    q.state = candidate if speculative else D.UNBOUND
    if speculative:
      proposed[1:, candidate // q.count] = proposals  # column = first candidate row / rows per query, as the engine packs them
      candidate += q.count
    stops[slot, :len(stop)], counts[slot] = stop, len(stop)
    sampled += rows
    logit += len(rows)
    queries.append(q)
  rng = np.random.default_rng(3)
  candidates = rng.integers(0, 2**31, (candidate, state_bytes // 4), dtype=np.int64).astype(np.uint32)
  following = dev.empty((8, state_bytes // 4), np.uint32)
  next_addresses = np.array([following.ptr + slot * state_bytes for slot in range(8)], np.uint64)
  candidate_buffer = dev.array(candidates)
  device_queries, verdict = dev.queries(queries), dev.empty(3 * len(queries), np.uint32)
  dev.verify_drafts(device_queries, len(queries), dev.array(np.array(sampled, np.int32)), dev.array(proposed), width, dev.array(stops), stride,
                    dev.array(counts), verdict)
  dev.commit_states(device_queries, len(queries), verdict, dev.array(next_addresses), candidate_buffer.ptr, state_bytes)
  dev.commit()
  got = verdict.download().reshape(-1, 3).tolist()
  want = [list(host_acceptance(len(rows), speculative, rows, proposals, width, stop)) for speculative, rows, proposals, stop in cases]
  assert got == want
  assert want[0] == [4, 5, 0] and want[1] == [0, 1, 0] and want[2] == [2, 2, 1] and want[3] == [0, 1, 1] and want[4] == [0, 0, 0]
  states = following.download()
  for q, (accepted, _, _) in zip(queries, want):
    if q.state != D.UNBOUND:
      assert np.array_equal(states[q.slot], candidates[q.state + accepted]), q.slot


# chunks of one logit less, as many and one more than the 256 that a warp asks for at once, with eight CTAs for a row; 300 and 17 with one
@pytest.mark.parametrize("rows,vocab", [(16, 1024 * 255), (16, 1024 * 256), (16, 1024 * 256 + 7), (150, 128 * 300 - 5), (150, 2100)])
def test_chunks_of_plain_temperature_sampling(dev, rows, vocab):
  rng = np.random.default_rng(vocab)
  logits = (2.0 * rng.standard_normal((rows, vocab))).astype(np.float32)
  queries, count = make_queries([(0.9, 1.0, 0, 1)] * rows)
  tokens = dev.empty(count, np.int32)
  dev.sample(dev.array(logits), vocab, dev.queries(queries), len(queries), count, 0, tokens)
  got, sure = tokens.download().tolist(), 0
  for row, (token, q) in enumerate(zip(got, queries)):
    # the weights' exponents as the kernel rounds them, everything else in 64 bits: weights off by 2^-23 each move the sums by less than 1e-7 of the whole
    exponent = logits[row] / np.float32(q.temperature) - logits[row].max() / np.float32(q.temperature)
    sums = np.cumsum(np.exp(exponent.astype(np.float64)))
    target = float(oracle.uniform(q.seed, q.position + q.count - q.samples + 1)) * sums[-1]
    want = int(np.searchsorted(sums, target))
    clear = np.abs(sums[max(want - 1, 0):want + 1] - target).min() > 1e-7 * sums[-1]  # no boundary within rounding of the target
    sure += clear
    assert token == want if clear else abs(token - want) <= 1, row
  assert sure >= 3 * rows // 4
