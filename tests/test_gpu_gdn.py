"""GPU: gated delta-rule layer against the sequential CPU oracle."""
import numpy as np
import pytest

import oracle
from mtlqwen_b200 import device as D
from mtlqwen_b200.testing import images, synth

pytestmark = pytest.mark.gpu
TOL = 1e-3  # BASELINE: GDN outputs within 1e-3 relative error in fp32 accumulation
LAYER = D.GDN_LAYER_STATE_BYTES


def rel_err(got, want):
  want = want.astype(np.float64)
  return float(np.abs(got - want).max() / max(np.abs(want).max(), 1e-30))


def layer_weights(rng):
  return dict(w_beta=(rng.standard_normal((32, 4096)) / 64).astype(np.float32), w_alpha=(rng.standard_normal((32, 4096)) / 64).astype(np.float32),
              ssm_a=(-rng.uniform(1, 16, 32)).astype(np.float32), ssm_dt=(0.1 * rng.standard_normal(32)).astype(np.float32),
              conv=(0.5 * rng.standard_normal((8192, 4))).astype(np.float32), norm=(1 + 0.01 * rng.standard_normal(128)).astype(np.float32))


def run_layer(dev, rng, lengths, fresh=(), speculative=(), prefill=False, fused=False, outputs=None):
  """One GDN layer over len(lengths) queries packed back to back. `fresh` queries start from no state,
  `speculative` ones write one candidate state row per token."""
  w = layer_weights(rng)
  rows, nq = int(sum(lengths)), len(lengths)
  x = rng.standard_normal((rows, 4096)).astype(np.float32)
  mixed = rng.standard_normal((rows, 8192)).astype(np.float32)
  z = rng.standard_normal((rows, 4096)).astype(np.float32)
  conv0 = rng.standard_normal((nq, 8192, 4)).astype(np.float32)
  S0 = (0.01 * rng.standard_normal((nq, 32, 128, 128))).astype(np.float32)
  records = np.concatenate([conv0.reshape(nq, -1), S0.reshape(nq, -1)], axis=1)
  previous = dev.array(records)
  next_ = dev.empty((nq, LAYER // 4))
  candidate_rows = int(sum(lengths[i] for i in speculative))
  candidates = dev.empty((max(candidate_rows, 1), LAYER // 4))
  queries, start, cand = [], 0, 0
  for i, count in enumerate(lengths):
    q = D.Query()
    q.previous = 0 if i in fresh else previous.ptr + i * LAYER
    q.next = candidates.ptr + cand * LAYER if i in speculative else next_.ptr + i * LAYER
    q.start, q.count, q.position, q.slot = start, count, 0 if i in fresh else 77, i
    q.state = cand if i in speculative else D.UNBOUND
    if i in speculative:
      cand += count
    queries.append(q)
    start += count
  dq = dev.queries(queries)
  bufs = {name: dev.array(value) for name, value in w.items()}
  q_out, k_out, v_out = dev.empty((rows, 16, 128)), dev.empty((rows, 16, 128)), dev.empty((rows, 32, 128))
  beta, g, out = dev.empty((rows, 32)), dev.empty((rows, 32)), dev.empty((rows, 32, 128))
  if not fused:
    dev.gdn_prepare(dev.array(x), dev.array(mixed), bufs["w_beta"], bufs["w_alpha"], bufs["ssm_a"], bufs["ssm_dt"], bufs["conv"], dq, nq, rows, 0,
                    LAYER, q_out, k_out, v_out, beta, g)
  # The kernel also writes the quantised image of its output when asked; it must equal the quantisation of `out`.
  image, want_image = dev.empty(dev.image_bytes(rows, 4096), np.uint8), dev.empty(dev.image_bytes(rows, 4096), np.uint8)
  capture = rows < 256 and not prefill  # the prefill variant writes no image
  if capture:
    dev.image_capture(image)
  if fused:  # preparation and recurrence in one launch
    dev.gdn_decode(dev.array(x), dev.array(mixed), bufs["w_beta"], bufs["w_alpha"], bufs["ssm_a"], bufs["ssm_dt"], bufs["conv"], dev.array(z),
                   bufs["norm"], dq, nq, 0, D.CONV_STATE_BYTES, LAYER, out)
  else:
    dev.delta_rule(q_out, k_out, v_out, g, beta, dev.array(z), bufs["norm"], dq, nq, D.CONV_STATE_BYTES, LAYER, out, prefill=prefill)
  dev.quantize(out, rows, 4096, want_image)
  dev.commit()
  if capture:
    for a, b in zip(images.decode(image.download(), rows, 4096), images.decode(want_image.download(), rows, 4096)):
      assert a.tobytes() == b.tobytes()
  got_out, got_next, got_cand = out.download(), next_.download(), candidates.download()
  if outputs is not None:
    outputs.extend([got_out, got_next, got_cand])
  worst, start, cand = 0.0, 0, 0
  for i, count in enumerate(lengths):
    rows_i = slice(start, start + count)
    b, gg = oracle.gdn_ba(x[rows_i], w["w_beta"], w["w_alpha"], w["ssm_a"], w["ssm_dt"])
    spec = i in speculative
    qo, ko, vo, states = oracle.gdn_conv(mixed[rows_i], w["conv"], None if i in fresh else conv0[i], every_token=spec)
    S_init = np.zeros((32, 128, 128), np.float32) if i in fresh else S0[i]
    o, S_final, snaps = oracle.delta_rule(qo, ko, vo, gg, b, S_init, snapshots=spec)
    y = oracle.gated_rms_norm(o, z[rows_i], w["norm"])
    worst = max(worst, rel_err(got_out[rows_i], y))
    if spec:
      for t in range(count):
        rec = got_cand[cand + t]
        worst = max(worst, rel_err(rec[:8192 * 4], states[t].reshape(-1)), rel_err(rec[8192 * 4:], snaps[t].reshape(-1)))
      cand += count
    else:
      rec = got_next[i]
      worst = max(worst, rel_err(rec[:8192 * 4], states[0].reshape(-1)), rel_err(rec[8192 * 4:], S_final.reshape(-1)))
    start += count
  return worst


def test_gdn_decode_eight_sequences(dev):
  assert run_layer(dev, np.random.default_rng(1), [1] * 8) < TOL


def test_gdn_ragged_prefill_config2(dev):
  """8 sequences, ragged chunk lengths uniform in [1, 512], state initialised from N(0, 0.01)."""
  rng = np.random.default_rng(2)
  lengths = [int(v) for v in rng.integers(1, 513, 8)]
  assert run_layer(dev, rng, lengths) < TOL


def test_gdn_mixed_pass_fresh_and_speculative(dev):
  rng = np.random.default_rng(3)
  assert run_layer(dev, rng, [1, 37, 5, 1, 128, 5, 2, 1], fresh=(1, 3), speculative=(2, 5)) < TOL


def test_gdn_preparation_across_row_groups(dev):
  """Query boundaries at every place of the eight-row groups the preparation kernel works in, and a ragged last group."""
  rng = np.random.default_rng(8)
  assert run_layer(dev, rng, [3, 1, 2, 9, 8, 17, 7, 4], fresh=(0, 4), speculative=(3, 7)) < 1e-4


@pytest.mark.parametrize("lengths", [[1], [15], [33, 1, 30], [33, 1, 31], [3, 60, 2, 9, 8, 17, 7, 4]])
def test_gdn_preparation_at_the_line_between_its_forms(dev, lengths):
  """Up to 64 rows a thread has one row and a CTA one head, from 65 on eight of each."""
  rng = np.random.default_rng(sum(lengths))
  assert run_layer(dev, rng, lengths, speculative=(1,) if len(lengths) > 2 else ()) < 1e-4


def test_gdn_single_query_edge_lengths(dev):
  rng = np.random.default_rng(4)
  for lengths in ([1], [2], [3], [4], [512]):
    assert run_layer(dev, rng, lengths, fresh=(0, )) < TOL


def test_gdn_chunked_prefill_config2(dev):
  """The same ragged lengths through infdev_delta_rule_prefill: queries of 16 tokens or more take the chunked kernel."""
  rng = np.random.default_rng(2)
  lengths = [int(v) for v in rng.integers(1, 513, 8)]
  assert run_layer(dev, rng, lengths, prefill=True) < TOL


def test_gdn_chunked_mixed_pass(dev):
  """Chunked, sequential (short or speculative) and fresh queries in one pass; lengths around the 16-token chunk."""
  rng = np.random.default_rng(5)
  assert run_layer(dev, rng, [16, 15, 17, 1, 128, 40, 33, 31], fresh=(0, 4), speculative=(5, ), prefill=True) < TOL


def test_gdn_chunked_agrees_with_sequential(dev):
  """One form is fp32 on the CUDA cores, the other split operands on the tensor cores; both must lie far inside the tolerance
  against the oracle. How close the second one is to fp64: test_chunked_precision."""
  a = run_layer(dev, np.random.default_rng(6), [100, 64], prefill=False)
  b = run_layer(dev, np.random.default_rng(6), [100, 64], prefill=True)
  assert a < TOL and b < TOL and abs(a - b) < 2e-4


def run_rule(dev, q, k, v, g, beta, S0, prefill=True):
  """One query through the recurrence alone (no preparation, no gated norm): outputs and the final state."""
  T = v.shape[0]
  previous, next_, out = dev.array(S0.astype(np.float32)), dev.empty((32, 128, 128)), dev.empty((T, 32, 128))
  info = D.Query()
  info.previous, info.next, info.start, info.count, info.position, info.slot, info.state = previous.ptr, next_.ptr, 0, T, 77, 0, D.UNBOUND
  inputs = [dev.array(np.asarray(a, np.float32)) for a in (q, k, v, g, beta)]
  dev.delta_rule(*inputs, None, None, dev.queries([info]), 1, 0, LAYER, out, prefill=prefill)
  dev.commit()
  return out.download(), next_.download()


def rule_inputs(rng, T, decay=0.05):
  g = -decay * rng.uniform(0.2, 1.8, (T, 32))
  return [rng.standard_normal((T, 16, 128)), rng.standard_normal((T, 16, 128)), rng.standard_normal((T, 32, 128)), g, rng.uniform(0.1, 0.9, (T, 32)),
          0.5 * rng.standard_normal((32, 128, 128))]


@pytest.mark.parametrize("what", ["beta 0, no decay", "fresh state, v 0", "a block of 16 columns", "one column", "a chunk of zeros behind others", "deltas of 1e-36",
                                  "everything 0"])
def test_chunk_whose_deltas_are_zero_leaves_the_state_alone(dev, what):
  """The chunked form scales deltas to the range of fp16: zero ones, or ones far below the state, must not disturb the state."""
  rng = np.random.default_rng(20)
  q, k, v, g, beta, S = rule_inputs(rng, 50)
  if what == "beta 0, no decay":
    beta[16:], g[16:] = 0.0, 0.0
  elif what == "fresh state, v 0":
    S[:], v[:] = 0.0, 0.0
  elif what == "a block of 16 columns":
    S[:, :, 32:48], v[:, :, 32:48] = 0.0, 0.0
  elif what == "one column":
    S[:, :, 77], v[:, :, 77] = 0.0, 0.0
  elif what == "a chunk of zeros behind others":
    q[16:32], k[16:32], v[16:32] = 0.0, 0.0, 0.0
  elif what == "deltas of 1e-36":
    beta[:] *= 1e-36
  else:
    q[:], k[:], v[:], g[:], beta[:], S[:] = 0.0, 0.0, 0.0, 0.0, 0.0, 0.0
  out, state = run_rule(dev, q, k, v, g, beta, S)
  want_out, want_state, _ = oracle.delta_rule(q, k, v, g, beta, S)
  assert np.isfinite(out).all() and np.isfinite(state).all()
  assert rel_err(out, want_out) < 1e-5 and rel_err(state, want_state) < 1e-5


def rule_in_fp64(q, k, v, g, beta, S):
  q, k, v, g, beta, S = (np.asarray(a, np.float32).astype(np.float64) for a in (q, k, v, g, beta, S))
  heads = np.arange(32) % 16
  q = q / np.sqrt((q * q).sum(-1, keepdims=True) + 1e-6) / np.sqrt(128.0)
  k = k / np.sqrt((k * k).sum(-1, keepdims=True) + 1e-6)
  out = []
  for t in range(v.shape[0]):
    S = S * np.exp(g[t])[:, None, None]
    delta = (v[t] - np.einsum("hk,hkv->hv", k[t][heads], S)) * beta[t][:, None]
    S = S + k[t][heads][:, :, None] * delta[:, None, :]
    out.append(np.einsum("hk,hkv->hv", q[t][heads], S))
  return np.stack(out), S


def norm_err(got, want, axes=None):
  return np.sqrt(((got - want)**2).sum(axes) / (want**2).sum(axes)).max()


@pytest.mark.parametrize("what", ["as in a model", "little decay", "columns of very different size", "tokens of very different size"])
def test_chunked_precision(dev, what):
  """Against fp64. Operands are rounded to 22 bits or better (2^-23 of two factors, 2.4e-7 when nothing averages out) and sums to
  fp32: 3e-7 over all, an outer bound of 2e-6 for a value column of its own, whatever its neighbours hold."""
  rng = np.random.default_rng(70)
  T = 160
  q, k, v, g, beta, S = rule_inputs(rng, T, decay=1e-3 if what == "little decay" else 0.2)
  S *= 0.02
  if what == "as in a model":
    g = -np.log1p(np.exp(rng.standard_normal((T, 32)))) * rng.uniform(1, 16, 32)
  elif what == "columns of very different size":
    size = np.exp(4 * rng.standard_normal((32, 128)))
    v, S = v * size, S * size[:, None, :]
  elif what == "tokens of very different size":
    g = -np.log1p(np.exp(rng.standard_normal((T, 32)))) * rng.uniform(1, 16, 32)
    v = v * np.exp(4 * rng.standard_normal((T, 1, 1)))
  out, state = run_rule(dev, q, k, v, g, beta, S)
  want_out, want_state = rule_in_fp64(q, k, v, g, beta, S)
  assert norm_err(state, want_state) < 3e-7 and norm_err(state, want_state, 1) < 2e-6
  if what == "tokens of very different size":
    # an output that is a small difference of large terms keeps few digits in any fp32 form (1.6e-4 of its own size with plain FMAs)
    assert norm_err(out, want_out, 2) < 1e-3
  else:
    assert norm_err(out, want_out) < 3e-7


@pytest.mark.parametrize("T", [17, 32, 33, 49])
def test_first_chunks_have_their_own_decays(dev, T):
  """The preparation of the second chunk may start while the first one's weights are still being formed. Decays of the two differ
  by e^8 here, so that weights formed with the wrong ones would show; and every run gives the same bits."""
  rng = np.random.default_rng(T)
  q, k, v, g, beta, S = rule_inputs(rng, T)
  g[:16], g[16:] = -0.01, -0.5
  want, want_state, _ = oracle.delta_rule(q, k, v, g, beta, S)
  first = None
  for _ in range(20):
    out, state = run_rule(dev, q, k, v, g, beta, S)
    assert rel_err(out, want) < 1e-5 and rel_err(state, want_state) < 1e-5
    first = first or (out.tobytes(), state.tobytes())
    assert first == (out.tobytes(), state.tobytes())


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("where", ["v", "k", "q", "g", "beta"])
def test_tokens_before_one_that_is_not_finite_do_not_notice(dev, where, value):
  """The chunked form computes 16 tokens together; the ones before a broken one must come out as if it were not there."""
  rng = np.random.default_rng(60)
  q, k, v, g, beta, S = rule_inputs(rng, 45)
  clean, _, _ = oracle.delta_rule(q, k, v, g, beta, S)
  token = 27
  if where == "v":
    v[token, 5, 33] = value
  elif where in ("k", "q"):
    (k if where == "k" else q)[token, 5, 33] = value
  else:
    (g if where == "g" else beta)[token, 5] = value
  out, _ = run_rule(dev, q, k, v, g, beta, S)
  assert rel_err(out[:token], clean[:token]) < 1e-5
  others = [h for h in range(32) if h % 16 != 5]
  assert rel_err(out[:, others], clean[:, others]) < 1e-5
  if where == "v":  # one value column of one head
    columns = [c for c in range(128) if c != 33]
    assert rel_err(out[:, 5][:, columns], clean[:, 5][:, columns]) < 1e-5 and not np.isfinite(out[token:, 5, 33]).any()
  elif where != "g" or value != -np.inf:  # (a decay of zero leaves the token itself finite)
    assert not np.isfinite(out[token, 5]).any()


class View:
  """`count` floats of a buffer from float number `offset` on."""

  def __init__(self, dev, values=None, count=0, offset=1):
    self.count, self.offset = count if values is None else values.size, offset
    whole = np.zeros(self.count + 8, np.float32)
    if values is not None:
      whole[offset:offset + self.count] = values.reshape(-1)
    self.buffer = dev.array(whole)
    self.ptr = self.buffer.ptr + 4 * offset

  def download(self):
    return self.buffer.download()[self.offset:self.offset + self.count]


@pytest.mark.parametrize("lengths", [[1], [5, 2, 40], [100, 3]])
@pytest.mark.parametrize("unaligned", ["mixed", "conv", "q", "k", "v"])
def test_preparation_takes_views_at_any_float(dev, lengths, unaligned):
  rng = np.random.default_rng(40)
  rows, nq = sum(lengths), len(lengths)
  w = layer_weights(rng)
  x, mixed = rng.standard_normal((rows, 4096)).astype(np.float32), rng.standard_normal((rows, 8192)).astype(np.float32)
  previous = dev.array(rng.standard_normal((nq, LAYER // 4)).astype(np.float32))
  fixed = {name: dev.array(w[name]) for name in ("w_beta", "w_alpha", "ssm_a", "ssm_dt")}

  def run(offsets):
    next_ = dev.empty((nq, LAYER // 4))
    queries, start = [], 0
    for i, count in enumerate(lengths):
      q = D.Query()
      q.previous, q.next = previous.ptr + i * LAYER, next_.ptr + i * LAYER
      q.start, q.count, q.position, q.slot, q.state = start, count, 77, i, D.UNBOUND
      queries.append(q)
      start += count
    at = lambda name: offsets.get(name, 0)
    out = [View(dev, count=rows * 2048, offset=at("q")), View(dev, count=rows * 2048, offset=at("k")), View(dev, count=rows * 4096, offset=at("v"))]
    beta, g = dev.empty((rows, 32)), dev.empty((rows, 32))
    dev.gdn_prepare(dev.array(x), View(dev, mixed, offset=at("mixed")), fixed["w_beta"], fixed["w_alpha"], fixed["ssm_a"], fixed["ssm_dt"],
                    View(dev, w["conv"], offset=at("conv")), dev.queries(queries), nq, rows, 0, LAYER, *out, beta, g)
    dev.commit()
    return [buffer.download().tobytes() for buffer in (*out, beta, g, next_)]

  want = run({})
  for offset in (1, 2, 3):
    assert run({unaligned: offset}) == want


@pytest.mark.parametrize("between", ["nothing", "rms_norm", "linear"])
def test_steps_follow_each_other_without_a_commit(dev, between):
  """Each decode step reads the records that the step before it wrote, two sets in turn. What lies between two steps lets its
  successor start early; the step must still wait for its records."""
  rng = np.random.default_rng(30)
  w = {name: dev.array(value) for name, value in layer_weights(rng).items()}
  nq, steps = 3, 12
  x, mixed, z = (dev.array(rng.standard_normal((nq, width)).astype(np.float32)) for width in (4096, 8192, 4096))
  norm, small = dev.array(np.ones(4096, np.float32)), dev.array(synth.weight(D.Q4_K, 16, 4096, 31))
  start = np.concatenate([rng.standard_normal((nq, 8192 * 4)), 0.01 * rng.standard_normal((nq, 32 * 128 * 128))], axis=1).astype(np.float32)
  scratch, y, out = dev.empty((nq, 4096)), dev.empty((nq, 16)), dev.empty((nq, 32, 128))

  def run(commit):
    records = [dev.array(start), dev.empty((nq, LAYER // 4))]
    tables = []
    for turn in range(2):
      queries = []
      for i in range(nq):
        q = D.Query()
        q.previous, q.next = records[turn].ptr + i * LAYER, records[1 - turn].ptr + i * LAYER
        q.start, q.count, q.position, q.slot, q.state = i, 1, 77, i, D.UNBOUND
        queries.append(q)
      tables.append(dev.queries(queries))
    for step in range(steps):
      dev.gdn_decode(x, mixed, w["w_beta"], w["w_alpha"], w["ssm_a"], w["ssm_dt"], w["conv"], z, w["norm"], tables[step % 2], nq, 0, D.CONV_STATE_BYTES,
                     LAYER, out)
      if between == "rms_norm":
        dev.rms_norm(x, norm, nq, 4096, scratch)
      elif between == "linear":
        dev.linear(D.Q4_K, small, 16, 4096, x, nq, y)
      if commit:
        dev.commit()
    dev.commit()
    return out.download().tobytes(), records[steps % 2].download().tobytes()

  want = run(True)
  for _ in range(5):
    assert run(False) == want


def test_settled_records_give_the_same_bits(dev):
  lengths, a, b = [1, 3, 1, 2], [], []
  run_layer(dev, np.random.default_rng(32), lengths, speculative=(1, ), fused=True, outputs=a)
  dev.set_settled_records(1)  # every input was uploaded and committed before the step
  try:
    run_layer(dev, np.random.default_rng(32), lengths, speculative=(1, ), fused=True, outputs=b)
  finally:
    dev.set_settled_records(0)
  for x, y in zip(a, b):
    assert x.tobytes() == y.tobytes()


def test_prefill_variant_refuses_an_image(dev):
  dev.image_capture(dev.empty(dev.image_bytes(8, 4096), np.uint8))
  with pytest.raises(RuntimeError, match="no image"):
    dev.delta_rule(dev.empty(1), dev.empty(1), dev.empty(1), dev.empty(1), dev.empty(1), None, None, dev.queries([D.Query()]), 1, 0, LAYER, dev.empty(1),
                   prefill=True)


def test_gdn_fused_decode_is_identical_to_the_two_launches(dev):
  """infdev_gdn_decode = infdev_gdn_prepare + infdev_delta_rule with the same arithmetic: outputs, recurrent states, conv
  taps and speculative candidate records must agree bit for bit, and with the oracle within the tolerance."""
  lengths, fresh, speculative = [1, 1, 5, 1, 3, 1, 1, 2], (1, ), (2, 4)
  a, b = [], []
  assert run_layer(dev, np.random.default_rng(7), lengths, fresh=fresh, speculative=speculative, outputs=a) < TOL
  assert run_layer(dev, np.random.default_rng(7), lengths, fresh=fresh, speculative=speculative, fused=True, outputs=b) < TOL
  for x, y in zip(a, b):
    assert x.tobytes() == y.tobytes()
