"""GPU: the block formats of the real Qwen3.5 GGUF files beyond Q4_K / Q6_K - Q5_K, Q8_0, IQ4_XS, F16 - through
dequantisation (bit-exact against the gguf-py golden vectors), the linear and gate / up kernels, the embedding gather,
and a whole reduced model that mixes all of them, against the CPU oracle."""
from pathlib import Path

import numpy as np
import pytest

import oracle
from mtlqwen_b200 import device as D
from mtlqwen_b200.inference import InferenceEngine
from mtlqwen_b200.testing import synth

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden" / "kquant_dequant.npz"
TYPES = [("q5k", D.Q5_K), ("q8_0", D.Q8_0), ("iq4xs", D.IQ4_XS)]
TOL = 1e-3  # BASELINE tolerance for GEMV / GEMM; these kernels accumulate in fp32 and measure about 1e-6


def rel_err(got, want):
  want64 = want.astype(np.float64)
  return float(np.abs(got - want64).max() / np.abs(want64).max())


@pytest.mark.parametrize("name,qtype", TYPES)
def test_dequant_bit_exact_against_golden(dev, name, qtype):
  golden = np.load(GOLDEN)
  blocks, want = golden[name + "_blocks"], golden[name + "_values"]
  out = dev.empty(want.shape)
  dev.dequant(qtype, dev.array(blocks), blocks.shape[0], out)
  assert out.download().tobytes() == want.tobytes()


def test_f16_rows_widen_exactly(dev):
  values = (np.random.default_rng(0).standard_normal(32 * 4096) / 64).astype(np.float16)
  out = dev.empty(values.size)
  dev.dequant(D.F16, dev.array(values.view(np.uint8)), values.size // 256, out)
  assert out.download().tobytes() == values.astype(np.float32).tobytes()


@pytest.mark.parametrize("name,qtype", TYPES)
@pytest.mark.parametrize("n,k,m", [(1024, 4096, 1), (520, 8192, 8), (256, 12288, 21)])
def test_linear_matches_oracle(dev, name, qtype, n, k, m):
  w, x, res = synth.weight(qtype, n, k, 60), synth.activations(m, k, 61), synth.activations(m, n, 62)
  y = dev.array(res)
  dev.linear(qtype, dev.array(w), n, k, dev.array(x), m, y, y)  # residual aliases the result, as in the decoder
  assert rel_err(y.download(), oracle.linear(w, qtype, n, k, x, res)) < 1e-5


@pytest.mark.parametrize("name,qtype", TYPES + [("q6k", D.Q6_K)])
@pytest.mark.parametrize("n,k,m", [(16, 2048, 1), (2400, 2048, 3), (48, 10240, 8), (16, 256, 2), (32, 1536, 7), (160, 1280, 5), (24, 4096, 4)])
def test_tensor_core_gemv_edges(dev, name, qtype, n, k, m):
  """One tile, more tiles than SMs with a ragged last round, a last K chunk of one stage, rows shorter than a stage, and
  shapes the tensor-core kernel leaves to the plain one (n not a multiple of 16, rows that are not 16-byte aligned). The
  activations span what fp32 holds and fp16 does not: the kernel scales every (row, super-block) by a power of two."""
  if qtype == D.Q6_K and (k % 2048 or n % 16):
    pytest.skip("Q6_K takes rows of whole 2048-value spans and tiles of 16 rows")
  w, x = synth.weight(qtype, n, k, 63), synth.activations(m, k, 64)
  x[:, :256] *= 1.0e6
  x[m - 1] *= 1.0e-9
  y = dev.empty((m, n))
  dev.linear(qtype, dev.array(w), n, k, dev.array(x), m, y)
  got, want = y.download(), oracle.linear(w, qtype, n, k, x)
  for row in range(m):  # row by row: their magnitudes differ by fifteen orders
    assert rel_err(got[row], want[row]) < 1e-5, row


@pytest.mark.parametrize("name,qtype", TYPES)
def test_gate_up_matches_oracle(dev, name, qtype):
  n, k, m = 768, 4096, 5
  wg, wu, x = synth.weight(qtype, n, k, 70), synth.weight(qtype, n, k, 71), synth.activations(m, k, 72)
  y = dev.empty((m, n))
  dev.gate_up(qtype, dev.array(wg), dev.array(wu), n, k, dev.array(x), m, y)
  assert rel_err(y.download(), oracle.gate_up(wg, wu, qtype, n, k, x)) < 1e-5


WIDE_TYPES = [*TYPES, ("q6_k", D.Q6_K)]


@pytest.mark.parametrize("m,n,k", [(9, 16, 2048), (16, 4096, 4096), (17, 208, 6144), (24, 1024, 2048), (33, 48, 12288), (40, 2512, 4096), (43, 96, 2048),
                                   (56, 160, 4096), (64, 4096, 4096), (65, 16, 2048), (128, 1040, 12288), (131, 64, 4096), (137, 32, 2048),
                                   (15, 21008, 2048), (40, 21008, 2048)])
@pytest.mark.parametrize("name,qtype", WIDE_TYPES)
def test_many_rows_share_a_decode(dev, name, qtype, m, n, k):
  """9 rows and up: every tile count, the last tile of a row group partly filled, tiles fewer and several times more than all warps, K in
  one chunk, several chunks and several slices; with a residual that the result overwrites. 22-bit activations, exact quants
  and fp32 sums as with up to eight rows, so the bound is that of the calls above."""
  w, x, y = synth.weight(qtype, n, k, 90), synth.activations(m, k, 91), synth.activations(m, n, 92)
  x[m - 1] *= 1.0e6
  x[m // 2] *= 1.0e-9
  buffer = dev.array(y)
  dev.linear(qtype, dev.array(w), n, k, dev.array(x), m, buffer, buffer)
  got, want = buffer.download() - y, oracle.linear(w, qtype, n, k, x)
  # adding the residual rounds to its own last place: 1.2e-7 of it beside the products' bound
  for row in range(m):
    assert np.linalg.norm(got[row] - want[row]) < 1e-5 * np.linalg.norm(want[row]) + 2.4e-7 * np.linalg.norm(y[row]), row


@pytest.mark.parametrize("m,n,k", [(16, 2368, 2048), (16, 2384, 2048), (17, 32, 2048), (9, 32, 4096), (16, 32, 2304)])
@pytest.mark.parametrize("name,qtype", WIDE_TYPES)
def test_either_side_of_the_line_to_the_slices(dev, name, qtype, m, n, k):
  """Up to 16 rows of a matrix with few tiles and K of 2048 at the most go through the GEMV in two slices."""
  if qtype == D.Q6_K and k % 2048:
    pytest.skip("Q6_K takes rows of whole 2048-value spans")
  w, x = synth.weight(qtype, n, k, 87), synth.activations(m, k, 88)
  y = dev.empty((m, n))
  dev.linear(qtype, dev.array(w), n, k, dev.array(x), m, y)
  assert rel_err(y.download(), oracle.linear(w, qtype, n, k, x)) < 1e-5


@pytest.mark.parametrize("m", [1, 8, 24, 40])
@pytest.mark.parametrize("k", [2048, 6144])
@pytest.mark.parametrize("name,qtype", WIDE_TYPES)
def test_linear_precision(dev, name, qtype, m, k):
  """Against fp64 over the exact weights. Activations are rounded to 22 bits, products are exact, sums fp32: 1.8e-7 over all,
  about what fp32 multiply-adds give (1.5e-7 at K = 2048, 2.1e-7 at 4096)."""
  n = 1024
  w, x = synth.weight(qtype, n, k, 85), synth.activations(m, k, 86)
  y = dev.empty((m, n))
  dev.linear(qtype, dev.array(w), n, k, dev.array(x), m, y)
  want = x.astype(np.float64) @ oracle.dequant(w, qtype).reshape(n, k).astype(np.float64).T
  assert np.linalg.norm(y.download() - want) < 1.8e-7 * np.linalg.norm(want)


@pytest.mark.parametrize("m", [3, 8, 9, 40])
@pytest.mark.parametrize("name,qtype", WIDE_TYPES)
def test_activations_at_the_ends_of_the_range(dev, name, qtype, m):
  """Rows that fp32 only just holds, whose power of two and its inverse must stay normal numbers; and rows with one infinite
  activation, whose results are infinite with the sign of its weight, beside finite rows that must not notice."""
  n, k = 64, 4096
  w, x = synth.weight(qtype, n, k, 97), synth.activations(m, k, 98)
  x[0] *= 3.0e-37
  x[1, 300] = np.inf
  x[2, 4095], x[2, 100] = -np.inf, 1.0e30
  y = dev.empty((m, n))
  dev.linear(qtype, dev.array(w), n, k, dev.array(x), m, y)
  with np.errstate(all="ignore"):
    got, want = y.download(), oracle.linear(w, qtype, n, k, x)
  assert not np.isfinite(want[1:3]).any() and np.array_equal(got[1:3], want[1:3], equal_nan=True)
  for row in [0, *range(3, m)]:
    assert rel_err(got[row], want[row]) < 1e-5, row


@pytest.mark.parametrize("m", [11, 40, 100, 128])
@pytest.mark.parametrize("name,qtype", TYPES)
def test_many_rows_of_a_pair_and_of_a_group(dev, name, qtype, m):
  n, k = 768, 4096
  wg, wu, x = synth.weight(qtype, n, k, 93), synth.weight(qtype, n, k, 94), synth.activations(m, k, 95)
  y, z = dev.empty((m, n)), dev.empty((m, n))
  dev.gate_up(qtype, dev.array(wg), dev.array(wu), n, k, dev.array(x), m, y)
  assert rel_err(y.download(), oracle.gate_up(wg, wu, qtype, n, k, x)) < 1e-5
  dev.linear_group(qtype, [dev.array(wg), dev.array(wu)], [n, n], k, dev.array(x), m, [y, z])
  assert rel_err(y.download(), oracle.linear(wg, qtype, n, k, x)) < 1e-5
  assert rel_err(z.download(), oracle.linear(wu, qtype, n, k, x)) < 1e-5


@pytest.mark.parametrize("name,qtype", TYPES)
def test_embedding_rows_are_the_oracle_rows(dev, name, qtype):
  n, k, ids = 96, 4096, np.array([0, 95, 7, 7, 41], np.int32)
  table = synth.weight(qtype, n, k, 80)
  out = dev.empty((ids.size, k))
  dev.embedding(qtype, dev.array(table), k, dev.array(ids), ids.size, out)
  assert out.download().tobytes() == oracle.embedding(table, qtype, k, ids).tobytes()


def test_model_with_the_type_mix_of_the_real_files_matches_the_oracle(tmp_path):
  """A reduced model (4 layers + MTP block) whose projections cycle through Q4_K, Q5_K, IQ4_XS, Q6_K and Q8_0, with a
  Q4_K embedding table, F16 ssm_beta / ssm_alpha and a Q8_0 eh_proj: greedy tokens teacher-forced against the oracle
  (margin rule), through a prefill of more than 8 rows and decode steps, with the MTP tail running."""
  layers, vocab = 4, 4096
  path = tmp_path / "mixed.gguf"
  synth.write_gguf(path, layers=layers, vocab=vocab, mtp=True, seed=17, mixed=True)
  tensors = synth.read_gguf(path)
  kinds = {kind for _, kind in tensors.values()}
  assert {D.Q4_K, D.Q5_K, D.Q6_K, D.Q8_0, D.IQ4_XS, D.F16, D.F32} <= kinds
  engine = InferenceEngine(path, draft_weights=path, max_context=256)
  try:
    prompt = [int(t) for t in np.random.default_rng(2).integers(0, vocab, 45)]
    sequence = engine.sequence()
    cursor, generated = sequence.append(prompt), []
    while len(generated) < 14:
      generated.append(sequence.read(cursor))
      cursor += 1
    sequence.cancel()
    sequence.close()
    reference = oracle.Model(tensors, layers, vocab, 256)
    _, logits = reference.forward(prompt, 1)
    checked = 0
    for index, token in enumerate(generated):
      expected, margin = oracle.sample(logits[-1] if logits.ndim == 2 else logits)
      if margin > 1e-2:
        assert token == expected, (index, margin)
        checked += 1
      _, logits = reference.step(token)
    assert checked >= 10
  finally:
    engine.close()
