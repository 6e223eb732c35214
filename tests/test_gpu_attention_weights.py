"""GPU: the softmax weights of prompt rows, and their results, against 64 bits."""
import numpy as np
import pytest

from mtlqwen_b200 import device as D

pytestmark = pytest.mark.gpu
CONTEXT, ROWS, BLOCK = 2048, 128, 128
BLOCKS = CONTEXT // BLOCK


def attend(dev, q, keys, values, pieces=32):
  """Attention of the last ROWS of CONTEXT tokens, without gates, in up to `pieces` pieces; keys, values: [token, 4, 256]."""
  paged = [np.ascontiguousarray(cache.reshape(BLOCKS, BLOCK, 4, 256).transpose(0, 2, 1, 3)).view(np.uint16) for cache in (keys, values)]
  qg = np.full((ROWS, 16, 512), 60.0, np.float32)  # a sigmoid of 1
  info = D.Query()
  info.start, info.count, info.position, info.slot, info.state = 0, ROWS, CONTEXT - ROWS, 0, D.UNBOUND
  out, partials = dev.empty((ROWS, 16, 256)), dev.empty(dev.attention_scratch_bytes(ROWS, pieces) // 4)
  dev.attention(dev.array(q), dev.array(qg), dev.array(paged[0]), dev.array(paged[1]), dev.queries([info]), 1, ROWS,
                dev.array(np.arange(BLOCKS, dtype=np.int32)[None]), BLOCKS, BLOCK, pieces, partials, out)
  dev.commit()
  return out.download().astype(np.float64)


def test_weights_have_the_accuracy_of_expf(dev):
  """256 tokens are attended to, each alone in a value column, with scores that fp32 holds exactly, the first with a score of 0: the other results divided by
  its own are the weights. From 1/4 to 1/2 they are off by 8.1e-8 (rms; 1.1e-8 on average): the operands' 2^-25, the roundings of result and quotient
  and expf. As powers of two, ex2.approx of a product rounded once, they were off by 8.8e-8 (-3.7e-8)."""
  rng = np.random.default_rng(1)
  keys, values, q = np.zeros((CONTEXT, 4, 256), np.float16), np.zeros((CONTEXT, 4, 256), np.float16), np.zeros((ROWS, 16, 256), np.float32)
  seen = np.concatenate([[0], 1 + rng.permutation(CONTEXT - ROWS - 1)[:255]])
  factor, scale = -rng.uniform(0, 1, 256).astype(np.float16), rng.uniform(1, 64, (ROWS, 16)).astype(np.float16)
  factor[0] = 0
  keys[:, :, 0], q[:, :, 0] = -1000.0, scale
  keys[seen, :, 0], values[seen, :, np.arange(256)] = factor[:, None], 1.0
  got = attend(dev, q, keys, values, 1)
  want = np.exp(scale.astype(np.float64)[:, :, None] * factor.astype(np.float64) / 16)
  error = (got / got[..., :1] / want - 1)[(want >= 0.25) & (want < 0.5)]
  assert error.size > 100000
  assert np.sqrt((error**2).mean()) <= 8.4e-8 and abs(error.mean()) <= 2.4e-8


@pytest.mark.parametrize("scale", [1, 4])  # weights of all tokens alike, and of few above the others
def test_results_against_64_bits(dev, scale):
  """Off by 1.4e-6 and 1.8e-6: what the tensor cores cut from sums of up to 2048 products."""
  rng = np.random.default_rng(3)
  keys, values = (rng.standard_normal((CONTEXT, 4, 256)).astype(np.float16) for _ in range(2))
  q = (scale * rng.standard_normal((ROWS, 16, 256))).astype(np.float32)
  got, want = attend(dev, q, keys, values), np.empty((ROWS, 16, 256))
  ahead = np.arange(CONTEXT)[None] > CONTEXT - ROWS + np.arange(ROWS)[:, None]
  for head in range(16):
    score = q[:, head].astype(np.float64) @ keys[:, head // 4].astype(np.float64).T / 16
    score[ahead] = -np.inf
    weight = np.exp(score - score.max(axis=1, keepdims=True))
    want[:, head] = weight / weight.sum(axis=1, keepdims=True) @ values[:, head // 4].astype(np.float64)
  assert np.linalg.norm(got - want) <= 2.2e-6 * np.linalg.norm(want)
