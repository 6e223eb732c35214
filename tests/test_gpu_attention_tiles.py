"""GPU: the tensor-memory attention kernel where its tiles of 32 rows, rounds of 256 tokens and items per CTA end."""
import numpy as np
import pytest

from test_gpu_attention import run_attention

pytestmark = pytest.mark.gpu


# The bound is that of test_rows_that_share_a_tile: fp16 hi + lo operands, sums of up to 2,000 fp32 terms.
@pytest.mark.parametrize("contexts,counts,block_tokens,max_splits", [
  ([31, 1700], [31, 31], 16, 32), ([65, 1700], [65, 31], 16, 32), ([96, 64, 1700], [96, 32, 2], 128, 32),  # one row fewer, more, whole tiles
  ([256, 1700], [40, 40], 16, 1), ([257, 1700], [40, 40], 16, 1), ([513, 1030], [64, 64], 128, 1),  # one piece: one round exactly, two, three and more
  ([320, 640], [33, 95], 16, 2), ([1900], [128], 128, 5),  # pieces of more than a round, the last of them short
  ([2600, 300] * 18, [20, 1] * 18, 16, 32), ([1300, 640, 90], [1100, 1, 33], 16, 32),  # more than 32 queries; more than 32 tiles, decode rows between
  ([700] * 12, [40] * 12, 16, 32), ([1200] * 8, [24] * 8, 128, 32),  # more items than CTAs: rings and phases go on from item to item
  ([256], [96], 16, 32), ([256], [95], 16, 32),  # the line to the tiles of 16 rows, and those:
  ([31], [31], 16, 32), ([65], [65], 16, 32), ([500, 300] * 18, [20, 1] * 18, 16, 32), ([270, 100], [60, 34], 16, 1),
])
def test_tiles_rounds_and_items(dev, contexts, counts, block_tokens, max_splits):
  rng = np.random.default_rng(sum(contexts) + 7 * len(counts) + max_splits)
  assert run_attention(dev, rng, contexts, counts, block_tokens, max_splits) < 1e-5
