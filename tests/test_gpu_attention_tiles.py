"""GPU: the attention kernels for the rows of a prompt where their tiles, rounds of 256 tokens, items per CTA and the line between them end."""
import numpy as np
import pytest

from mtlqwen_b200 import device as D
from test_gpu_attention import run_attention

pytestmark = pytest.mark.gpu


# The bound is that of test_rows_that_share_a_tile: fp16 hi + lo operands, sums of up to 2,000 fp32 terms.
@pytest.mark.parametrize("contexts,counts,block_tokens,max_splits", [
  ([31, 1700], [31, 31], 16, 32), ([65, 1700], [65, 31], 16, 32), ([96, 64, 1700], [96, 32, 2], 128, 32),  # one row fewer, more, whole tiles
  ([256, 1700], [40, 40], 16, 1), ([257, 1700], [40, 40], 16, 1), ([513, 1030], [64, 64], 128, 1),  # one piece: one round exactly, two, three and more
  ([900, 1300], [33, 95], 16, 2), ([1900], [128], 128, 5),  # pieces of more than a round, the last of them short
  ([2600, 300] * 18, [20, 1] * 18, 16, 32), ([1300, 640, 90], [1100, 1, 33], 16, 32),  # more than 32 queries; more than 32 tiles, decode rows between
  ([700] * 12, [40] * 12, 16, 32), ([1200] * 8, [24] * 8, 128, 32),  # more items than CTAs: rings and phases go on from item to item
  # passes of less work, in tiles of 16 rows
  ([320, 640], [33, 95], 16, 2), ([256], [96], 16, 32), ([256], [95], 16, 32), ([31], [31], 16, 32), ([65], [65], 16, 32), ([500, 300] * 18, [20, 1] * 18, 16, 32), ([270, 100], [60, 34], 16, 1),
])
def test_tiles_rounds_and_items(dev, contexts, counts, block_tokens, max_splits):
  rng = np.random.default_rng(sum(contexts) + 7 * len(counts) + max_splits)
  assert run_attention(dev, rng, contexts, counts, block_tokens, max_splits) < 1e-5


class Pass:
  """Queries of `counts` rows at the end of `contexts` tokens, with a table of `stride` blocks a slot."""

  def __init__(self, dev, seed, contexts, counts, block_tokens=16, stride=None):
    rng = np.random.default_rng(seed)
    blocks = [-(-c // block_tokens) for c in contexts]
    self.dev, self.contexts, self.counts, self.block_tokens, self.stride = dev, contexts, counts, block_tokens, stride or max(blocks)
    order = rng.permutation(sum(blocks)).astype(np.int32)
    self.table, at = np.zeros((len(contexts), self.stride), np.int32), 0
    for i, n in enumerate(blocks):
      self.table[i, :n] = order[at:at + n]
      at += n
    self.rows = sum(counts)
    self.keys, self.values = (rng.standard_normal((sum(blocks), 4, block_tokens, 256)).astype(np.float16) for _ in range(2))
    self.q, self.qg = (rng.standard_normal((self.rows, 16, width)).astype(np.float32) for width in (256, 512))
    self.starts = np.concatenate([[0], np.cumsum(counts)])[:-1]
    queries = []
    for i, (context, count) in enumerate(zip(contexts, counts)):
      info = D.Query()
      info.start, info.count, info.position, info.slot, info.state = int(self.starts[i]), count, context - count, i, D.UNBOUND
      queries.append(info)
    self.held = [dev.array(self.q), dev.array(self.qg), dev.array(self.keys.view(np.uint16)), dev.queries(queries), dev.array(self.table)]

  def run(self, values=None, context=0, max_splits=32, offset=0):
    """offset: floats by which the partial results miss a 16-byte boundary."""
    dev, (q, qg, keys, queries, table) = self.dev, self.held
    out, partials = dev.empty((self.rows, 16, 256)), dev.empty(dev.attention_scratch_bytes(self.rows, max_splits) // 4 + 4)
    if context:
      dev.attention_context(context)
    dev.attention(q, qg, keys, dev.array((self.values if values is None else values).view(np.uint16)), queries, len(self.counts), self.rows, table, self.stride,
                  self.block_tokens, max_splits, type("View", (), {"ptr": partials.ptr + 4 * offset}), out)
    dev.commit()
    return out.download()


@pytest.mark.parametrize("contexts,counts", [([64], [64]), ([33, 64, 80], [33, 64, 30]), ([700] * 8, [6] * 8), ([700, 40], [20, 40])])
def test_the_longest_context_counts_and_not_the_width_of_the_table(dev, contexts, counts):
  narrow = Pass(dev, 81, contexts, counts).run()
  wide = Pass(dev, 81, contexts, counts, stride=512)
  assert wide.run(context=max(contexts)).tobytes() == narrow.tobytes()
  other = wide.run()  # the bound is gone after one call: tiles of 32 rows
  assert other.tobytes() != narrow.tobytes() and np.abs(other - narrow).max() < 1e-5 * np.abs(narrow).max()


# The work of a pass (rows x the tokens a table row holds) below the line between the two kinds of tiles and on it: whole passes, passes of few rows, several
# queries of 17 to 31 rows; queries of 33 to 63 rows, which are reckoned as two tiles each, and one beside a decode row.
@pytest.mark.parametrize("contexts,counts,block_tokens", [
  ([752], [128], 16), ([768], [128], 16), ([14560], [9], 16), ([14576], [9], 16), ([1520, 900], [24, 24], 16), ([1536, 900], [24, 24], 16),
  ([320, 640, 1700], [33, 95, 40], 16), ([1000] * 4, [48] * 4, 16), ([1400, 1500, 1700], [40, 33, 62], 16), ([2000, 1500], [63, 1], 128)])
def test_either_side_of_the_line_between_the_tiles(dev, contexts, counts, block_tokens):
  rng = np.random.default_rng(sum(contexts) + len(counts))
  assert run_attention(dev, rng, contexts, counts, block_tokens) < 1e-5


@pytest.mark.parametrize("operand,offset", [("q", 1), ("partials", 1), ("partials", 3), ("keys", 2), ("values", 4)])
def test_operands_that_the_copies_cannot_take_are_refused(dev, operand, offset):
  """Floats by which q and the partial results miss a multiple of 8 bytes, halves by which the cache misses one of 16."""
  work = Pass(dev, 93, [40], [1])
  q, qg, keys, queries, table = work.held
  values, out = dev.array(work.values.view(np.uint16)), dev.empty((1, 16, 256))
  partials = dev.empty(dev.attention_scratch_bytes(1, 32) // 4 + 4)
  operands = {"q": q.ptr, "keys": keys.ptr, "values": values.ptr, "partials": partials.ptr}
  operands[operand] += offset * (2 if operand in ("keys", "values") else 4)
  view = {name: type("View", (), {"ptr": ptr}) for name, ptr in operands.items()}
  before = dev.lib.infdev_launch_count(dev.ctx)
  with pytest.raises(RuntimeError, match="boundaries"):
    dev.attention(view["q"], qg, view["keys"], view["values"], queries, 1, 1, table, work.stride, work.block_tokens, 32, view["partials"], out)
  if operand != "partials":
    with pytest.raises(RuntimeError, match="boundaries"):
      dev.check(dev.lib.infdev_attention_static(dev.ctx, operands["q"], qg.ptr, operands["keys"], operands["values"], queries.ptr, 1, 1, table.ptr, work.stride,
                                                work.block_tokens, out.ptr))
  assert dev.lib.infdev_launch_count(dev.ctx) == before


def broken_rows(work, clean, got, query, token, dims):
  """The rows of `query` from `token` on, in the heads of kv head 1, and nothing else, are not finite."""
  first = int(work.starts[query]) + max(0, token - (work.contexts[query] - work.counts[query]))
  hit = np.zeros_like(clean, bool)
  for dim in dims:
    hit[first:int(work.starts[query]) + work.counts[query], 4:8, dim] = True
  assert not np.isfinite(got[hit]).any()
  assert got[~hit].tobytes() == clean[~hit].tobytes()


def break_value(work, values, query, token, dims, value):
  values[work.table[query, token // work.block_tokens], 1, token % work.block_tokens, dims] = value


# Contexts that the table is cut to, so that the first ones are served in tiles of 16 rows; the others in tiles of 32: several rounds of 256 tokens in one
# piece, with the value in the first, at the ends and in the last; pieces of several rounds.
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("context,rows,token,max_splits", [
  (40, 40, 39, 32), (40, 40, 17, 32), (200, 64, 150, 32), (90, 48, 60, 32), (90, 48, 3, 32),
  (1200, 1100, 100, 1), (1200, 1100, 355, 1), (1200, 1100, 356, 1), (1200, 1100, 1199, 1), (1300, 64, 1260, 1), (1300, 64, 700, 1), (1300, 400, 1100, 2)])
def test_rows_before_a_value_that_is_not_finite_do_not_notice(dev, context, rows, token, max_splits, value):
  work, dims = Pass(dev, token, [context], [rows]), [7, 200]
  clean, values = work.run(max_splits=max_splits), work.values.copy()
  break_value(work, values, 0, token, dims, value)
  broken_rows(work, clean, work.run(values, max_splits=max_splits), 0, token, dims)


# 40 tiles of 32 rows in one piece each are 160 items: some CTAs take two, one after the other. The value is in an item of the first
# turn, of the second, or in a tile that several items later has nothing of it.
@pytest.mark.parametrize("query", [0, 17, 18, 19])
def test_a_broken_value_stays_with_its_item(dev, query):
  contexts, counts = [600 + 8 * i for i in range(20)], [64] * 20
  work, dims = Pass(dev, 90, contexts, counts), [0, 255]
  clean, values, token = work.run(max_splits=1), work.values.copy(), contexts[query] - 20
  break_value(work, values, query, token, dims, np.nan)
  broken_rows(work, clean, work.run(values, max_splits=1), query, token, dims)


@pytest.mark.parametrize("contexts,counts", [([300], [128]), ([2000, 50], [100, 28])])
def test_partial_results_eight_bytes_off(dev, contexts, counts):
  work = Pass(dev, 91, contexts, counts)
  want = work.run()
  assert np.abs(work.run(offset=2) - want).max() < 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("which", ["qg", "k", "v", "q_norm", "rope", "q", "cache"])
def test_preparation_at_any_element(dev, which):
  """An operand that misses a 16-byte boundary is read or written element by element, to the same bits."""
  rows, block_tokens, rng = 37, 16, np.random.default_rng(92)
  qg, k, v, q_norm, k_norm = (rng.standard_normal(shape).astype(np.float32) for shape in ((rows, 16, 512), (rows, 4, 256), (rows, 4, 256), 256, 256))
  rope, blocks = dev.rope_table(rows + 5), -(-(rows + 5) // block_tokens)
  table = dev.array(rng.permutation(blocks).astype(np.int32))
  info = D.Query()
  info.start, info.count, info.position, info.slot, info.state = 0, rows, 5, 0, D.UNBOUND

  def run(moved):
    def place(array, name):
      array = np.ascontiguousarray(array)
      shift = int(name == moved)
      buffer = dev.array(np.concatenate([np.zeros(shift, array.dtype), array.reshape(-1), np.zeros(8, array.dtype)]))
      return buffer, type("View", (), {"ptr": buffer.ptr + shift * array.itemsize}), lambda: buffer.download()[shift:shift + array.size].tobytes()

    inputs = [place(a, name) for a, name in ((qg, "qg"), (k, "k"), (v, "v"), (q_norm, "q_norm"), (k_norm, "k_norm"), (rope.download(), "rope"))]
    outputs = [place(np.zeros((rows, 16, 256), np.float32), "q")] + [place(np.zeros((blocks, 4, block_tokens, 256), np.uint16), "cache") for _ in range(2)]
    dev.attention_prepare(*(view for _, view, _ in inputs), dev.queries([info]), 1, rows, table, blocks, block_tokens, *(view for _, view, _ in outputs))
    dev.commit()
    return [download() for _, _, download in outputs]

  assert run(which) == run(None)
