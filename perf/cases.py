"""The work a user of this framework has it do, as cases that can be timed and compared.

Two faces of the framework are covered. `engine` cases go through `mtlqwen_b200.inference` (append a prompt, read tokens
until the stop token), which is what a serving program calls. The other cases go through `mtlqwen_b200.device`, one call
per kernel, which is what a program with a forward pass of its own calls: block-quantised projections (`linear`,
`layer`), the output head with sampling (`head`), paged attention (`attention`) and the gated delta rule (`gdn`).

All sizes are those of the decoder the benchmark runs (hidden 4096, intermediate 12288, vocabulary 248320, 32 layers =
8 x (3 gated delta rule + 1 attention), 8 live sequences, passes of up to 128 rows) or ragged ones around them.
"""
import os
import tempfile
from pathlib import Path

import numpy as np
import torch

from mtlqwen_b200 import device as D
from mtlqwen_b200.inference import InferenceEngine
from mtlqwen_b200.testing import synth

HIDDEN, INTERMEDIATE, VOCAB, LAYERS = 4096, 12288, 248320, 32
DRAFT_WIDTH = 4
TYPES = {"q4_k": D.Q4_K, "q5_k": D.Q5_K, "q6_k": D.Q6_K, "q8_0": D.Q8_0, "iq4_xs": D.IQ4_XS}
BLOCK_VALUES = {D.Q4_K: 256, D.Q5_K: 256, D.Q6_K: 256, D.Q8_0: 32, D.IQ4_XS: 256}
# The projections of one gated-delta-rule layer and the block types they come in: all Q4_K as in the benchmark's model,
# or the mix of types that the published files of such models hold. `gate` and `up` are one fused call.
PROJECTIONS = {"qkv": (8192, HIDDEN), "z": (HIDDEN, HIDDEN), "out": (HIDDEN, HIDDEN), "gate": (INTERMEDIATE, HIDDEN),
               "up": (INTERMEDIATE, HIDDEN), "down": (HIDDEN, INTERMEDIATE)}
MIXES = {"q4_k": {name: D.Q4_K for name in PROJECTIONS},
         "mixed": {"qkv": D.Q5_K, "z": D.Q5_K, "out": D.Q8_0, "gate": D.IQ4_XS, "up": D.IQ4_XS, "down": D.Q6_K}}


def listed():
  return [
    # One small projection of one token: the key projection of an attention layer in a single-user decode step.
    {"name": "linear_1024x4096_m1", "kind": "linear", "type": "q4_k", "n": 1024, "k": 4096, "m": 1},
    # All projections of a layer in a decode step of eight sequences, and of a full prompt pass.
    {"name": "layer_q4k_m8", "kind": "layer", "mix": "q4_k", "m": 8},
    {"name": "layer_q4k_m128", "kind": "layer", "mix": "q4_k", "m": 128},
    # The same decode step on a file that mixes block types, with an odd number of live sequences.
    {"name": "layer_mixed_m7", "kind": "layer", "mix": "mixed", "m": 7},
    # The end of a decode step: final norm, output head, top-k / top-p sampling for eight sequences.
    {"name": "head_m8", "kind": "head", "m": 8, "temperature": 0.7, "top_p": 0.9, "top_k": 40},
    # Attention of a decode step over long contexts (uniform in 1 .. 32768) in 16-token blocks.
    {"name": "attention_decode_8x32k", "kind": "attention", "contexts": "30963,20484,22420,29400,18950,25418,27318,7380", "rows": "1,1,1,1,1,1,1,1",
     "block": 16},
    # Attention of a prompt pass: 128 new tokens of one sequence behind 1920 earlier ones, in the engine's 128-token blocks.
    {"name": "attention_prompt_128", "kind": "attention", "contexts": "2048", "rows": "128", "block": 128},
    # The gated delta rule over prompt chunks uniform in 1 .. 512.
    {"name": "gdn_prompt_8x512", "kind": "gdn", "rows": "216,446,493,147,59,309,342,399", "decode": False},
    # One user: latency of a short answer to a short prompt.
    {"name": "engine_decode_1", "kind": "engine", "prompts": "24", "generated": 64, "temperature": 0.0, "top_k": 0, "speculative": False},
    # Eight users, ragged short prompts, greedy answers: decode throughput.
    {"name": "engine_decode_8", "kind": "engine", "prompts": "5,12,17,33,48,64,80,117", "generated": 64, "temperature": 0.0, "top_k": 0,
     "speculative": False},
    # Eight users with longer prompts and the first few sampled tokens of each: prompt processing mixed with decoding.
    {"name": "engine_prompt_8", "kind": "engine", "prompts": "512,431,377,256,201,129,77,18", "generated": 8, "temperature": 0.7, "top_k": 40,
     "speculative": False},
    # Eight users with speculative decoding, four drafted tokens a step.
    {"name": "engine_draft_8", "kind": "engine", "prompts": "5,12,17,33,48,64,80,117", "generated": 64, "temperature": 0.0, "top_k": 0, "speculative": True},
  ]


def _log_uniform(rng, low, high):
  return max(low, min(high, round(low * (high / low)**rng.random())))


def _join(values):
  return ",".join(str(v) for v in values)


def _numbers(text):
  return [int(v) for v in text.split(",")]


def draw(rng):
  kind = rng.choice(["linear", "layer", "layer", "head", "attention", "attention", "gdn", "engine", "engine"])
  if kind == "linear":
    name = rng.choice(sorted(TYPES))
    k = 2048 * rng.choice((1, 2, 4, 6)) if name == "q6_k" else 256 * rng.randint(1, 48)
    return {"kind": kind, "type": name, "n": 16 * _log_uniform(rng, 1, 512), "k": k, "m": rng.randint(1, 8)}
  if kind == "layer":
    mix = rng.choice(sorted(MIXES))
    return {"kind": kind, "mix": mix, "m": _log_uniform(rng, 1, 512 if mix == "q4_k" else 128)}
  if kind == "head":
    greedy = rng.random() < 0.5
    # up to eight rows in a plain step, five for each of several sequences in a speculative one
    m = rng.randint(1, 8) if rng.random() < 0.6 else (DRAFT_WIDTH + 1) * rng.randint(2, 8)
    return {"kind": kind, "m": m, "temperature": 0.0 if greedy else round(rng.uniform(0.3, 1.5), 2), "top_p": round(rng.uniform(0.5, 1.0), 2),
            "top_k": rng.randint(1, 64)}
  if kind == "attention":
    block = rng.choice((16, 128))
    if rng.random() < 0.5:
      count = rng.randint(1, 8)
      return {"kind": kind, "contexts": _join(_log_uniform(rng, 1, 24000) for _ in range(count)), "rows": _join([1] * count), "block": block}
    rows = [_log_uniform(rng, 1, 128) for _ in range(rng.randint(1, 4))]
    rows = [max(1, r * 128 // max(128, sum(rows))) for r in rows]
    return {"kind": kind, "contexts": _join(r + _log_uniform(rng, 1, 2000) - 1 for r in rows), "rows": _join(rows), "block": block}
  if kind == "gdn":
    decode = rng.random() < 0.5
    return {"kind": kind, "rows": _join([1] * rng.randint(1, 8) if decode else [_log_uniform(rng, 2, 400) for _ in range(rng.randint(1, 8))]),
            "decode": decode}
  long = rng.random() < 0.5
  count = rng.randint(1, 8)
  sampled = rng.random() < 0.5
  return {"kind": "engine", "prompts": _join(_log_uniform(rng, 1, 400 if long else 96) for _ in range(count)),
          "generated": rng.randint(2, 8) if long else _log_uniform(rng, 8, 64), "temperature": 0.7 if sampled else 0.0,
          "top_k": rng.choice((0, 20, 40)) if sampled else 0, "speculative": rng.random() < 0.35}


# ---- what a program holds before the call ---------------------------------------------------------------------------
class Held:
  """A torch tensor where the device calls expect a buffer."""

  def __init__(self, tensor):
    self.tensor, self.ptr = tensor, tensor.data_ptr()


_shared = {}


def _device():
  if "device" not in _shared:
    _shared["device"] = D.Device(0)
    _shared["rope"] = _shared["device"].rope_table(33000)
  return _shared["device"]


def _blocks(gen, qtype, n, k, std=0.02):
  """Random blocks of a weight matrix: uniform quants and sub-scales, block scales for weights of about N(0, std)."""
  count, size = n * (k // BLOCK_VALUES[qtype]), D.BLOCK_BYTES[qtype]
  raw = torch.randint(0, 256, (count, size), dtype=torch.uint8, device="cuda", generator=gen)
  unit = {D.Q4_K: 258.3, D.Q5_K: 527.0, D.Q6_K: 18.47 * 73.9, D.Q8_0: 73.9, D.IQ4_XS: 1330.0}[qtype]
  d = ((std / unit) * (0.8 + 0.4 * torch.rand(count, device="cuda", generator=gen))).half()
  at = 208 if qtype == D.Q6_K else 0
  raw[:, at:at + 2] = d.view(torch.uint8).view(count, 2)
  if qtype in (D.Q4_K, D.Q5_K):  # the minimum that centres the weights
    raw[:, 2:4] = (d.float() * (7.5 if qtype == D.Q4_K else 15.5)).half().view(torch.uint8).view(count, 2)
  return Held(raw)


def _normal(gen, *shape, scale=1.0, shift=0.0):
  return Held(torch.randn(shape, device="cuda", generator=gen) * scale + shift)


def _empty(*shape, dtype=torch.float32):
  return Held(torch.zeros(shape, device="cuda", dtype=dtype))


def _prepare_linear(case, gen):
  qtype, n, k, m = TYPES[case["type"]], case["n"], case["k"], case["m"]
  return {"type": qtype, "n": n, "k": k, "m": m, "w": _blocks(gen, qtype, n, k), "x": _normal(gen, m, k), "y": _empty(m, n)}


def _run_linear(dev, s):
  dev.linear(s["type"], s["w"], s["n"], s["k"], s["x"], s["m"], s["y"])
  return s["y"].tensor


def _prepare_layer(case, gen):
  mix, m = MIXES[case["mix"]], case["m"]
  state = {"m": m, "mix": mix, "w": {name: _blocks(gen, mix[name], *shape) for name, shape in PROJECTIONS.items()}}
  state.update({name: _normal(gen, m, HIDDEN) for name in ("x", "mixer", "x2", "hidden")})
  state.update({name: _empty(m, width) for name, width in (("qkv", 8192), ("z", HIDDEN), ("after", HIDDEN), ("mlp", INTERMEDIATE), ("next", HIDDEN))})
  return state


def _run_layer(dev, s):
  w, mix, m = s["w"], s["mix"], s["m"]
  dev.linear_group(mix["qkv"], [w["qkv"], w["z"]], [8192, HIDDEN], HIDDEN, s["x"], m, [s["qkv"], s["z"]])
  dev.linear(mix["out"], w["out"], HIDDEN, HIDDEN, s["mixer"], m, s["after"], s["hidden"])
  dev.gate_up(mix["gate"], w["gate"], w["up"], INTERMEDIATE, HIDDEN, s["x2"], m, s["mlp"])
  dev.linear(mix["down"], w["down"], HIDDEN, INTERMEDIATE, s["mlp"], m, s["next"], s["after"])
  return [s[name].tensor for name in ("qkv", "z", "after", "mlp", "next")]


def _prepare_head(case, gen):
  m, queries = case["m"], []
  for i in range(m):
    q = D.Query()
    q.start, q.count, q.position, q.slot, q.state, q.logit, q.samples = i, 1, 100 + i, i % 8, D.UNBOUND, i, 1
    q.temperature, q.topP, q.topK, q.seed = case["temperature"], case["top_p"], case["top_k"], 1000 + i
    queries.append(q)
  return {"m": m, "queries": _device().queries(queries), "w": _blocks(gen, D.Q6_K, VOCAB, HIDDEN), "norm": _normal(gen, HIDDEN, scale=0.01, shift=1.0),
          "hidden": _normal(gen, m, HIDDEN), "x": _empty(m, HIDDEN), "logits": _empty(m, VOCAB), "tokens": _empty(m, dtype=torch.int32)}


def _run_head(dev, s):
  m = s["m"]
  dev.rms_norm(s["hidden"], s["norm"], m, HIDDEN, s["x"])
  dev.linear(D.Q6_K, s["w"], VOCAB, HIDDEN, s["x"], m, s["logits"])
  dev.sample(s["logits"], VOCAB, s["queries"], m, m, 0, s["tokens"])
  return s["logits"].tensor, s["tokens"].tensor


def _prepare_attention(case, gen):
  contexts, rows, block = _numbers(case["contexts"]), _numbers(case["rows"]), case["block"]
  blocks = [-(-c // block) for c in contexts]
  physical, total = sum(blocks), sum(rows)
  order = torch.randperm(physical, device="cuda", generator=gen).int()
  table = torch.zeros((len(contexts), max(blocks)), device="cuda", dtype=torch.int32)
  queries, start, at = [], 0, 0
  for i, (context, count) in enumerate(zip(contexts, rows)):
    table[i, :blocks[i]] = order[at:at + blocks[i]]
    at += blocks[i]
    q = D.Query()
    q.start, q.count, q.position, q.slot, q.state = start, count, context - count, i, D.UNBOUND
    queries.append(q)
    start += count
  dev = _device()
  cache = [Held(torch.randn((physical, 4, block, 256), device="cuda", generator=gen, dtype=torch.float16)) for _ in range(2)]
  return {"rows": total, "count": len(contexts), "queries": dev.queries(queries), "table": Held(table), "stride": max(blocks), "block": block,
          "cache": cache, "qg": _normal(gen, total, 16, 512), "k": _normal(gen, total, 4, 256), "v": _normal(gen, total, 4, 256),
          "q_norm": _normal(gen, 256, scale=0.01, shift=1.0), "k_norm": _normal(gen, 256, scale=0.01, shift=1.0), "q": _empty(total, 16, 256),
          "partials": _empty(dev.attention_scratch_bytes(total, 32) // 4), "out": _empty(total, 16, 256)}


def _run_attention(dev, s):
  dev.attention_prepare(s["qg"], s["k"], s["v"], s["q_norm"], s["k_norm"], _shared["rope"], s["queries"], s["count"], s["rows"], s["table"], s["stride"],
                        s["block"], s["q"], *s["cache"])
  dev.attention(s["q"], s["qg"], *s["cache"], s["queries"], s["count"], s["rows"], s["table"], s["stride"], s["block"], 32, s["partials"], s["out"])
  return s["out"].tensor, s["q"].tensor, s["cache"][0].tensor, s["cache"][1].tensor


def _prepare_gdn(case, gen):
  lengths = _numbers(case["rows"])
  rows, count, record = sum(lengths), len(lengths), D.GDN_LAYER_STATE_BYTES
  previous = torch.cat([torch.randn((count, 8192 * 4), device="cuda", generator=gen), 0.01 * torch.randn((count, 32 * 128 * 128), device="cuda", generator=gen)],
                       dim=1)
  state = {"rows": rows, "count": count, "decode": case["decode"], "previous": Held(previous), "next": _empty(count, record // 4)}
  queries, start = [], 0
  for i, length in enumerate(lengths):
    q = D.Query()
    q.previous, q.next = state["previous"].ptr + i * record, state["next"].ptr + i * record
    q.start, q.count, q.position, q.slot, q.state = start, length, 77, i, D.UNBOUND
    queries.append(q)
    start += length
  state["queries"] = _device().queries(queries)
  state.update(beta_w=_normal(gen, 32, HIDDEN, scale=1 / 64), alpha_w=_normal(gen, 32, HIDDEN, scale=1 / 64), dt=_normal(gen, 32, scale=0.1),
               a=Held(-1 - 15 * torch.rand(32, device="cuda", generator=gen)), conv=_normal(gen, 8192, 4, scale=0.5),
               norm=_normal(gen, 128, scale=0.01, shift=1.0), x=_normal(gen, rows, HIDDEN), mixed=_normal(gen, rows, 8192), z=_normal(gen, rows, HIDDEN),
               out=_empty(rows, 32, 128))
  if not case["decode"]:
    state.update(q=_empty(rows, 16, 128), k=_empty(rows, 16, 128), v=_empty(rows, 32, 128), beta=_empty(rows, 32), g=_empty(rows, 32))
  return state


def _run_gdn(dev, s):
  record = D.GDN_LAYER_STATE_BYTES
  if s["decode"]:
    dev.gdn_decode(s["x"], s["mixed"], s["beta_w"], s["alpha_w"], s["a"], s["dt"], s["conv"], s["z"], s["norm"], s["queries"], s["count"], 0,
                   D.CONV_STATE_BYTES, record, s["out"])
  else:
    dev.gdn_prepare(s["x"], s["mixed"], s["beta_w"], s["alpha_w"], s["a"], s["dt"], s["conv"], s["queries"], s["count"], s["rows"], 0, record, s["q"], s["k"],
                    s["v"], s["beta"], s["g"])
    dev.delta_rule(s["q"], s["k"], s["v"], s["g"], s["beta"], s["z"], s["norm"], s["queries"], s["count"], D.CONV_STATE_BYTES, record, s["out"], prefill=True)
  return s["out"].tensor, s["next"].tensor


# ---- the engine -----------------------------------------------------------------------------------------------------
def _model_path():
  """A random-init file of the full decoder with its MTP block, written once per machine (5.7 GB). Random logits have
  many near ties; a trained model's mostly have not, so here token t + 1 follows token t by a wide margin: row t + 1 of
  the output head is row t of the (large) embedding, and the MTP projection passes the embedding on. Which token comes
  next does then not hang on the last bits of a sum; the recurrent states, which do, are compared as numbers."""
  path = Path(tempfile.gettempdir()) / f"mtlqwen_b200_cases_{LAYERS}x{VOCAB}_v1.gguf"
  if path.exists():
    return path
  tensors = [(name, qtype, shape, make) for name, qtype, shape, make in synth.model_tensors(LAYERS, VOCAB, True)]
  rng = np.random.default_rng(2024)
  pool = {D.Q4_K: synth.q4k_blocks(1 << 20, rng)}  # tensors are windows of one pool: 150 MB drawn instead of 5 GB
  table = synth.q6k_blocks(VOCAB * HIDDEN // 256, rng, target_std=8.0)
  head = np.roll(table.reshape(VOCAB, -1), 1, axis=0).reshape(table.shape)
  scale = head[:, 208:210].copy().view(np.float16).astype(np.float32) * (0.02 / 8.0)
  head[:, 208:210] = scale.astype(np.float16).view(np.uint8).reshape(-1, 2)
  through = np.zeros((HIDDEN, 2 * HIDDEN // 256, 144), np.uint8)  # 4 on the diagonal of the embedding half
  row = np.arange(HIDDEN)
  block, element = row // 256, row % 256
  through[row, block, 0:2] = np.frombuffer(np.float16(4.0 / 945).tobytes(), np.uint8)
  through[row, block, 4:16] = 0xff  # sub-block scales 63 (and minima, times a zero dmin)
  through[row, block, 16 + element // 64 * 32 + element % 32] = np.where(element % 64 < 32, 0x0f, 0xf0)

  def content(i, name, qtype, shape, make):
    if name == "token_embd.weight":
      return table
    if name == "output.weight":
      return head
    if name.endswith("eh_proj.weight"):
      return through
    if qtype == D.Q4_K:
      count = shape[0] * shape[1] // 256
      at = (i * 104729) % ((1 << 20) - count)
      return pool[qtype][at:at + count]
    return make()

  def text(value):
    return np.uint64(len(value)).tobytes() + value.encode()

  header = np.uint32(synth.GGUF_MAGIC).tobytes() + np.uint32(3).tobytes() + np.uint64(len(tensors)).tobytes() + np.uint64(1).tobytes()
  header += text("general.architecture") + np.uint32(8).tobytes() + text("qwen35")
  align, offset, offsets = synth.GGUF_ALIGNMENT, 0, []
  for name, qtype, shape, _ in tensors:
    header += text(name) + np.uint32(len(shape)).tobytes() + b"".join(np.uint64(d).tobytes() for d in reversed(shape))
    header += np.uint32(qtype).tobytes() + np.uint64(offset).tobytes()
    offsets.append(offset)
    offset += -(-synth.tensor_bytes(qtype, int(np.prod(shape))) // align) * align
  data = -(-len(header) // align) * align
  temporary = path.with_suffix(f".{os.getpid()}.tmp")
  with open(temporary, "wb") as out:
    out.write(header)
    for i, (tensor, at) in enumerate(zip(tensors, offsets)):
      out.seek(data + at)
      out.write(np.ascontiguousarray(content(i, *tensor)).data)
    out.truncate(data + offset)
  os.replace(temporary, path)
  return path


def _engine(speculative):
  """One engine per process and kind, as a server keeps it: the plain model, or the model with its MTP drafter."""
  key = "drafting" if speculative else "plain"
  if key not in _shared:
    settings = {"INFENG_KV_BLOCKS": "384", "INFENG_SEED": "1", "INFENG_DRAFT_WIDTH": str(DRAFT_WIDTH)}
    before = {name: os.environ.get(name) for name in settings}
    os.environ.update(settings)
    try:
      path = _model_path()
      _shared[key] = InferenceEngine(path, draft_weights=path if speculative else None, max_context=4096)
    finally:
      for name, value in before.items():
        os.environ.pop(name) if value is None else os.environ.__setitem__(name, value)
  return _shared[key]


def _prepare_engine(case, seed):
  rng = np.random.default_rng(seed)
  requests = []
  for i, length in enumerate(_numbers(case["prompts"])):
    prompt = [int(t) for t in rng.integers(0, VOCAB - 1024, length)]
    requests.append((prompt, [prompt[-1] + case["generated"]], int(rng.integers(1 << 40))))  # prompt, stop tokens, sampling key
  return {"engine": _engine(case["speculative"]), "requests": requests, "temperature": case["temperature"], "top_k": case["top_k"],
          "speculative": case["speculative"]}


# The recurrent state of the last gated-delta-rule layer: every layer below and every token of the sequence goes into it.
LAST_STATE = 23 * D.GDN_LAYER_STATE_BYTES + D.CONV_STATE_BYTES


def _run_engine(s):
  engine, tokens, states = s["engine"], [], []
  sequences = [engine.sequence(stop_token_ids=stops, temperature=s["temperature"], top_p=0.9, top_k=s["top_k"], speculative=s["speculative"], seed=key)
               for _, stops, key in s["requests"]]
  cursors = [sequence.append(prompt) for sequence, (prompt, _, _) in zip(sequences, s["requests"])]
  for sequence, cursor in zip(sequences, cursors):
    answer = []
    while (token := sequence.read(cursor)) is not None:
      answer.append(token)
      cursor += 1
    tokens.append(np.array(answer, np.int32))
  for sequence in sequences:
    states.append(sequence.state(LAST_STATE, D.RECURRENT_STATE_BYTES // 4))
    sequence.close()
  return {"tokens": tokens, "states": states}


PREPARE = {"linear": _prepare_linear, "layer": _prepare_layer, "head": _prepare_head, "attention": _prepare_attention, "gdn": _prepare_gdn}
RUN = {"linear": _run_linear, "layer": _run_layer, "head": _run_head, "attention": _run_attention, "gdn": _run_gdn}


def prepare(case, seed):
  if case["kind"] == "engine":
    return {"kind": "engine", **_prepare_engine(case, seed)}
  _device()
  return {"kind": case["kind"], **PREPARE[case["kind"]](case, torch.Generator("cuda").manual_seed(seed))}


def run(state):
  if state["kind"] == "engine":
    return _run_engine(state)
  return RUN[state["kind"]](_device(), state)


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def _matrix_bytes(qtype, n, k):
  return n * (k // BLOCK_VALUES[qtype]) * D.BLOCK_BYTES[qtype]


GDN_LAYER = sum(n * k for n, k in PROJECTIONS.values())
ATTENTION_LAYER = (8192 + 2 * 1024 + 4096) * HIDDEN + 3 * INTERMEDIATE * HIDDEN
BODY = 24 * GDN_LAYER + 8 * ATTENTION_LAYER  # weights of the decoder layers
HEAD_BYTES = _matrix_bytes(D.Q6_K, VOCAB, HIDDEN)
STATE_BYTES = 24 * D.GDN_LAYER_STATE_BYTES


def _engine_work(case):
  prompts, generated = _numbers(case["prompts"]), case["generated"]
  # One reading of the weights for all prompts, then one per decode step (per accepted run of drafts when speculating);
  # the states are read and written once a step.
  steps = -(-(generated - 1) // (DRAFT_WIDTH + 1)) if case["speculative"] else generated - 1
  sequences, rows = len(prompts), sum(prompts) + len(prompts) * (generated - 1)
  weights = BODY // 256 * 144 + HEAD_BYTES
  drafting = (ATTENTION_LAYER + 2 * HIDDEN * HIDDEN) // 256 * 144 + HEAD_BYTES if case["speculative"] else 0
  keys = sum(8 * 4096 * (p + generated // 2) for p in prompts)
  flops = 2 * BODY * rows + 2 * VOCAB * HIDDEN * sequences * generated
  return {"bytes": (steps + 1) * (weights + 2 * sequences * STATE_BYTES) + steps * (keys + DRAFT_WIDTH * drafting), "flops": flops}


def work(case):
  kind = case["kind"]
  if kind == "engine":
    return _engine_work(case)
  if kind == "linear":
    n, k, m = case["n"], case["k"], case["m"]
    return {"bytes": _matrix_bytes(TYPES[case["type"]], n, k) + 4 * m * (n + k), "flops": 2 * m * n * k}
  if kind == "layer":
    mix, m = MIXES[case["mix"]], case["m"]
    weights = sum(_matrix_bytes(mix[name], *shape) for name, shape in PROJECTIONS.items())
    return {"bytes": weights + 4 * m * (4 * HIDDEN + 8192 + 3 * HIDDEN + INTERMEDIATE), "flops": 2 * m * GDN_LAYER}
  if kind == "head":
    m = case["m"]
    return {"bytes": HEAD_BYTES + 4 * m * (HIDDEN + VOCAB), "flops": 2 * m * VOCAB * HIDDEN}
  if kind == "attention":
    contexts, rows = _numbers(case["contexts"]), _numbers(case["rows"])
    attended = sum(r * c - r * (r - 1) // 2 for c, r in zip(contexts, rows))
    return {"bytes": 4096 * sum(contexts) + 4 * sum(rows) * (16 * 512 + 2 * 4 * 256 + 2 * 16 * 256), "flops": 4 * 16 * 256 * attended}
  rows = _numbers(case["rows"])
  per_row = 4 * (HIDDEN + 8192 + HIDDEN + HIDDEN)
  return {"bytes": 2 * len(rows) * D.GDN_LAYER_STATE_BYTES + sum(rows) * per_row + 2 * 32 * HIDDEN * 4, "flops": sum(rows) * (32 * 128 * 128 * 8 + 2 * 64 * HIDDEN)}


def tolerance(case):
  """About four times what switching the arithmetic was seen to change (relative 2-norm, largest element): against fp64
  the fp32-accurate kernels are off by 4e-7 and 2e-6, the 16-bit activation grid of the Q4_K decode kernel by 3e-5 and
  1e-4 (a chain of projections by 6e-5 and 4e-4), the fp16 operands of Q4_K with more than eight rows by 5e-4 and 2e-3
  (a chain by 7e-4 and 8e-3); another split of attention changes 3e-6 and 1e-5 (and a rounding of a stored fp16 key 1e-3 of
  it), the delta rule token by token instead of in chunks 2e-7 and 2e-5, the engine with other kernels throughout the last
  recurrent state by 2e-3 and 7e-2. Tokens do not depend on such differences."""
  kind = case["kind"]
  if kind == "engine":
    return {"rel": 1e-2, "max": 0.3, "differ": 0.0}
  if kind == "attention":
    return {"rel": 1.5e-5, "max": 4e-3}
  if kind == "gdn":
    return {"rel": 1e-5, "max": 1e-4}
  if kind in ("linear", "layer") and case.get("type", case.get("mix")) == "q4_k":
    return {"rel": 2.5e-3, "max": 3e-2} if case["m"] > 8 else {"rel": 2.5e-4, "max": 2e-3}
  return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
