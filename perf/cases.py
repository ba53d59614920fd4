"""The work whose speed counts: steps and generations of whole models through the engine's public calls.

A case names a model, a storage type, a kind of call and its sizes:

* `prompt`   `Engine.step_raw` on whole prompts, the logits of each prompt's last token wanted: the
             first token of one request, or of several that arrive together;
* `decode`   `Engine.step_raw(..., from_graph=True)` on live requests that bring one token each, as
             trace replay with graphs and every step of generation does it; the requests grow by a
             token a pass, and start again when they reach the engine's longest sequence;
* `score`    `Engine.score_tokens`, the log-likelihood of a text;
* `generate` `Engine.generate`, greedy, continuous batching over the engine's slots.

Models: the Gemma 2 shapes of the presets and the layer shapes of the design benchmark (`2b-like` and
`8b-like`), with random weights.  Sapivik stands for routed experts and gated recurrences, Zesapel for
latent attention, the delta rule, the state-space mixer and several residual streams.

The weights have the spread of trained ones (rows that keep the size of what they multiply, peaked
routers, decays of a few to thousands of tokens), and the output rows lean towards one token per input
token, so that the likeliest token is as clear as in text.
"""

import functools
import math
import random
import zlib

import torch

from simply_b200 import Engine, EngineConfig, SamplingParams, StepEntry, design_bench
from simply_b200.config import config_from_dict, preset
from simply_b200.parts.model import tensor_specs

LONGEST = 8192
PORTION = 2048  # tokens of one step when contexts are written in `prepare`
WANTED_LOGPROB = -2.0  # of the likeliest token, about


# ---- cases -----------------------------------------------------------------------------------------

def listed():
  case = lambda name, model, kind, batch, low, high, new=0, slots=8, burst=1, dtype="bfloat16": dict(
      name=name, model=model, dtype=dtype, kind=kind, batch=batch, low=low, high=high, new=new, slots=slots, burst=burst)
  return [
      # A short question: the whole model for a handful of tokens, where launches and the host count.
      case("prompt 13 2B", "gemma2-2b", "prompt", 1, 13, 13),
      # The ordinary prompt of one request, the size the benchmark prints.
      case("prompt 2048 2B", "gemma2-2b", "prompt", 1, 2048, 2048),
      # Requests of all lengths that arrive together and share a step.
      case("prompts together 2B", "gemma2-2b", "prompt", 7, 3, 1500),
      # A document for the larger model: the largest step.
      case("prompt 3001 9B", "gemma2-9b", "prompt", 1, 3001, 3001),
      # One user's tokens, one after the other: latency.
      case("decode 1 2B", "gemma2-2b", "decode", 1, 700, 1100),
      # The benchmark's headline: eight requests near the longest context.
      case("decode 8 long 2B", "gemma2-2b", "decode", 8, 7040, 7168),
      # Serving: requests of all sizes come and go, prompts beside decoded tokens in one step.
      case("serve 64 2B", "gemma2-2b", "generate", 64, 24, 640, new=64, slots=40, burst=4),
      # The 32-bit path, which users take to check results: a text's likelihood.
      case("score 301 in float32", "gemma2 2b-like", "score", 1, 301, 301, dtype="float32"),
      # Routed experts and a gated recurrence: a prompt, and eight users.
      case("prompt 2048 experts", "sapivik 2b-like", "prompt", 1, 2048, 2048),
      case("decode 8 experts", "sapivik 2b-like", "decode", 8, 500, 1500),
      # Latent attention, delta rule, state space: two prompts of odd lengths, and eight users.
      case("prompts 2 latent", "zesapel 2b-like", "prompt", 2, 517, 1531),
      case("decode 8 latent", "zesapel 2b-like", "decode", 8, 500, 1500),
  ]


def draw(rng):
  spread = lambda low, high: int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
  model = rng.choice(["gemma2-2b"] * 4 + ["gemma2 8b-like", "sapivik 2b-like", "sapivik 8b-like", "zesapel 2b-like",
                                         "zesapel 8b-like", "gemma2 2b-like"])
  kind = rng.choice(["prompt", "prompt", "decode", "decode", "score", "generate"])
  dtype = "float32" if model == "gemma2 2b-like" else "bfloat16"
  c = dict(model=model, dtype=dtype, kind=kind, batch=1, low=1, high=1, new=0, slots=8, burst=1)
  if dtype == "float32":  # the checking path: small batches
    c["kind"] = kind = rng.choice(["prompt", "score"])
  if kind == "prompt":
    c["batch"] = rng.choice([1, 1, 1, 2, 3, 5, 8])
    c["high"] = spread(5, (600 if dtype == "float32" else 6000) // c["batch"])
    c["low"] = c["high"] if c["batch"] == 1 else max(1, c["high"] // 8)
  elif kind == "decode":
    c["batch"] = c["slots"] = spread(1, 48)
    c["high"] = spread(40, 24000 // max(c["batch"], 4))
    c["low"] = max(1, c["high"] // 2)
  elif kind == "score":
    c["low"] = c["high"] = spread(40, 400 if dtype == "float32" else 2000)
  else:
    c["slots"] = rng.choice([4, 8, 16, 32])
    c["batch"] = c["slots"] + rng.randrange(0, c["slots"])
    c["high"] = spread(30, 600)
    c["low"] = max(1, c["high"] // 8)
    c["new"] = spread(8, 48)
    c["burst"] = rng.choice([1, 4, 8])
  return c


def _lengths(case):
  """Lengths of the case's prompts: spread between its bounds, the same for every seed."""
  if case["low"] == case["high"]:
    return [case["low"]] * case["batch"]
  rng = random.Random(case["batch"] * 7919 + case["high"])
  got = [round(math.exp(rng.uniform(math.log(case["low"]), math.log(case["high"])))) for _ in range(case["batch"])]
  got[0], got[-1] = case["low"], case["high"]
  return got


def _new_tokens(case):
  rng = random.Random(case["batch"] + case["new"])
  return [rng.randint(max(1, case["new"] // 4), case["new"]) for _ in range(case["batch"])]


def _prompts(case, seed, vocab, more=0):
  rng = random.Random(seed * 1000003 + 11)
  return [[rng.randrange(16, vocab) for _ in range(n + more)] for n in _lengths(case)]


@functools.cache
def _config(model):
  """The model's config and the family whose rules it follows."""
  if " " not in model:
    return preset(model), "gemma2"
  family, size = model.split(" ")
  return config_from_dict(design_bench.DICTS[family](design_bench.SIZES[size])), family


# ---- weights ------------------------------------------------------------------------------------------

def _weights(case, seed):
  """Every tensor of the model, from the seed and the tensor's name."""
  cfg, family = _config(case["model"])
  dtype = getattr(torch, case["dtype"])
  specs = {s.name: s for s in tensor_specs(cfg.model_spec()) if not s.optional}
  out = {}
  for name, s in specs.items():
    gen = torch.Generator(device="cuda").manual_seed((seed << 32) + zlib.crc32(name.encode()))
    if s.kind == "table":
      order = torch.rand((s.shape[0], s.choices), generator=gen, device="cuda").argsort(dim=1)
      out[name] = order[:, :s.shape[1]].to(torch.int32).contiguous()
      continue
    # (drawn in the storage type where matrices are large: a model has billions of them)
    t = torch.randn(s.shape, generator=gen, device="cuda", dtype=dtype if s.kind == "matrix" else torch.float32)
    out[name] = _shaped(family, name, s, t, specs).to(dtype)
  if "head" in out:  # the output rows lean towards the row that leads to them
    follow = _follower(seed, out["embed"].shape[0])
    out["head"] = out["head"].mul_(_HEAD_STD[family] * 0.5).index_add_(
        0, follow, out["embed"], alpha=_HEAD_STD[family])
  return out


def _follower(seed, vocab):
  gen = torch.Generator(device="cuda").manual_seed((seed << 32) + 5)
  return torch.randperm(vocab, generator=gen, device="cuda")


_HEAD_STD = {"sapivik": 0.25, "zesapel": 0.3}


def _shaped(family, name, s, t, specs):
  """Standard normal values made into those of a tensor of this name."""
  last = name.rsplit(".", 1)[-1]
  if family == "gemma2":
    if s.kind == "matrix":
      return t.mul_(s.shape[-1] ** -0.5)
    if "post_" in name:  # branches so small that the likeliest token of the tied output is clear
      width, vocab = s.shape[0], specs["model.embed_tokens.weight"].shape[0]
      share = (math.log(vocab) + WANTED_LOGPROB) / math.sqrt(width)
      branches = sum("post_" in n for n in specs)
      return t * 0.05 + (math.sqrt((1.0 / share ** 2 - 1.0) / branches) - 1.0)
    return t * 0.1
  if name in ("embed", "head"):
    return t
  if name == "pos":
    return t.mul_(0.1)
  if last in ("conv", "canon1"):
    return t.mul_(0.5 if last == "conv" else 0.2)
  if last == "router":
    return t.mul_(2.5 * s.shape[-1] ** -0.5)
  if s.kind == "matrix" and last not in ("mix", "in", "out"):
    return t.mul_(s.shape[-1] ** -0.5)
  if name.endswith(".mix.in"):
    return t.mul_(s.shape[-1] ** -0.5)
  if ".hc" in name:
    streams = s.shape[-1]
    if last == "in":
      return 1.0 / streams + 0.1 * t
    if last == "out":
      return 1.0 + 0.1 * t
    return torch.eye(streams, device=t.device) + 0.05 * t
  if last == "lower":  # least share of the state that is kept
    return torch.sigmoid(t)
  if name.endswith(".f.b"):
    return 2.0 + t
  if last == "correction":
    return t * 0.002
  if last == "A_log":  # rates of 1 to 16, steps of 0.001 to 0.1
    return torch.special.ndtr(t) * math.log(16.0)
  if last == "dt_bias":
    step = torch.exp(math.log(0.001) + torch.special.ndtr(t) * math.log(100.0))
    return step + torch.log(-torch.expm1(-step))
  if last == "w0":
    return t - 2.0
  if s.kind == "gain":
    return 1.0 + 0.1 * t
  return t * 0.5  # sinks and offsets


# ---- a pass ---------------------------------------------------------------------------------------------

def _engine_config(case):
  lengths = _lengths(case)
  page = 64
  longest = max(lengths) + 1 + (max(_new_tokens(case)) if case["new"] else 0)
  if case["kind"] == "decode":
    longest = min(LONGEST, 2 * max(lengths) + 1024)
  portion = sum(lengths) if case["kind"] == "prompt" else PORTION
  slots = case["slots"] if case["kind"] == "generate" else case["batch"]
  return EngineConfig(activation_dtype=case["dtype"], page_size=page, batch_size=slots, max_seq_len=longest,
                      max_cache_tokens=slots * (longest + page), max_num_issue_tokens=max(portion, 512),
                      intermediate_steps=case["burst"])


def prepare(case, seed):
  cfg, _ = _config(case["model"])
  engine = Engine(cfg, _weights(case, seed), _engine_config(case), device="cuda")
  vocab = engine.model.spec.vocab_size
  state = dict(kind=case["kind"], engine=engine, prompts=_prompts(case, seed, vocab, case["kind"] == "decode"))
  if case["kind"] == "generate":
    state["params"] = [SamplingParams(temperature=0.0, max_decode_steps=n) for n in _new_tokens(case)]
  if case["kind"] == "decode":
    if engine._decode_runner is not None:  # (as trace replay sets it: the graphs' logits are wanted)
      engine._decode_runner.keep_logits = True
    state["follow"] = random.Random(seed).choices(range(16, vocab), k=4096)
    _start_requests(state)
  return state


def _start_requests(state):
  engine = state["engine"]
  state["slots"] = []
  for i, p in enumerate(state["prompts"]):
    slot = engine.open_request(i)
    for at in range(0, len(p) - 1, PORTION):
      engine.step_raw([StepEntry(slot, p[at:min(at + PORTION, len(p) - 1)])])
    state["slots"].append(slot)
  state["next"] = [p[-1] for p in state["prompts"]]
  state["room"] = engine.engine_config.max_seq_len - max(len(p) - 1 for p in state["prompts"])
  state["done"] = 0


def run(state):
  engine, kind = state["engine"], state["kind"]
  if kind == "generate":
    results = engine.generate(state["prompts"], state["params"])
    return torch.tensor([t for r in results for t in r.output_token_ids])
  if kind == "score":
    return torch.tensor(engine.score_tokens(state["prompts"][0]))
  if kind == "prompt":
    slots = [engine.open_request(i) for i in range(len(state["prompts"]))]
    logits = engine.step_raw([StepEntry(s, p, (len(p) - 1,)) for s, p in zip(slots, state["prompts"])])
    for s in slots:
      engine.close_request(s)
    return logits
  if state["done"] == state["room"]:
    for s in state["slots"]:
      engine.close_request(s)
    _start_requests(state)
  logits = engine.step_raw([StepEntry(s, [t], (0,)) for s, t in zip(state["slots"], state["next"])], from_graph=True)
  state["done"] += 1
  follow = state["follow"]
  state["next"] = [follow[(state["done"] * 31 + 7 * i) % len(follow)] for i in range(len(state["next"]))]
  return logits


# ---- what a pass cannot do without --------------------------------------------------------------------------

@functools.cache
def _sizes(model):
  """Numbers of values: matrices that every token multiplies and that a step reads, all experts' likewise."""
  cfg, family = _config(model)
  d = cfg.to_dict()
  specs = [s for s in tensor_specs(cfg.model_spec()) if not s.optional]
  runs = {}  # how often a layer runs in one step
  if family == "sapivik":
    loop = d["loop"]
    runs = {i: loop["times"] for i in range(loop["start"], loop["stop"])}
  dense = expert = expert_read = top = experts = read = 0
  for s in specs:
    n = math.prod(s.shape)
    if s.kind == "table" or s.name in ("embed", "pos"):
      continue
    times = runs.get(int(s.name[1:].split(".")[0]), 1) if s.name[0] == "l" and s.name[1].isdigit() else 1
    if ".mlp.e" in s.name and family != "gemma2":
      expert += n * times
      expert_read += n
    elif s.kind == "matrix" and s.name not in ("head", "model.embed_tokens.weight"):
      dense += n * times
      read += n
    elif s.kind != "matrix":
      read += n
  if family != "gemma2":
    mlp = next(layer["mlp"] for layer in d["layers"] if layer["mlp"]["kind"] == "moe")
    experts, top = mlp["router"]["experts"], mlp["router"]["top"]
  vocab, width = next(s.shape for s in specs if s.name in ("head", "model.embed_tokens.weight"))
  return dict(dense=dense, expert=expert, expert_read=expert_read, experts=experts, top=top, read=read, vocab=vocab, width=width)


def _attention(model):
  """Of every attention layer that runs: (window or None, flops per query and key, cached values per token); of
  all recurrent layers: values of state per request."""
  cfg, family = _config(model)
  d = cfg.to_dict()
  layers, state = [], 0
  if family == "gemma2":
    types = d.get("layer_types") or ["sliding_attention" if i % 2 == 0 else "full_attention" for i in range(d["num_hidden_layers"])]
    for t in types:
      layers.append((d["sliding_window"] if t == "sliding_attention" else None, 4 * d["num_attention_heads"] * d["head_dim"],
                     2 * d["num_key_value_heads"] * d["head_dim"]))
    return layers, state
  loop = d.get("loop") or {"start": 0, "stop": 0, "times": 1}
  for i, layer in enumerate(d["layers"]):
    m = layer["mixer"]
    for _ in range(loop["times"] if loop["start"] <= i < loop["stop"] else 1):
      if layer["type"] == "attention":
        layers.append((None, 4 * m["heads"] * m["dim"], m["kv_heads"] * m["dim"]))
      elif layer["type"] == "latent_attention":
        layers.append((m["mask"]["size"], 2 * m["heads"] * (2 * m["kv_rank"] + m["rot_dim"]), m["kv_rank"] + m["rot_dim"]))
      elif layer["type"] == "mamba2":
        state += m["heads"] * m["vdim"] * m["state"]
      else:
        state += m["heads"] * m["dim"] * m.get("vdim", m["dim"])
  return layers, state


def work(case):
  z = _sizes(case["model"])
  layers, state = _attention(case["model"])
  item = 2 if case["dtype"] == "bfloat16" else 4
  total = dict(bytes=0.0, flops=0.0)

  def step(tokens, rows):
    """One step's weights and products: `tokens` rows through the layers, `rows` through the output."""
    touched = min(1.0, tokens * z["top"] / z["experts"]) if z["experts"] else 0.0
    total["bytes"] += item * (z["read"] + z["expert_read"] * touched + z["vocab"] * z["width"] * (rows > 0))
    total["bytes"] += tokens * z["width"] * item + rows * z["vocab"] * 4
    total["flops"] += 2.0 * tokens * z["dense"] + 2.0 * rows * z["vocab"] * z["width"]
    if z["experts"]:
      total["flops"] += 2.0 * tokens * z["top"] * z["expert"] / z["experts"]

  def sequence(start, n):
    """One request's attention and states in a step that adds n tokens to `start`."""
    for window, per_pair, kept in layers:
      w = window or LONGEST * 2
      seen = sum(min(p + 1, w) for p in range(start, start + n))
      total["flops"] += float(per_pair) * seen
      total["bytes"] += item * kept * (min(start, w) + n)
    total["bytes"] += 4.0 * state * (2 if start else 1)
    total["flops"] += 5.0 * state * n

  lengths = _lengths(case)
  if case["kind"] == "prompt":
    step(sum(lengths), len(lengths))
    for n in lengths:
      sequence(0, n)
  elif case["kind"] == "score":
    n = lengths[0] - 1
    for at in range(0, n, 256):  # (score_tokens goes by portions of 256)
      step(min(256, n - at), min(256, n - at))
      sequence(at, min(256, n - at))
  elif case["kind"] == "decode":
    step(len(lengths), len(lengths))
    for n in lengths:
      sequence(n, 1)
  else:
    new = _new_tokens(case)
    steps = -(-sum(new) // case["slots"])  # as many as full slots would need
    for _ in range(steps):
      step(0, case["slots"])
      total["bytes"] -= case["slots"] * z["vocab"] * 4  # the logits stay inside
    for n, m in zip(lengths, new):
      total["flops"] += 2.0 * (n + m) * z["dense"]
      if z["experts"]:
        total["flops"] += 2.0 * (n + m) * z["top"] * z["expert"] / z["experts"]
      sequence(0, n)
      for k in range(m - 1):
        sequence(n + k, 1)
  return total


def tolerance(case):
  if case["kind"] == "generate":
    return {"differ": 0.01}
  if case["dtype"] == "float32":  # 3e-7 off the exact values, measured
    return {"rel": 3e-6, "max": 1e-4}
  return {"rel": 0.03, "max": 0.3}  # 0.002 to 0.01 off, the most with the most layers


# ---- the same in 64 bits --------------------------------------------------------------------------------------

def exact(case, seed):
  if case["kind"] == "generate":
    return None  # tokens, no computed numbers
  cfg, family = _config(case["model"])
  d = cfg.to_dict()
  w = _weights(case, seed)
  forward = {"gemma2": _gemma2, "sapivik": _sapivik, "zesapel": _zesapel}[family]
  prompts = _prompts(case, seed, w["embed" if "embed" in w else "model.embed_tokens.weight"].shape[0], case["kind"] == "decode")
  if case["kind"] == "score":
    tokens = torch.tensor(prompts[0], device="cuda")
    logits = forward(d, w, tokens[:-1], slice(None))
    return torch.log_softmax(logits, -1).gather(1, tokens[1:, None])[:, 0]
  rows = [forward(d, w, torch.tensor(p, device="cuda"), slice(-1, None)) for p in prompts]
  return torch.cat(rows)


def _rms(x, eps, weight=None, plus=0.0):
  y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)
  return y if weight is None else y * (weight.double() + plus)


def _mm(x, w):
  """x times a weight's transpose, in 64 bits, by blocks of the weight's rows."""
  if w.shape[0] <= 32768:
    return x @ w.double().T
  return torch.cat([x @ part.double().T for part in w.split(32768)], dim=-1)


def _turn(x, dims, base, neighbours=False):
  """x [T, heads, n]: the first `dims` dims turn by position * base^(-2i/dims)."""
  half = dims // 2
  angle = (torch.arange(x.shape[0], device=x.device, dtype=torch.float64)[:, None, None]
           * base ** (-2.0 * torch.arange(half, device=x.device, dtype=torch.float64) / dims))
  c, s = torch.cos(angle), torch.sin(angle)
  out = x.clone()
  first, second = (slice(0, dims, 2), slice(1, dims, 2)) if neighbours else (slice(0, half), slice(half, dims))
  out[..., first] = x[..., first] * c - x[..., second] * s
  out[..., second] = x[..., second] * c + x[..., first] * s
  return out


def _attend(q, k, v, scale, cap=0.0, window=None, sink=None):
  """q [T, H, d], k [T, G, d], v [T, G, dv] -> [T, H, dv]: causal, in blocks of 1,024 queries."""
  t, heads, groups = q.shape[0], q.shape[1], k.shape[1]
  at = torch.arange(t, device=q.device)
  out = []
  for lo in range(0, t, 1024):
    hi = min(lo + 1024, t)
    first = 0 if window is None else max(0, lo - window + 1)
    qb = q[lo:hi].reshape(hi - lo, groups, heads // groups, -1)
    s = torch.einsum("tgrd,sgd->grts", qb, k[first:hi]) * scale
    if cap:
      s = cap * torch.tanh(s / cap)
    gap = at[lo:hi, None] - at[None, first:hi]
    s = s.masked_fill((gap < 0) | (gap >= (window or t)), -math.inf)
    if sink is not None:
      extra = sink.double().reshape(groups, -1, 1, 1).expand(-1, -1, hi - lo, 1)
      p = torch.softmax(torch.cat([s, extra], -1), -1)[..., :-1]
    else:
      p = torch.softmax(s, -1)
    out.append(torch.einsum("grts,sgd->tgrd", p, v[first:hi]).reshape(hi - lo, heads, -1))
  return torch.cat(out)


def _gemma2(d, w, tokens, rows):
  eps, heads, groups, n = d["rms_norm_eps"], d["num_attention_heads"], d["num_key_value_heads"], d["head_dim"]
  table = w["model.embed_tokens.weight"]
  scale = torch.tensor(d["hidden_size"] ** 0.5).to(table.dtype).item()  # the factor is kept in the storage type
  x = table[tokens].double() * scale
  t = len(tokens)
  for i in range(d["num_hidden_layers"]):
    p = f"model.layers.{i}."
    y = _rms(x, eps, w[p + "input_layernorm.weight"], 1.0)
    q = _turn(_mm(y, w[p + "self_attn.q_proj.weight"]).reshape(t, heads, n), n, d["rope_theta"])
    k = _turn(_mm(y, w[p + "self_attn.k_proj.weight"]).reshape(t, groups, n), n, d["rope_theta"])
    v = _mm(y, w[p + "self_attn.v_proj.weight"]).reshape(t, groups, n)
    types = d.get("layer_types")
    local = types[i] == "sliding_attention" if types else i % 2 == 0
    o = _attend(q, k, v, d["query_pre_attn_scalar"] ** -0.5, d["attn_logit_softcapping"], d["sliding_window"] if local else None)
    x = x + _rms(_mm(o.reshape(t, -1), w[p + "self_attn.o_proj.weight"]), eps, w[p + "post_attention_layernorm.weight"], 1.0)
    y = _rms(x, eps, w[p + "pre_feedforward_layernorm.weight"], 1.0)
    y = torch.nn.functional.gelu(_mm(y, w[p + "mlp.gate_proj.weight"]), approximate="tanh") * _mm(y, w[p + "mlp.up_proj.weight"])
    x = x + _rms(_mm(y, w[p + "mlp.down_proj.weight"]), eps, w[p + "post_feedforward_layernorm.weight"], 1.0)
  cap = d["final_logit_softcapping"]
  return cap * torch.tanh(_mm(_rms(x[rows], eps, w["model.norm.weight"], 1.0), table) / cap)


def _sapivik(d, w, tokens, rows):
  eps, loop, t = d["norm"]["eps"], d["loop"], len(tokens)
  x = first = w["embed"][tokens].double()
  order = [(i, False) for i in range(loop["start"])]
  order += [(i, n > 0 and i == loop["start"]) for n in range(loop["times"]) for i in range(loop["start"], loop["stop"])]
  order += [(i, False) for i in range(loop["stop"], len(d["layers"]))]
  for i, again in order:
    layer, p = d["layers"][i], f"l{i}"
    m, mlp = layer["mixer"], layer["mlp"]
    x = x + first if again else x
    y = _rms(x, eps, w[p + ".norm1"])
    if layer["type"] == "attention":
      q = _mm(y, w[p + ".mix.q"]).reshape(t, m["heads"], -1)
      v = _mm(y, w[p + ".mix.k"]).reshape(t, m["kv_heads"], -1)  # values are the keys as projected
      q, k = (_rms(_turn(u, m["rot"]["dims"], m["rot"]["base"], neighbours=True), eps) for u in (q, v))
      o = _attend(q, k, v, m["scale"], m["softcap"]).reshape(t, -1) * torch.sigmoid(_mm(y, w[p + ".mix.g"]))
    else:
      q = torch.nn.functional.silu(_mm(y, w[p + ".mix.q"])).reshape(t, m["heads"], -1)
      v = _mm(y, w[p + ".mix.v"]).reshape(t, m["heads"], -1)
      low = w[p + ".mix.lower"].double()
      f = (low + (1.0 - low) * torch.sigmoid(_mm(y, w[p + ".mix.f"]) + w[p + ".mix.f.b"].double())).reshape(t, m["heads"], -1)
      state = torch.zeros(m["heads"], m["dim"], m["vdim"], device=x.device, dtype=torch.float64)
      o = torch.empty_like(v)
      kept = 1.0 - f
      for n in range(t):
        state = state * f[n, :, :, None] + kept[n, :, :, None] * v[n, :, None, :]
        o[n] = torch.bmm(q[n, :, None, :], state)[:, 0]
      o = _rms(o, eps, w[p + ".mix.norm"]).reshape(t, -1)
    x = x + d["residual_mult"] * _rms(_mm(o, w[p + ".mix.o"]), eps, w[p + ".norm1b"])
    y, p = _rms(x, eps, w[p + ".norm2"]), p + ".mlp"
    if mlp["kind"] == "dense":
      g = _mm(y, w[p + ".gate"]).clamp(max=mlp["limit"])
      z = _mm(g * torch.sigmoid(1.702 * g) * (_mm(y, w[p + ".up"]).clamp(-mlp["limit"], mlp["limit"]) + 1.0), w[p + ".down"])
    else:
      r = mlp["router"]
      score = torch.softmax(_mm(y, w[p + ".router"]), -1)
      chosen = (score + w[p + ".correction"].double()).topk(r["top"], dim=-1).indices
      share = torch.zeros_like(score).scatter(1, chosen, score.gather(1, chosen) * r["scale"])
      z = share[:, r["experts"]:].sum(-1, keepdim=True) * y  # identity experts
      part = lambda e, u: _mm(torch.nn.functional.silu(_mm(u, w[f"{p}.{e}.gate"])) * _mm(u, w[f"{p}.{e}.up"]), w[f"{p}.{e}.down"])
      for e in range(r["experts"]):
        at = share[:, e].nonzero()[:, 0]
        z.index_add_(0, at, part(f"e{e}", y[at]) * share[at, e, None])
      z = z + torch.sigmoid(_mm(y, w[p + ".shared.sg"])) * part("shared", y)
    x = x + d["residual_mult"] * _rms(z, eps, w[f"l{i}.norm2b"])
  return _mm(_rms(x[rows], eps, w["final.norm"]), w["head"])


def _convolve(x, taps, bias=None):
  """x [T, C], taps [C, K], the last tap for the token itself, nothing before the start."""
  k = taps.shape[1]
  padded = torch.cat([x.new_zeros(k - 1, x.shape[1]), x])
  y = sum(padded[j:j + x.shape[0]] * taps[:, j].double() for j in range(k))
  return y if bias is None else y + bias.double()


def _zesapel(d, w, tokens, rows):
  eps, t = d["norm"]["eps"], len(tokens)
  x = w["embed"][tokens].double() * d["embedding"]["scale"] + w["pos"][:t].double()
  lanes = torch.stack([x] * d["streams"])
  for i, layer in enumerate(d["layers"]):
    for sub, at in (("mix", 1), ("mlp", 2)):
      p = f"l{i}"
      h = _rms(torch.einsum("s,stw->tw", w[f"{p}.hc{at}.in"].double(), lanes), eps, w[f"{p}.norm{at}"])
      if sub == "mix":
        h = h + _convolve(h, w[p + ".canon1"])
        y = _ZESAPEL_MIXERS[layer["type"]](layer["mixer"], w, p + ".mix", h, eps)
      else:
        top, y = layer["mlp"]["router"]["top"], torch.zeros_like(h)
        table = w[p + ".mlp.table"][tokens]
        for e in range(layer["mlp"]["router"]["experts"]):
          at_e = (table == e).any(-1).nonzero()[:, 0]
          y.index_add_(0, at_e, _mm(torch.nn.functional.gelu(_mm(h[at_e], w[f"{p}.mlp.e{e}.up"])), w[f"{p}.mlp.e{e}.down"]) / top)
      lanes = torch.einsum("sr,stw->rtw", w[f"{p}.hc{at}.mix"].double(), lanes) + w[f"{p}.hc{at}.out"].double()[:, None, None] * y
  return _mm(_rms(lanes.sum(0)[rows], eps, w["final.norm"]), w["head"])


def _latent(m, w, p, h, eps):
  t, heads, dim, rank = h.shape[0], m["heads"], m["dim"], m["kv_rank"]
  q = _mm(_rms(_mm(h, w[p + ".dq"]), eps, w[p + ".dq.norm"]), w[p + ".uq"]).reshape(t, heads, -1)
  down = _mm(h, w[p + ".dkv"])
  c = _rms(down[:, :rank], eps, w[p + ".dkv.norm"])
  turned = _turn(down[:, None, rank:], m["rot"]["dims"], m["rot"]["base"]).expand(-1, heads, -1)
  q = torch.cat([q[..., :dim], _turn(q[..., dim:], m["rot"]["dims"], m["rot"]["base"])], -1)
  k = torch.cat([_mm(c, w[p + ".uk"]).reshape(t, heads, dim), turned], -1)
  v = _mm(c, w[p + ".uv"]).reshape(t, heads, -1)
  o = _attend(q, k, v, m["scale"], window=m["mask"]["size"], sink=w[p + ".sink"])
  return _mm((o * torch.sigmoid(_mm(h, w[p + ".g"]))[..., None]).reshape(t, -1), w[p + ".o"])


def _delta(m, w, p, h, eps):
  t, heads = h.shape[0], m["heads"]
  r, k, v = (_mm(h, w[f"{p}.{n}"]).reshape(t, heads, -1) for n in "rkv")
  low = _mm(torch.tanh(_mm(h, w[p + ".w1"])), w[p + ".w2"]) + w[p + ".w0"].double()
  decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(low)).reshape(t, heads, -1)
  take = torch.sigmoid(_mm(h, w[p + ".a"]) + w[p + ".a.b"].double()).reshape(t, heads, -1)
  unit = k * torch.rsqrt(k.square().sum(-1, keepdim=True) + 1e-6)
  state = torch.zeros(heads, m["dim"], m["dim"], device=h.device, dtype=torch.float64)
  o = torch.empty_like(v)
  for n in range(t):
    seen = torch.bmm(unit[n, :, None, :], state)
    state = (decay[n, :, :, None] * state - (take[n] * unit[n])[:, :, None] * seen + k[n, :, :, None] * v[n, :, None, :])
    o[n] = torch.bmm(r[n, :, None, :], state)[:, 0]
  o = _rms(o, eps).reshape(t, -1) * w[p + ".norm"].double() * torch.sigmoid(_mm(h, w[p + ".g"]))
  return _mm(o, w[p + ".o"])


def _state_space(m, w, p, h, eps):
  t, heads, n = h.shape[0], m["heads"], m["state"]
  inner = heads * m["vdim"]
  z, xbc, dt = _mm(h, w[p + ".in"]).split([inner, inner + 2 * n, heads], dim=-1)  # (one group)
  xbc = torch.nn.functional.silu(_convolve(xbc, w[p + ".conv"], w[p + ".conv.b"]))
  x, b, c = xbc.split([inner, n, n], dim=-1)
  x = x.reshape(t, heads, -1)
  dt = torch.nn.functional.softplus(dt + w[p + ".dt_bias"].double())
  keep = torch.exp(-torch.exp(w[p + ".A_log"].double()) * dt)
  state = torch.zeros(heads, n, m["vdim"], device=h.device, dtype=torch.float64)
  y = torch.empty_like(x)
  for i in range(t):
    state = state * keep[i, :, None, None] + (dt[i, :, None] * b[i])[:, :, None] * x[i, :, None, :]
    y[i] = torch.matmul(c[i], state)
  y = (y + w[p + ".D"].double()[:, None] * x).reshape(t, -1) * torch.nn.functional.silu(z)
  y = _rms(y.reshape(t, m["norm_groups"], -1), eps).reshape(t, -1) * w[p + ".norm"].double()
  return _mm(y, w[p + ".o"])


_ZESAPEL_MIXERS = {"latent_attention": _latent, "general_delta": _delta, "mamba2": _state_space}
