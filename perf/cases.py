"""The work a user has this framework do, as cases that can be timed and compared.

A case is a dict of plain values.  `prepare` makes what a program holds before the call (weights bound to a plan, prompts,
activations), `run` is one pass through the public entry points, `exact` the same result in 64 bits by plain torch.

Kinds of cases:
  product  one quantised projection of a few rows on device buffers (gf_matmul), what a host engine calls per operator
  decode   teacher-forced passes behind a context, candidates selected and read after each, rows published; then the context
           is taken back, so that every pass sees the same positions (rows = 2: the verification of one drafted token)
  prompt   a plan reset and a whole prompt ingested; the logits behind it
  chat     a request to the speculative engine: a short prompt into both plans, then generation
  batch    several conversations on one plan: slots given back, prompts ingested, steps of one token each
Weights are random, in the formats and distributions of guffin_b200.synthetic; layers cut their matrices out of one pool
per format at places of their own, so that a 12B plan is made in a second or two.
"""
import math

import numpy as np
import torch

from guffin_b200 import engine as ge
from guffin_b200 import lib
from guffin_b200 import model as gm
from guffin_b200 import synthetic as syn

FORMATS = {"q4_k": syn.Q4_K, "q6_k": syn.Q6_K, "q8_0": syn.Q8_0}
GEMMA = ("gemma3-12b", "gemma3-270m", "gemma2-9b")
RETAIN = 40                       # candidates per row: the default top_k of the sampler
VOCAB = 32768                     # of the layered models


def listed():
    layered = dict(layers=8, width=2048, heads=16, ff=8192)
    zasevik = dict(model="zasevik", rank=512, experts=0, top=0, expert_ff=0, shared_ff=0, **layered)
    tufirax = dict(model="tufirax", kv_heads=4, state_heads=64, **layered)
    return [
        # The smallest call: a projection of the drafter, 1.4 MB of weights, all latency.
        dict(name="product-q8_0-640x2048-1", kind="product", format="q8_0", k=640, n=2048, rows=1),
        # The projection a target spends its time in, two rows of a verification pass.
        dict(name="product-q4_k-3840x15360-2", kind="product", format="q4_k", k=3840, n=15360, rows=2),
        # Plain decoding of a small model: one row, an f32 cache, the whole vocabulary for a head.
        dict(name="decode-270m-512", kind="decode", model="gemma3-270m", context=512, rows=1, steps=8),
        # A drafter (or small model) taking in a prompt of no round length.
        dict(name="prompt-270m-777", kind="prompt", model="gemma3-270m", tokens=777),
        # The headline: a short question to the pair, answered speculatively.
        dict(name="chat-12b-48", kind="chat", model="gemma3-12b", tokens=48, generate=32),
        # The verification pass of a long conversation.
        dict(name="verify-12b-2048", kind="decode", model="gemma3-12b", context=2048, rows=2, steps=1),
        # A long prompt into the large model: the largest case.
        dict(name="prompt-12b-2048", kind="prompt", model="gemma3-12b", tokens=2048),
        # Serving: eight conversations share the weights, prompts of unequal length, then steps.
        dict(name="batch-9b-8", kind="batch", model="gemma2-9b", streams=8, tokens=192, steps=16),
        # Layered models: dense and routed layers in turn, a long prompt; dense layers, decoding.
        dict(zasevik, name="prompt-zasevik-experts-2048", kind="prompt", tokens=2048, experts=64, top=6, expert_ff=1024, shared_ff=2048),
        dict(zasevik, name="decode-zasevik-2048", kind="decode", context=2048, rows=1, steps=8),
        # Attention and state-space layers in turn: decoding, and a prompt that fills its last chunk half.
        dict(tufirax, name="decode-tufirax-2048", kind="decode", context=2048, rows=1, steps=8),
        dict(tufirax, name="prompt-tufirax-1500", kind="prompt", tokens=1500),
    ]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["product"] * 4 + ["decode"] * 3 + ["prompt"] * 3 + ["batch", "chat"])
    if kind == "product":
        name = rng.choice(sorted(FORMATS))
        unit = 128 if name == "q8_0" else 256
        k = unit * _spread(rng, 2, 15360 // unit)
        return dict(kind=kind, format=name, k=k, n=_spread(rng, 64, min(262144, 120_000_000 // k)), rows=rng.randint(1, 8))
    if kind == "chat":
        return dict(kind=kind, model="gemma3-12b", tokens=rng.randint(3, 64), generate=rng.randint(8, 40))
    if kind == "batch":
        return dict(kind=kind, model="gemma2-9b", streams=rng.randint(2, 12), tokens=_spread(rng, 20, 256), steps=rng.randint(2, 16))
    model = rng.choice(GEMMA + ("zasevik", "tufirax") * 2)
    case = dict(kind=kind, model=model)
    if model not in GEMMA:
        heads, size = rng.choice([8, 12, 16, 32]), rng.choice([1536, 2048, 2560, 3840])
        case.update(layers=rng.randint(2, 8), width=size, heads=heads, ff=8 * rng.randint(size // 4, size // 2))
        if model == "zasevik":
            experts = rng.choice([0, 32, 64])
            case.update(rank=rng.choice([384, 512]), experts=experts, top=rng.randint(2, 8) if experts else 0,
                        expert_ff=8 * rng.randint(64, 160) if experts else 0, shared_ff=8 * rng.randint(64, 256) if experts else 0)
        else:
            case.update(kv_heads=heads // 4, state_heads=rng.choice([32, 64, 96]))
    if kind == "prompt":
        return dict(case, tokens=_spread(rng, 66, 2048))
    rows = rng.choice([1, 1, 2, 4])
    return dict(case, context=_spread(rng, 16, 3000), rows=rows, steps=8 // rows)


# ---------------------------------------------------------------------------- weights

def _generator(seed):
    g = torch.Generator("cuda")
    g.manual_seed(seed)
    return g


def _blocks(fmt, count, sigma, g):
    """`count` native blocks as bytes on the GPU, distributed as guffin_b200.synthetic says."""
    def scale(shape):
        return (torch.randn(shape, generator=g, device="cuda") * sigma).abs().half().clamp_min(6e-8).view(torch.uint8)
    raw = torch.randint(0, 256, (count, syn.BLOCK_BYTES[fmt]), dtype=torch.uint8, device="cuda", generator=g)
    if fmt == syn.Q4_K:
        raw[:, 0:4] = scale((count, 2))
    elif fmt == syn.Q6_K:
        raw[:, 192:208] = torch.randint(-64, 64, (count, 16), dtype=torch.int8, device="cuda", generator=g).view(torch.uint8)
        raw[:, 208:210] = scale((count, 1))
    else:
        raw[:, 0:2] = scale((count, 1))
        raw[:, 2:][raw[:, 2:] == 128] = 0          # codes from -127 to 127
    return raw


_SIGMA = {syn.Q4_K: 1e-3, syn.Q6_K: 1e-3, syn.Q8_0: 1e-2}
_TABLE_RMS = {syn.Q6_K: 685.0, syn.Q8_0: 73.3}


def _gemma_weights(name, seed):
    """(GGUF tensor name, value) of a Gemma plan: (format, K, N, bytes) or an f32 vector."""
    config, g, rng = syn.model_config(name), _generator(seed), np.random.default_rng(seed)
    types, shapes, hidden, vocab = syn.tensor_types(name, config), syn.matrix_shapes(config), config["hidden"], config["vocab"]
    for table in ("token_embd.weight", "output.weight"):
        if table in types:
            fmt = types[table]
            count = vocab * hidden // syn.BLOCK_ELEMENTS[fmt]
            yield table, (fmt, hidden, vocab, _blocks(fmt, count, 1.0 / (_TABLE_RMS[fmt] * math.sqrt(hidden)), g).reshape(-1).cpu().numpy())
    pools, slack, cut = {}, 20011, 0
    for layer in range(config["layers"]):
        for short, (k, n) in shapes.items():
            key = f"blk.{layer}.{short}.weight"
            fmt = types[key]
            if fmt not in pools:
                pools[fmt] = _blocks(fmt, max(a * b for a, b in shapes.values()) // syn.BLOCK_ELEMENTS[fmt] + slack, _SIGMA[fmt], g).reshape(-1).cpu().numpy()
            cut = (cut + 7919) % slack
            first = cut * syn.BLOCK_BYTES[fmt]
            yield key, (fmt, k, n, pools[fmt][first:first + syn.weight_bytes(fmt, k, n)])
        vectors = {"attn_norm": hidden, "post_attention_norm": hidden, "ffn_norm": hidden, "post_ffw_norm": hidden}
        if config["uses_qk_norm"]:
            vectors.update(attn_q_norm=config["head_dim"], attn_k_norm=config["head_dim"])
        for short, size in vectors.items():
            yield f"blk.{layer}.{short}.weight", (1.0 + 0.1 * rng.standard_normal(size)).astype(np.float32)
    yield "output_norm.weight", (1.0 + 0.1 * rng.standard_normal(hidden)).astype(np.float32)


def _layered_config(case):
    dense = syn.dense_mlp(case["ff"])
    if case["model"] == "zasevik":
        routed = syn.expert_mlp(case["expert_ff"], case["experts"], case["top"], 7.0, case["shared_ff"], 7.0) if case["experts"] else dense
        return syn.zasevik_config(case["width"], case["layers"], case["heads"], 128, 128, case["rank"], VOCAB, [dense, routed])
    kinds = [syn.tufirax_attention(case["heads"], case["kv_heads"], 128, ff=case["ff"]),
             syn.tufirax_state_space(case["state_heads"], 64, 128, groups=8, norm_groups=8)]
    return syn.tufirax_config(case["width"], VOCAB, [kinds[i % 2] for i in range(case["layers"])])


def _layered_weights(case, config, seed):
    """(tensor name, array): bfloat16 bits of matrices, f32 vectors."""
    g, rng = _generator(seed), np.random.default_rng(seed)
    shapes = (syn.zasevik_shapes if case["model"] == "zasevik" else syn.tufirax_shapes)(config)
    pools, slack, cut = {}, 200003, 0
    largest = {}
    for shape in shapes.values():
        if len(shape) == 2:
            largest[shape[1]] = max(largest.get(shape[1], 0), shape[0] * shape[1])
    for name, shape in shapes.items():
        if len(shape) == 2:
            fan = shape[1]
            if fan not in pools:
                pool = (torch.randn(largest[fan] + slack, generator=g, device="cuda") / math.sqrt(fan)).bfloat16()
                pools[fan] = pool.view(torch.int16).cpu().numpy().view(np.uint16)
            cut = (cut + 39119) % slack
            yield name, pools[fan][cut:cut + shape[0] * fan].reshape(shape)
        elif name.endswith(".sink"):
            yield name, rng.normal(1.0, 1.0, shape).astype(np.float32)
        elif name.endswith(".dt_bias"):
            steps = np.exp(rng.uniform(math.log(0.001), math.log(0.3), shape))
            yield name, (steps + np.log(-np.expm1(-steps))).astype(np.float32)
        elif name.endswith(".A_log"):
            yield name, np.log(rng.uniform(1.0, 16.0, shape)).astype(np.float32)
        elif name.endswith(".conv.b") or (case["model"] == "zasevik" and ".norm" in name and "dkv" not in name):
            yield name, rng.normal(0.0, 0.2, shape).astype(np.float32)
        else:
            yield name, rng.uniform(0.5, 1.5, shape).astype(np.float32)


def _model(case, seed, context, row_capacity):
    if case["model"] in GEMMA:
        return gm.Model(syn.model_config(case["model"]), _gemma_weights(case["model"], seed), context, row_capacity)
    config = _layered_config(case)
    return gm.Model.described(config, _layered_weights(case, config, seed), context, row_capacity)


# ---------------------------------------------------------------------------- inputs and passes

class _Words:
    """Device memory of a plan as torch sees it; a tensor made from it keeps the plan alive."""

    def __init__(self, owner, pointer, shape):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(pointer, False), shape=shape, typestr="<f4", version=2)


def _logits(model, rows):
    return torch.as_tensor(_Words(model, model.L.gf_model_logits_dev(model.handle), (rows, model.cfg.vocab)), device="cuda")


def _vocab(case):
    return syn.model_config(case["model"])["vocab"] if case["model"] in GEMMA else VOCAB


def _tokens(case, seed, count):
    return np.random.default_rng([seed, 5]).integers(0, _vocab(case), count).astype(np.uint32)


def _batch_lengths(case):
    """Prompts of unequal length around the case's."""
    return [max(1, case["tokens"] * (3 + (3 * i) % 5) // 5) for i in range(case["streams"])]


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    if case["kind"] == "product":
        fmt, k, n, rows = FORMATS[case["format"]], case["k"], case["n"], case["rows"]
        g, L = _generator(seed), lib.load()
        native = _blocks(fmt, n * k // syn.BLOCK_ELEMENTS[fmt], _SIGMA[fmt], g)
        s.weight = torch.empty(L.gf_packed_weight_bytes(fmt, k, n), dtype=torch.uint8, device="cuda")
        lib.check(L.gf_pack_weight(fmt, native.data_ptr(), k, n, s.weight.data_ptr(), None))
        s.x = torch.randn((rows, k), generator=g, device="cuda")
        s.y = torch.empty((rows, n), device="cuda")
        s.workspace = torch.empty(L.gf_matmul_workspace_bytes(fmt, rows, k, n) + 16, dtype=torch.uint8, device="cuda")
        s.arguments = (fmt, s.weight.data_ptr(), s.x.data_ptr(), s.y.data_ptr(), rows, k, n, s.workspace.data_ptr(), None)
        s.matmul = L.gf_matmul
        torch.cuda.synchronize()          # `native` goes back to the allocator
        return s
    if case["kind"] == "prompt":
        s.tokens = _tokens(case, seed, case["tokens"])
        s.model = _model(case, seed, case["tokens"] + 64, 2)
        s.logits = _logits(s.model, 2)
    elif case["kind"] == "decode":
        passes = case["rows"] * case["steps"]
        tokens = _tokens(case, seed, case["context"] + passes)
        s.passes = [tokens[case["context"] + i * case["rows"]:][:case["rows"]] for i in range(case["steps"])]
        s.model = _model(case, seed, case["context"] + passes + 8, passes)
        s.model.prefill(tokens[:case["context"]])
        s.requests = [gm.selection_request(RETAIN)] * case["rows"]
        s.logits = _logits(s.model, case["rows"])
    elif case["kind"] == "chat":
        s.tokens = _tokens(case, seed, case["tokens"])
        context = case["tokens"] + case["generate"] + 16
        s.model = _model(case, seed, context, 2)
        s.draft = _model(dict(model="gemma3-270m"), seed + 1, context, 2)
        s.options = ge.H1Options(ge.sampler_options(seed=seed), 1, 1, 0.7, seed, 0)
        s.engine = ge.H1(s.model, s.draft, s.options)
        s.logits = _logits(s.model, 1)
    else:
        lengths = _batch_lengths(case)
        tokens = _tokens(case, seed, sum(lengths) + case["steps"] * case["streams"])
        ends = np.cumsum(lengths)
        s.prompts = [tokens[e - n:e] for e, n in zip(ends, lengths)]
        s.steps = tokens[ends[-1]:].reshape(case["steps"], case["streams"])
        s.model = _model(case, seed, max(lengths) + case["steps"] + 8, 8)
        s.streams = gm.Streams(s.model, case["streams"])
        s.requests = [gm.selection_request(RETAIN)] * case["streams"]
    return s


def _best(results):
    """The logits of every row's candidates, best first."""
    return np.stack([np.frombuffer(r, np.float32, 2 * RETAIN, 8)[1::2] for r in results])


def run(s):
    kind = s.case["kind"]
    if kind == "product":
        lib.check(s.matmul(*s.arguments))
        return s.y
    if kind == "prompt":
        s.model.reset()
        s.model.prefill(s.tokens)
        return s.logits[s.model.prefill_logits_row]
    if kind == "decode":
        best = []
        for tokens in s.passes:
            s.model.forward(tokens)
            best.append(_best(s.model.select(s.requests)))
            s.model.publish(len(tokens))
        s.model.truncate(s.case["context"])
        return {"best": np.stack(best), "logits": s.logits}
    if kind == "chat":
        s.engine.reseed_schedule(s.options.schedule_seed)          # every pass with the same accepted and rejected drafts
        s.engine.prefill(s.tokens)
        return {"tokens": s.engine.generate(s.case["generate"]), "logits": s.logits}
    for i, prompt in enumerate(s.prompts):
        s.streams.release(i)
        s.streams.prefill(i, prompt)
    best = []
    for tokens in s.steps:
        s.streams.decode(tokens)
        best.append(_best(s.streams.select(s.requests)))
    return {"best": np.stack(best), "logits": np.stack([s.streams.logits(i) for i in range(s.case["streams"])])}


# ---------------------------------------------------------------------------- what a pass cannot do without

def _elements(case):
    """(matrix elements one token's pass multiplies with, bytes of all the matrices a pass over many tokens reads,
    bytes of those that a pass of one token reads) of a case's model, the output head included."""
    if case["model"] in GEMMA:
        config = syn.model_config(case["model"])
        size = config["hidden"] * config["vocab"] + config["layers"] * sum(k * n for k, n in syn.matrix_shapes(config).values())
        nbytes = syn.model_weight_bytes(case["model"])
        return size, nbytes, nbytes
    config = _layered_config(case)
    if case["model"] == "zasevik":
        active, shapes = syn.zasevik_active_parameters(config), syn.zasevik_shapes(config)
    else:
        active, shapes = syn.tufirax_active_parameters(config), syn.tufirax_shapes(config)
    return active, 2 * sum(s[0] * s[1] for n, s in shapes.items() if len(s) == 2 and (n != "embed" or case["model"] == "zasevik")), 2 * active


def _cache(case, context):
    """(bytes of cache and state a pass at this context reads, multiply-adds of a token's attention there)."""
    if case["model"] in GEMMA:
        c = syn.model_config(case["model"])
        seen = [context if not c["sliding_pattern"] or (l + 1) % c["sliding_pattern"] == 0 else min(context, c["sliding_window"]) for l in range(c["layers"])]
        return sum(seen) * c["kv_heads"] * 256 * 2 * (2 if c["kv_f16"] else 4), sum(seen) * c["heads"] * 256 * 2
    if case["model"] == "zasevik":
        return case["layers"] * context * case["rank"] * 2, case["layers"] * context * case["heads"] * 256
    attention, states = (case["layers"] + 1) // 2, case["layers"] // 2
    return (attention * context * case["kv_heads"] * 128 * 4 + states * case["state_heads"] * 64 * 128 * 8,
            attention * context * case["heads"] * 256 + states * case["state_heads"] * 64 * 128 * 3)


def work(case):
    kind = case["kind"]
    if kind == "product":
        k, n, rows = case["k"], case["n"], case["rows"]
        return {"bytes": syn.weight_bytes(FORMATS[case["format"]], k, n) + 4 * rows * (k + n), "flops": 2 * rows * k * n}
    active, whole, single = _elements(case)
    vocab = _vocab(case)
    head = vocab * (syn.model_config(case["model"])["hidden"] if case["model"] in GEMMA else case["width"])
    if kind == "decode":
        read, attended = _cache(case, case["context"])
        rows, steps = case["rows"], case["steps"]
        return {"bytes": steps * (min(whole, single * rows) + read + 4 * rows * vocab), "flops": 2 * steps * rows * (active + attended)}

    def ingest(tokens):
        return 2 * (tokens * (active - head + _cache(case, tokens)[1] // 2) + head)
    if kind == "prompt":
        return {"bytes": whole + _cache(case, case["tokens"])[0] + 4 * vocab, "flops": ingest(case["tokens"])}
    if kind == "chat":
        drafts = dict(model="gemma3-270m")
        cycles = case["generate"] / 1.7
        small = _elements(drafts)
        return {"bytes": (1 + cycles) * (whole + small[1]), "flops": ingest(case["tokens"]) + 2 * cycles * (2 * active + small[0])}
    lengths = _batch_lengths(case)
    read, attended = _cache(case, case["tokens"])
    return {"bytes": whole + case["steps"] * (whole + case["streams"] * (read + 4 * vocab)),
            "flops": sum(ingest(n) for n in lengths) + 2 * case["steps"] * case["streams"] * (active + attended)}


def tolerance(case):
    if case["kind"] == "product":
        return {"rel": 1e-6, "max": 1e-5}          # 32-bit sums: 8e-8 off the exact result
    if case["kind"] == "chat" or (case["model"] in GEMMA and case.get("context", 65) < 65):
        return {"rel": 1e-3, "max": 1e-2}          # prompts of up to 64 tokens and passes are 32-bit throughout, the cache binary16
    if case["model"] in ("gemma3-12b", "gemma2-9b"):
        return {"rel": 5e-3, "max": 5e-2}          # a prompt's products take bf16 operands: up to 1.2e-3 off
    return {"rel": 3e-2, "max": 0.2}               # the same in a few narrow layers: up to 1e-2 off


# ---------------------------------------------------------------------------- the same in 64 bits

def _decoded(value):
    """A native matrix (format, K, N, bytes) as f64 [N, K] on the GPU."""
    fmt, k, n, raw = value
    raw = (raw if isinstance(raw, torch.Tensor) else torch.from_numpy(raw).cuda()).reshape(-1, syn.BLOCK_BYTES[fmt])

    def half(first):
        return raw[:, first:first + 2].contiguous().view(torch.float16).double()
    if fmt == syn.Q8_0:
        return (half(0) * raw[:, 2:].contiguous().view(torch.int8).double()).reshape(n, k)
    if fmt == syn.Q4_K:
        b = raw[:, 4:16].int()
        scales = torch.cat([b[:, 0:4] & 63, (b[:, 8:12] & 15) | ((b[:, 0:4] >> 6) << 4)], 1)
        minima = torch.cat([b[:, 4:8] & 63, (b[:, 8:12] >> 4) | ((b[:, 4:8] >> 6) << 4)], 1)
        codes = raw[:, 16:].reshape(-1, 4, 1, 32)
        codes = torch.cat([codes & 15, codes >> 4], 2).reshape(-1, 8, 32)
        return (codes.double() * (half(0) * scales)[:, :, None] - (half(2) * minima)[:, :, None]).reshape(n, k)
    low, high, scales = raw[:, :128].reshape(-1, 2, 2, 32), raw[:, 128:192].reshape(-1, 2, 1, 32), raw[:, 192:208].contiguous().view(torch.int8)
    low = torch.cat([low & 15, low >> 4], 2)                                         # quarters of 32 codes
    high = torch.cat([(high >> shift) & 3 for shift in (0, 2, 4, 6)], 2)
    codes = (low | (high << 4)).double() - 32.0                                      # [blocks, 2, 4, 32]
    return (codes.reshape(-1, 16, 16) * (half(208) * scales.double())[:, :, None]).reshape(n, k)


def _rms(x, eps, gain=1.0):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * gain


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _attend(q, k, v, seen, scale, cap, sink=None):
    """q [T, H, d], k and v [S, G, d]; `seen` [T, S]."""
    share = q.shape[1] // k.shape[1]
    out = []
    for h in range(q.shape[1]):
        scores = q[:, h] @ k[:, h // share].T * scale
        if cap:
            scores = cap * torch.tanh(scores / cap)
        scores = scores.masked_fill(~seen, -math.inf)
        if sink is None:
            weights = torch.softmax(scores, -1)
        else:
            weights = torch.softmax(torch.cat([scores, sink[h].expand(len(scores), 1)], -1), -1)[:, :-1]
        out.append(weights @ v[:, h // share])
    return torch.stack(out, 1)


def _causal(rows, window=0):
    at = torch.arange(rows, device="cuda")
    seen = at[None, :] <= at[:, None]
    return seen & (at[None, :] + window > at[:, None]) if window else seen


def _turn(x, base, dims, scale=1.0):
    """x [T, H, d] at positions 0..: dimension i turns with dimension i + dims / 2."""
    half = dims // 2
    frequency = torch.tensor([base ** (-2.0 * i / dims) for i in range(half)], dtype=torch.float64, device="cuda")
    angle = torch.arange(len(x), device="cuda").double()[:, None] * scale * frequency
    c, s = torch.cos(angle)[:, None, :], torch.sin(angle)[:, None, :]
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], -1)


def _gemma_logits(case, seed, sequences, want):
    """Logits [len(want[i]), vocab] of the wanted places of every sequence."""
    c, eps = syn.model_config(case["model"]), syn.model_config(case["model"])["rms_eps"]
    lengths = [len(t) for t in sequences]
    at = torch.from_numpy(np.concatenate(sequences).astype(np.int64)).cuda()
    head, x, layer = None, None, {}
    for name, value in _gemma_weights(case["model"], seed):
        if name == "token_embd.weight":
            head, fmt = value, value[0]
            row = value[1] // syn.BLOCK_ELEMENTS[fmt] * syn.BLOCK_BYTES[fmt]
            rows = torch.from_numpy(value[3].reshape(value[2], row)[at.cpu().numpy()]).cuda()
            x = _decoded((fmt, value[1], len(at), rows.reshape(-1))) * math.sqrt(c["hidden"])
            continue
        if name == "output.weight":
            head = value
            continue
        if name == "output_norm.weight":
            layer["output_norm"] = torch.from_numpy(value).cuda().double()
            continue
        index, short = int(name.split(".")[1]), name.split(".")[2]
        layer[short] = value if isinstance(value, tuple) else torch.from_numpy(value).cuda().double()
        if short != ("attn_k_norm" if c["uses_qk_norm"] else "post_ffw_norm"):
            continue
        local = (index + 1) % 6 != 0 if c["sliding_pattern"] == 6 else index % 2 == 0
        h = _rms(x, eps, layer["attn_norm"])
        q, k, v = (h @ _decoded(layer[n]).T for n in ("attn_q", "attn_k", "attn_v"))
        outs, first = [], 0
        for length in lengths:
            part = slice(first, first + length)
            first += length
            qs, ks, vs = (t[part].reshape(length, -1, c["head_dim"]) for t in (q, k, v))
            if c["uses_qk_norm"]:
                qs, ks = _rms(qs, eps, layer["attn_q_norm"]), _rms(ks, eps, layer["attn_k_norm"])
            base, scale = (c["rope_base_local"], c["rope_scale_local"]) if local else (c["rope_base_global"], c["rope_scale_global"])
            qs, ks = _turn(qs, base, c["head_dim"], scale), _turn(ks, base, c["head_dim"], scale)
            seen = _causal(length, c["sliding_window"] if local else 0)
            outs.append(_attend(qs, ks, vs, seen, c["attention_scale"], c["attn_softcap"]).reshape(length, -1))
        x = x + _rms(torch.cat(outs) @ _decoded(layer["attn_output"]).T, eps, layer["post_attention_norm"])
        h = _rms(x, eps, layer["ffn_norm"])
        h = _gelu(h @ _decoded(layer["ffn_gate"]).T) * (h @ _decoded(layer["ffn_up"]).T)
        x = x + _rms(h @ _decoded(layer["ffn_down"]).T, eps, layer["post_ffw_norm"])
    starts = np.concatenate([[0], np.cumsum(lengths)[:-1]])
    places = np.concatenate([s + np.asarray(w) for s, w in zip(starts, want)])
    h = _rms(x[torch.from_numpy(places).cuda()], eps, layer["output_norm"])
    fmt, k, n, raw = head
    row, out = len(raw) // n, []
    for first in range(0, n, 32768):
        count = min(32768, n - first)
        out.append(h @ _decoded((fmt, k, count, raw[first * row:(first + count) * row])).T)
    return torch.cat(out, -1)


def _layered_logits(case, seed, tokens, want):
    config = _layered_config(case)
    w = {n: v for n, v in _layered_weights(case, config, seed)}
    eps, T = config["norm"]["eps"], len(tokens)

    def matrix(name):
        return torch.from_numpy(np.ascontiguousarray(w[name]).view(np.int16)).cuda().view(torch.bfloat16).double()

    def vector(name):
        return torch.from_numpy(w[name]).cuda().double()

    def gained(x, name):
        return _rms(x, eps, 1.0 + vector(name))

    def clamped(h, prefix, limit, scale=None):
        h = h if scale is None else h * scale[:, None]
        g = (h @ matrix(prefix + ".gate").T).clamp(max=limit)
        u = (h @ matrix(prefix + ".up").T).clamp(-limit, limit)
        return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ matrix(prefix + ".down").T
    at = torch.from_numpy(tokens.astype(np.int64)).cuda()
    seen = _causal(T)
    if case["model"] == "zasevik":
        x = matrix("embed")[at] * config["embedding"]["scale"]
        for i, layer in enumerate(config["layers"]):
            p, m, f = f"l{i}", layer["mixer"], layer["mlp"]
            h = gained(x, p + ".norm1")
            c = _rms(h @ matrix(p + ".mix.dkv").T, eps, vector(p + ".mix.dkv.norm"))
            q, k, v = (t.reshape(T, m["heads"], -1) for t in (h @ matrix(p + ".mix.q").T, c @ matrix(p + ".mix.uk").T, c @ matrix(p + ".mix.uv").T))
            y = _attend(q, k, v, seen, m["scale"], 0.0, vector(p + ".mix.sink")).reshape(T, -1) @ matrix(p + ".mix.o").T
            x = x + gained(y, p + ".norm1b") * vector(p + ".ls1")
            h = gained(x, p + ".norm2")
            if f["kind"] == "dense":
                y = (h @ matrix(p + ".mlp.up").T).clamp(min=0.0) ** 2 @ matrix(p + ".mlp.down").T
            else:
                scores, chosen = torch.sigmoid(h @ matrix(p + ".mlp.router").T).topk(f["router"]["top"], -1)
                y = torch.sigmoid(h @ matrix(p + ".mlp.shared.sg").T) * clamped(h, p + ".mlp.shared", f["shared"]["limit"])
                for e in range(f["router"]["experts"]):
                    token, slot = (chosen == e).nonzero(as_tuple=True)
                    if len(token):
                        y[token] += clamped(h[token], f"{p}.mlp.e{e}", f["expert"]["limit"], scores[token, slot])
            x = x + gained(y, p + ".norm2b") * vector(p + ".ls2")
        return gained(x[want], "final.norm") @ matrix("embed").T
    x = matrix("embed")[at]
    for i, layer in enumerate(config["layers"]):
        p, m = f"l{i}", layer["mixer"]
        if layer["type"] == "attention":
            heads, groups, dim = m["heads"], m["kv_heads"], m["dim"]
            raw = x @ matrix(p + ".mix.k").T
            q = _rms(x @ matrix(p + ".mix.q").T, eps, vector(p + ".mix.q.norm")).reshape(T, heads, dim)
            k = _rms(raw, eps, vector(p + ".mix.k.norm")).reshape(T, groups, dim)
            q, k = (_turn(t, m["rot"]["base"], m["rot"]["dims"]) for t in (q, k))
            y = _attend(q, k, raw.reshape(T, groups, dim), seen, m["scale"], m["softcap"], vector(p + ".mix.sink"))
            y = (y * torch.sigmoid(x @ matrix(p + ".mix.g").T)[:, :, None]).reshape(T, -1)
        else:
            heads, vdim, N, G, taps = m["heads"], m["vdim"], m["state"], m["groups"], m["conv"]
            inner = heads * vdim
            z, xbc, dt = (x @ matrix(p + ".mix.in").T).split([inner, inner + 2 * G * N, heads], 1)
            weight, rows = matrix(p + ".mix.conv"), torch.cat([torch.zeros(taps - 1, xbc.shape[1], dtype=xbc.dtype, device="cuda"), xbc])
            mixed = sum(rows[j:j + T] * weight[:, j] for j in range(taps)) + vector(p + ".mix.conv.b")
            xs, b, c = (mixed * torch.sigmoid(mixed)).split([inner, G * N, G * N], 1)
            xs = xs.reshape(T, heads, vdim)
            b, c = (t.reshape(T, G, N).repeat_interleave(heads // G, 1) for t in (b, c))
            dt = torch.nn.functional.softplus(dt + vector(p + ".mix.dt_bias"))
            decay = torch.exp(-torch.exp(vector(p + ".mix.A_log")) * dt)
            state, outs = torch.zeros(heads, N, vdim, dtype=torch.float64, device="cuda"), []
            for t in range(T):
                state = decay[t, :, None, None] * state + (dt[t, :, None] * b[t])[:, :, None] * xs[t][:, None, :]
                outs.append((c[t][:, None, :] @ state)[:, 0])
            y = torch.stack(outs) + vector(p + ".mix.D")[:, None] * xs
            y = y.reshape(T, inner) * z * torch.sigmoid(z)
            y = _rms(y.reshape(T, m["norm_groups"], -1), eps).reshape(T, inner) * vector(p + ".mix.norm")
        x = x + _rms(y @ matrix(p + ".mix.o").T, eps, vector(p + ".norm1"))
        if layer["mlp"]:
            y = (_gelu(x @ matrix(p + ".mlp.gate").T) * (x @ matrix(p + ".mlp.up").T)) @ matrix(p + ".mlp.down").T
            x = x + _rms(y, eps, vector(p + ".norm2"))
    return _rms(x[want], eps, vector("final.norm")) @ matrix("head").T


def _all_logits(case, seed, sequences, want):
    if case["model"] in GEMMA:
        return _gemma_logits(case, seed, sequences, want)
    return _layered_logits(case, seed, sequences[0], want[0])


def _best_of(case, logits):
    cap = syn.model_config(case["model"])["final_softcap"] if case["model"] in GEMMA else 0.0
    return (cap * torch.tanh(logits / cap) if cap else logits).topk(RETAIN, -1).values


def exact(case, seed):
    """Generation depends on the sampler's draws, not on numbers alone: no exact result for it."""
    kind = case["kind"]
    if kind == "product":
        fmt, k, n, g = FORMATS[case["format"]], case["k"], case["n"], _generator(seed)
        weight = _decoded((fmt, k, n, _blocks(fmt, n * k // syn.BLOCK_ELEMENTS[fmt], _SIGMA[fmt], g)))
        return torch.randn((case["rows"], k), generator=g, device="cuda").double() @ weight.T
    if kind == "chat":
        return None
    if kind == "prompt":
        return _all_logits(case, seed, [_tokens(case, seed, case["tokens"])], [[case["tokens"] - 1]])[0]
    if kind == "decode":
        passes = case["rows"] * case["steps"]
        logits = _all_logits(case, seed, [_tokens(case, seed, case["context"] + passes)], [list(range(case["context"], case["context"] + passes))])
        return {"best": _best_of(case, logits).reshape(case["steps"], case["rows"], RETAIN), "logits": logits[-case["rows"]:]}
    lengths, steps = _batch_lengths(case), case["steps"]
    tokens = _tokens(case, seed, sum(lengths) + steps * case["streams"])
    ends, forced = np.cumsum(lengths), tokens[sum(lengths):].reshape(steps, -1)
    sequences = [np.concatenate([tokens[e - n:e], forced[:, i]]) for i, (e, n) in enumerate(zip(ends, lengths))]
    logits = _all_logits(case, seed, sequences, [list(range(n, n + steps)) for n in lengths]).reshape(case["streams"], steps, -1)
    return {"best": _best_of(case, logits).transpose(0, 1).contiguous(), "logits": logits[:, -1].contiguous()}
