"""The cases that the engine's speed is measured on: what a program does with it, through its public entry points.

Four kinds of pass:

  prompt   requests' prompts go through `Engine.step` in portions of 2,048 tokens at most (the portion `LLM` uses), the
           last place's logits come back, the requests end
  decode   one token each for requests with a history in the cache, through a `DecodeSession` (Qwen3)
  reply    requests' prompts in one step, then `steps` decoded tokens each, tokens given (as a trace is replayed): for the
           architectures whose requests keep a recurrent state, which cannot be rolled back to be decoded from again
  sample   the draw of a token for every row of logits

Three of the seven architectures are measured: dense Qwen3 and two designs which between them run every kernel family the
others are put together from (latent attention, decayed and corrected recurrences, a selective state space, softmax attention
in 32 bits, routed experts).  Weights are random, of the layer sizes that `bench.py` names.
"""
import math
import zlib

import torch

from llmx_b200.engine import Engine, EngineOptions, StepEntry
from llmx_b200.engine.decode_loop import DecodeSession
from llmx_b200.parts.base import Precision
from llmx_b200.registry import architecture_of
from llmx_b200.sampling import RequestSampling, SamplingParams, sample

PAGE, PORTION = 16, 2048
DEVICE = "cuda:0"

QWEN3 = dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=36, hidden_size=4096,
             intermediate_size=12288, num_attention_heads=32, num_key_value_heads=8, head_dim=128, vocab_size=151936,
             rope_theta=1000000.0, rms_norm_eps=1e-6, tie_word_embeddings=False, max_position_embeddings=40960)
QWEN3_SIZES = {"8b": {}, "0.6b": dict(num_hidden_layers=28, hidden_size=1024, intermediate_size=3072, num_attention_heads=16,
                                      tie_word_embeddings=True)}
DESIGN_SIZES = {
    "w2048": dict(width=2048, heads=16, ff=6144, vocab=32768, q_rank=768, kv_rank=512, rot=64, window=2048, layers=6),
    "w4096": dict(width=4096, heads=32, ff=12288, vocab=32768, q_rank=1536, kv_rank=512, rot=64, window=4096, layers=3)}


# ---- what is measured ------------------------------------------------------------------------------------------------
def listed():
    return [
        # One user's chat with the small model: a decode step of one request, launches and latency only.
        dict(name="qwen3_0.6b_decode_b1_c300", family="qwen3", size="0.6b", kind="decode", batch=1, context=300),
        # The small model serving many: the cache's keys and values outweigh the weights.
        dict(name="qwen3_0.6b_decode_b32_c3001", family="qwen3", size="0.6b", kind="decode", batch=32, context=3001),
        # The headline: eight requests at 8,192 tokens each.
        dict(name="qwen3_8b_decode_b8_c8192", family="qwen3", size="8b", kind="decode", batch=8, context=8192),
        # Three prompts of unequal, odd lengths admitted in one step of the small model.
        dict(name="qwen3_0.6b_prompt_3x611", family="qwen3", size="0.6b", kind="prompt", batch=3, tokens=611),
        # The headline's prompt: one full portion.
        dict(name="qwen3_8b_prompt_2048", family="qwen3", size="8b", kind="prompt", batch=1, tokens=2048),
        # A full portion through latent attention and recurrences.
        dict(name="buzetar_w2048_prompt_2048", family="buzetar", size="w2048", kind="prompt", batch=1, tokens=2048),
        # A long prompt in three portions: later ones read the cache, the state and a window that has begun to move.
        dict(name="buzetar_w4096_prompt_5003", family="buzetar", size="w4096", kind="prompt", batch=1, tokens=5003),
        # Eight short questions answered together: ragged prompts, then sixteen decode steps.
        dict(name="buzetar_w2048_reply_b8", family="buzetar", size="w2048", kind="reply", batch=8, tokens=190, steps=16),
        # A full portion through experts, a state space, attention beside a corrected recurrence.
        dict(name="kisepel_w2048_prompt_2048", family="kisepel", size="w2048", kind="prompt", batch=1, tokens=2048),
        # An ordinary prompt of an odd length at the wider size.
        dict(name="kisepel_w4096_prompt_1201", family="kisepel", size="w4096", kind="prompt", batch=1, tokens=1201),
        # Four users' replies, experts read by few rows.
        dict(name="kisepel_w4096_reply_b4", family="kisepel", size="w4096", kind="reply", batch=4, tokens=150, steps=16),
        # The draw after a decode step of 32 requests with the usual settings.
        dict(name="sample_b32_v151936", family="sampler", size="151936", kind="sample", batch=32, temp=0.8, top_k=40, top_p=0.95, min_p=0.0),
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["decode", "prompt", "prompt", "prompt", "reply", "reply", "sample"])
    if kind == "sample":
        temp, top_k, top_p, min_p = rng.choice([(0.0, 0, 1.0, 0.0), (0.8, 40, 0.95, 0.0), (1.0, 1000, 1.0, 0.0), (0.7, 20, 0.8, 0.05)])
        return dict(family="sampler", size=rng.choice(["151936", "32768"]), kind=kind, batch=_log_uniform(rng, 1, 64),
                    temp=temp, top_k=top_k, top_p=top_p, min_p=min_p)
    if kind == "decode":
        size = rng.choice(["0.6b", "8b"])
        batch = _log_uniform(rng, 1, 48)
        return dict(family="qwen3", size=size, kind=kind, batch=batch, context=_log_uniform(rng, 20, 65536 // batch if batch > 4 else 16000))
    if kind == "reply":
        return dict(family=rng.choice(["buzetar", "kisepel"]), size=rng.choice(["w2048", "w4096"]), kind=kind, batch=_log_uniform(rng, 1, 12),
                    tokens=_log_uniform(rng, 5, 160), steps=rng.randint(4, 16))
    family = rng.choice(["qwen3", "buzetar", "buzetar", "kisepel", "kisepel"])
    batch = rng.choice([1, 1, 2, 3])
    size = rng.choice(["0.6b", "8b"] if family == "qwen3" else ["w2048", "w4096"])
    return dict(family=family, size=size, kind=kind, batch=batch, tokens=_log_uniform(rng, 20, (2048 if size == "8b" else 4096) // batch))


def lengths(case):
    """The requests' prompt lengths: the first has `tokens`, the others are shorter by unequal steps."""
    t = case["tokens"]
    return [max(1, t - (i * 37) % max(1, t // 2)) for i in range(case["batch"])]


# ---- configurations and their weights --------------------------------------------------------------------------------
def config_of(case):
    """config.json of the case's model."""
    if case["family"] == "qwen3":
        return dict(QWEN3, **QWEN3_SIZES[case["size"]])
    z = DESIGN_SIZES[case["size"]]
    E, H, F, L = z["width"], z["heads"], z["ff"], z["layers"]
    G = H // 4
    lightning = {"type": "lightning", "mixer": {"heads": H, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** -(3 + 5 * h / H) for h in range(H)]}}
    if case["family"] == "buzetar":
        mlp = {"kind": "dense", "ff": F, "limit": 7.0}
        kinds = [
            lightning,
            {"type": "latent_attention", "mixer": {"heads": H, "dim": 128, "rot_dim": z["rot"], "vdim": 128, "q_rank": z["q_rank"], "kv_rank": z["kv_rank"],
                                                   "scale": (128 + z["rot"]) ** -0.5, "rot": {"base": 10000.0, "dims": z["rot"]}, "mask": {"size": z["window"]}}},
            {"type": "delta", "mixer": {"heads": H, "kv_heads": H // 2, "dim": 128, "vdim": 128, "conv": 4}}]
        name = "Buzetar"
    else:
        mlp = {"kind": "moe", "router": {"experts": 16, "top": 2}, "expert": {"ff": F // 4}, "shared": {"ff": F // 2}}
        kinds = [
            {"type": "mamba2", "mixer": {"heads": H, "vdim": 128, "state": 128, "groups": G, "conv": 4, "norm_groups": G}},
            {"type": "parallel", "mixer": {
                "left": {"heads": H, "kv_heads": G, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 4 * z["window"]},
                         "rot": {"base": 1000000.0, "dims": 64, "scaling": {"factor": 4.0}}},
                "right": {"heads": H, "kv_heads": H // 2, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": E // 16, "gate_rank": E // 16}}},
            lightning]
        name = "Kisepel"
    return {"architecture": name, "vocab": z["vocab"], "width": E, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0}, "logit_scale": 1.0,
            "layers": [dict(kinds[i % 3], mlp=mlp) for i in range(L)]}


def tensors_of(cfg):
    """{name: (shape, mean, standard deviation)} of the model's tensors; one-dimensional ones are held in 32 bits.  A routing
    table has the number of experts in the place of the mean and no deviation."""
    out = {}

    def matrix(name, *shape, std=0.02):
        out[name] = (shape, 0.0, std)

    def vector(name, n, mean=1.0, std=0.01):
        out[name] = ((n,), mean, std)

    if "model_type" in cfg:
        E, F, V, D = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"], cfg["head_dim"]
        Q, KV = cfg["num_attention_heads"] * D, cfg["num_key_value_heads"] * D
        matrix("model.embed_tokens.weight", V, E)
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            vector(p + "input_layernorm.weight", E)
            vector(p + "post_attention_layernorm.weight", E)
            for n, rows, cols in (("q", Q, E), ("k", KV, E), ("v", KV, E), ("o", E, Q)):
                matrix(f"{p}self_attn.{n}_proj.weight", rows, cols)
            vector(p + "self_attn.q_norm.weight", D)
            vector(p + "self_attn.k_norm.weight", D)
            for n, rows, cols in (("gate", F, E), ("up", F, E), ("down", E, F)):
                matrix(f"{p}mlp.{n}_proj.weight", rows, cols)
        vector("model.norm.weight", E)
        if not cfg["tie_word_embeddings"]:
            matrix("lm_head.weight", V, E)
        return out
    E, V = cfg["width"], cfg["vocab"]
    around_one = cfg["architecture"] == "Buzetar"       # Kisepel's norms over the width hold what is added to one

    def norm(name):
        vector(name, E, *((1.0, 0.01) if around_one else (0.0, 0.05)))

    def delta(p, m):
        qk, v = m["kv_heads"] * m["dim"], m["heads"] * m["vdim"]
        for n, rows in (("q", qk), ("k", qk), ("v", v)):
            matrix(p + n, rows, E)
            matrix(f"{p}{n}.conv", rows, m["conv"], std=0.3)
        matrix(p + "b", m["heads"], E)
        vector(p + "A_log", m["heads"], 0.0, 0.5)
        vector(p + "norm", m["vdim"])
        matrix(p + "o", E, v)
        if "decay_rank" in m:
            matrix(p + "a1", m["decay_rank"], E)
            matrix(p + "a2", m["heads"] * m["dim"], m["decay_rank"], std=0.1)
            vector(p + "dt_bias", m["heads"] * m["dim"], 0.0, 0.5)
            matrix(p + "g1", m["gate_rank"], E)
            matrix(p + "g2", v, m["gate_rank"], std=0.1)
        else:
            matrix(p + "a", m["heads"], E)
            vector(p + "dt_bias", m["heads"], 0.0, 0.5)
            matrix(p + "g", v, E)

    matrix("embed", V, E)
    for i, layer in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}.mix.", layer["mixer"], layer["mlp"]
        norm(f"l{i}.norm1")
        if layer["type"] == "lightning":
            for n in "qkvg":
                matrix(p + n, m["heads"] * 128, E)
            vector(p + "norm", m["heads"] * 128)
            matrix(p + "o", E, m["heads"] * 128)
        elif layer["type"] == "latent_attention":
            H, D, R, C, A = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"], m["q_rank"]
            matrix(p + "dq", A, E)
            vector(p + "dq.norm", A)
            matrix(p + "uq", H * (D + R), A)
            matrix(p + "dkv", C + R, E)
            vector(p + "dkv.norm", C)
            matrix(p + "uk", H * D, C)
            matrix(p + "uv", H * m["vdim"], C)
            matrix(p + "o", E, H * m["vdim"])
        elif layer["type"] == "delta":
            delta(p, m)
        elif layer["type"] == "mamba2":
            inner, conv = m["heads"] * m["vdim"], m["heads"] * m["vdim"] + 2 * m["groups"] * m["state"]
            matrix(p + "in", inner + conv + m["heads"], E)
            matrix(p + "conv", conv, m["conv"], std=0.3)
            vector(p + "conv.b", conv, 0.0, 0.1)
            vector(p + "dt_bias", m["heads"], 0.0, 0.5)
            vector(p + "A_log", m["heads"], 0.0, 0.5)
            vector(p + "D", m["heads"], 1.0, 0.1)
            vector(p + "norm", inner)
            matrix(p + "o", E, inner)
        else:
            left = m["left"]
            for n, heads in (("q", left["heads"]), ("k", left["kv_heads"]), ("v", left["kv_heads"])):
                matrix(f"{p}left.{n}", heads * 128, E)
            vector(p + "left.q.norm", 128)
            vector(p + "left.k.norm", 128)
            matrix(p + "left.o", E, left["heads"] * 128)
            vector(p + "left.out", E)
            delta(p + "right.", m["right"])
            vector(p + "right.out", E)
        p = f"l{i}.mlp."
        if mlp["kind"] == "dense":
            units = [(p, mlp["ff"])]
        else:
            n = mlp["router"]["experts"]
            out[p + "table"] = ((V, mlp["router"]["top"]), n, 0.0)
            units = [(f"{p}e{j}.", mlp["expert"]["ff"]) for j in range(n)] + [(p + "shared.", mlp["shared"]["ff"])]
        for unit, ff in units:
            matrix(unit + "gate", ff, E)
            matrix(unit + "up", ff, E)
            matrix(unit + "down", E, ff)
    norm("final.norm")
    if cfg["architecture"] == "Buzetar":
        matrix("head", V, E)
    return out


def _generator(seed, name):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed) * 1000003 + zlib.crc32(name.encode()))
    return g


class Weights:
    """A source of the model's tensors (as a folder of files would be), each made on the device from the seed and its name."""

    def __init__(self, cfg, seed):
        self.specs, self.seed = tensors_of(cfg), seed

    def names(self):
        return list(self.specs)

    def shape(self, name):
        return self.specs[name][0]

    def dtype(self, name):
        shape, _, std = self.specs[name]
        return torch.int32 if std == 0.0 else torch.float32 if len(shape) == 1 else torch.bfloat16

    def tensor(self, name):
        shape, mean, std = self.specs[name]
        g = _generator(self.seed, name)
        if std == 0.0:          # a routing table: distinct experts a token
            return torch.rand((shape[0], int(mean)), device=DEVICE, generator=g).argsort(1)[:, :shape[1]].to(torch.int32).contiguous()
        return torch.empty(shape, dtype=self.dtype(name), device=DEVICE).normal_(mean, std, generator=g)


def token_ids(vocab, seed, name, count):
    return torch.randint(0, vocab, (count,), device=DEVICE, generator=_generator(seed, name)).tolist()


def history(cfg, case, seed, layer):
    """Cached keys and values of one layer, [2, requests, context, kv heads, head width]: keys normed and turned already."""
    shape = (2, case["batch"], case["context"], cfg["num_key_value_heads"], cfg["head_dim"])
    return torch.empty(shape, dtype=torch.bfloat16, device=DEVICE).normal_(0.0, 1.0, generator=_generator(seed, f"history {layer}"))


# ---- the passes ------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    state = {"case": case}
    if case["kind"] == "sample":
        logits = torch.empty((case["batch"], int(case["size"])), device=DEVICE).normal_(0.0, 3.0, generator=_generator(seed, "logits"))
        params = [SamplingParams(temp=case["temp"], top_k=case["top_k"], top_p=case["top_p"], min_p=case["min_p"], seed=seed * 1009 + r + 1)
                  for r in range(case["batch"])]
        return dict(state, logits=logits, params=params)
    cfg = config_of(case)
    vocab = cfg["vocab_size"] if case["family"] == "qwen3" else cfg["vocab"]
    entry = architecture_of(cfg)
    model = entry.build(entry.config_cls.from_dict(cfg))
    model.load(Weights(cfg, seed), torch.device(DEVICE), Precision.of("bfloat16"))
    longest = case["context"] + 1 if case["kind"] == "decode" else case["tokens"] + case.get("steps", 0)
    pages = -(-longest // PAGE) + 1
    engine = Engine(model, EngineOptions(dtype="bfloat16", kv_tokens=case["batch"] * pages * PAGE, page_size=PAGE, max_requests=case["batch"]))
    state.update(engine=engine, requests=[f"request {r}" for r in range(case["batch"])])
    if case["kind"] == "decode":
        held = []
        for rid in state["requests"]:
            cache = engine.cache.new_request(rid)
            cache.prepare(case["context"])
            cache.commit()
            held.append(torch.tensor(cache.tables[0].pages, device=DEVICE))
        for layer in range(cfg["num_hidden_layers"]):
            kv = history(cfg, case, seed, layer)
            kv = torch.nn.functional.pad(kv, (0, 0, 0, 0, 0, len(held[0]) * PAGE - case["context"]))
            for r, at in enumerate(held):       # storage: [layer, page, keys or values, kv head, place, head width]
                engine.cache.groups[0].storage[layer][at] = kv[:, r].unflatten(1, (len(at), PAGE)).permute(1, 0, 3, 2, 4)
        state.update(tokens=token_ids(vocab, seed, "tokens", case["batch"]), session=DecodeSession(engine, state["requests"]))
    else:
        state["prompts"] = [token_ids(vocab, seed, f"prompt {r}", n) for r, n in enumerate(lengths(case))]
        state["replies"] = [token_ids(vocab, seed, f"reply {s}", case["batch"]) for s in range(case.get("steps", 0))]
    return state


def _prompts(engine, state):
    """Every request's prompt, portions of at most PORTION tokens filled in the requests' order; {request: logits row}."""
    todo = [(rid, prompt, 0) for rid, prompt in zip(state["requests"], state["prompts"])]
    rows = []
    while todo:
        room, entries = PORTION, []
        while todo and room:
            rid, prompt, at = todo.pop(0)
            n = min(room, len(prompt) - at)
            last = at + n == len(prompt)
            entries.append(StepEntry(rid, prompt[at:at + n], [n - 1] if last else []))
            room -= n
            if not last:
                todo.insert(0, (rid, prompt, at + n))
                break
        logits = engine.step(entries, record=True)
        if logits is not None:
            rows.append(logits)
    return rows


def run(state):
    case = state["case"]
    if case["kind"] == "sample":
        return torch.tensor(sample(state["logits"], [RequestSampling(p) for p in state["params"]]))
    engine = state["engine"]
    if case["kind"] == "decode":
        logits = state["session"].step(state["tokens"])
        for rid in state["requests"]:
            engine.truncate(rid, case["context"])
        return [logits]
    rows = _prompts(engine, state)
    if case["kind"] == "reply":
        session = DecodeSession(engine, state["requests"], plain_steps=4)
        for tokens in state["replies"]:
            rows.append(session.step(tokens).clone())       # the step's logits are overwritten by the next step's
        session.close()
    for rid in state["requests"]:
        engine.end(rid)
    return rows


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def work(case):
    if case["kind"] == "sample":
        return {"bytes": case["batch"] * int(case["size"]) * 4, "flops": 0}
    cfg = config_of(case)
    specs = tensors_of(cfg)
    matrices = {n: s[0] for n, s in specs.items() if len(s[0]) == 2 and s[2] and not n.endswith(".conv")}
    table, head = (matrices["model.embed_tokens.weight"], "model.embed_tokens.weight") if case["family"] == "qwen3" else (matrices["embed"], "embed")
    for other in ("lm_head.weight", "head"):
        head = other if other in matrices else head
    top = 2 / 16 if case["family"] == "kisepel" else 1.0
    weights = {n: r * c for n, (r, c) in matrices.items() if n not in ("model.embed_tokens.weight", "embed", head)}

    def step(rows, wanted):
        """(bytes, flops) of the products of a step of `rows` rows."""
        bytes_, flops = 2.0 * (math.prod(matrices[head]) if wanted else 0) + 2.0 * rows * table[1], 2.0 * math.prod(matrices[head]) * wanted
        for n, count in weights.items():
            routed = ".mlp.e" in n
            bytes_ += 2.0 * count * (1.0 - (1.0 - top) ** rows if routed else 1.0)
            flops += 2.0 * count * rows * (top if routed else 1.0)
        return bytes_, flops

    def mixing(before, rows):
        """(bytes, flops) of the mixers for `rows` rows of one request after `before` tokens."""
        if case["family"] == "qwen3":
            L, H, G, D = cfg["num_hidden_layers"], cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
            return L * 4.0 * G * D * (before + rows), L * 4.0 * H * D * (rows * before + rows * (rows + 1) / 2)
        bytes_ = flops = 0.0
        for layer in cfg["layers"]:
            m = layer["mixer"]
            if layer["type"] == "latent_attention":
                seen = sum(min(before + i + 1, m["mask"]["size"]) for i in range(rows))
                bytes_ += 2.0 * (m["kv_rank"] + m["rot_dim"]) * min(before + rows, m["mask"]["size"] + rows)
                flops += 2.0 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]) * seen
                continue
            sides = [m]
            if layer["type"] == "parallel":
                left, sides = m["left"], [m["right"]]
                bytes_ += 4.0 * left["kv_heads"] * 128 * (before + rows)
                flops += 4.0 * left["heads"] * 128 * (rows * before + rows * (rows + 1) / 2)
            for s in sides:
                cells = s["heads"] * s.get("dim", s.get("state")) * s["vdim"]
                bytes_ += 8.0 * cells
                flops += (6.0 if "conv" in s and "kv_heads" in s else 4.0) * cells * rows
        return bytes_, flops

    total = [0.0, 0.0]

    def add(pair):
        total[0] += pair[0]
        total[1] += pair[1]

    batch = case["batch"]
    if case["kind"] == "decode":
        add(step(batch, batch))
        for _ in range(batch):
            add(mixing(case["context"], 1))
    else:
        rows = sum(lengths(case))
        portions = -(-rows // PORTION)
        for p in range(portions):
            add(step(min(PORTION, rows - p * PORTION), batch if p == portions - 1 else 0))
        for n in lengths(case):
            add(mixing(0, n))
        for s in range(case.get("steps", 0)):
            add(step(batch, batch))
            for n in lengths(case):
                add(mixing(n + s, 1))
    return {"bytes": total[0], "flops": total[1]}


def tolerance(case):
    """bfloat16 products in another order, four times what two runs of the same pass were seen to differ by: sums of pieces
    meet by atomics, and a rounding that falls the other way travels through 28 or 36 layers (0.007 to 0.014 of the logits) or
    3 to 6 (0.001 to 0.0045)."""
    if case["kind"] == "sample":
        return "exact"
    return {"rel": 0.03, "max": 0.3} if case["family"] == "qwen3" else {"rel": 0.018, "max": 0.1}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------
D64 = torch.float64


class Exact64:
    """A model's formulas over whole sequences in float64 (plain torch on the same weights)."""

    def __init__(self, cfg, seed):
        self.cfg, self.weights = cfg, Weights(cfg, seed)

    def w(self, name):
        t = self.weights.tensor(name)
        return t if t.dtype == torch.int32 else t.to(D64)

    def lin(self, h, name):
        return h @ self.w(name).T

    def embed(self, name, ids):
        return self.weights.tensor(name)[torch.tensor(ids, device=DEVICE)].to(D64)


def rms(x, w, eps):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def turn(x, positions, base, dims, factor=1.0, neighbours=False):
    """Rotation of the first `dims` values of the last axis, x [tokens, heads, width]: value i with value i + dims / 2, or
    neighbouring values."""
    i = torch.arange(dims // 2, dtype=D64, device=x.device)
    angle = positions.to(D64)[:, None] * (base ** (-2.0 * i / dims) / factor)[None]
    c, s = angle.cos()[:, None], angle.sin()[:, None]
    first, second = (x[..., 0:dims:2], x[..., 1:dims:2]) if neighbours else (x[..., :dims // 2], x[..., dims // 2:dims])
    a, b = first * c - second * s, second * c + first * s
    turned = torch.stack([a, b], -1).flatten(-2) if neighbours else torch.cat([a, b], -1)
    return torch.cat([turned, x[..., dims:]], -1)


def attend(q, k, v, scale, window=None):
    """q [T, H, D] over k [S, G, D], v [S, G, V], the queries being the last T of the S places."""
    T, S, H, G = q.shape[0], k.shape[0], q.shape[1], k.shape[1]
    i, j = torch.arange(S - T, S, device=q.device)[:, None], torch.arange(S, device=q.device)[None]
    hidden = (j > i) if window is None else (j > i) | (i - j >= window)
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T * scale).masked_fill_(hidden, -math.inf)
        out.append(torch.softmax(s, -1) @ v[:, h * G // H])
    return torch.stack(out, 1)


def recur(q, k, v, decay, beta=None):
    """Per head S <- decay S + k v^T (v replaced by beta (v - S^T k) where there is a beta), o = S^T q.  q, k, decay [T, H, D]
    (a decay of width 1 is one for all channels), v [T, H, V], beta [T, H, 1]."""
    S = torch.zeros(q.shape[1], q.shape[2], v.shape[2], dtype=D64, device=q.device)
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = S * decay[t, :, :, None]
        u = v[t] if beta is None else beta[t] * (v[t] - torch.bmm(k[t, :, None], S)[:, 0])
        S = torch.baddbmm(S, k[t, :, :, None], u[:, None])
        out[t] = torch.bmm(q[t, :, None], S)[:, 0]
    return out


def short_filter(x, taps, bias=None):
    n = taps.shape[1]
    padded = torch.cat([torch.zeros(n - 1, x.shape[1], dtype=D64, device=x.device), x])
    y = sum(padded[j:j + x.shape[0]] * taps[:, j] for j in range(n))
    return y if bias is None else y + bias


silu = torch.nn.functional.silu
softplus = torch.nn.functional.softplus


class ExactDesign(Exact64):
    def lightning(self, h, p, m, eps):
        T, H = h.shape[0], m["heads"]
        q, k, v = (silu(self.lin(h, p + n)).view(T, H, 128) for n in "qkv")
        decay = torch.tensor(m["decay"], dtype=D64, device=DEVICE).view(1, H, 1).expand(T, H, 1)
        o = recur(q, k, v, decay).view(T, H * 128)
        return self.lin(rms(o, self.w(p + "norm"), eps) * torch.sigmoid(self.lin(h, p + "g")), p + "o")

    def latent_attention(self, h, p, m, eps):
        T, H, D, C = h.shape[0], m["heads"], m["dim"], m["kv_rank"]
        at, rot = torch.arange(T, device=DEVICE), m["rot"]
        q = self.lin(rms(self.lin(h, p + "dq"), self.w(p + "dq.norm"), eps), p + "uq").view(T, H, -1)
        kv = self.lin(h, p + "dkv")
        c = rms(kv[:, :C], self.w(p + "dkv.norm"), eps)
        k_rot = turn(kv[:, None, C:], at, rot["base"], rot["dims"], neighbours=True).expand(T, H, -1)
        q = torch.cat([q[..., :D], turn(q[..., D:], at, rot["base"], rot["dims"], neighbours=True)], -1)
        k = torch.cat([self.lin(c, p + "uk").view(T, H, D), k_rot], -1)
        o = attend(q, k, self.lin(c, p + "uv").view(T, H, -1), m["scale"], m["mask"]["size"])
        return self.lin(o.reshape(T, -1), p + "o")

    def delta(self, h, p, m, eps):
        T, H, G, D = h.shape[0], m["heads"], m["kv_heads"], m["dim"]
        q, k, v = (silu(short_filter(self.lin(h, p + n), self.w(f"{p}{n}.conv"))) for n in "qkv")
        q, k = (x.view(T, G, D).repeat_interleave(H // G, 1) for x in (q, k))
        q, k = (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
        step = self.lin(self.lin(h, p + "a1"), p + "a2") if "decay_rank" in m else self.lin(h, p + "a")
        step = softplus(step + self.w(p + "dt_bias")).view(T, H, -1)
        decay = torch.exp(-torch.exp(self.w(p + "A_log"))[None, :, None] * step)
        o = recur(q * D ** -0.5, k, v.view(T, H, -1), decay, torch.sigmoid(self.lin(h, p + "b"))[:, :, None])
        o = rms(o, self.w(p + "norm"), eps).reshape(T, -1)
        gate = torch.sigmoid(self.lin(self.lin(h, p + "g1"), p + "g2")) if "gate_rank" in m else silu(self.lin(h, p + "g"))
        return self.lin(o * gate, p + "o")

    def mamba2(self, h, p, m, eps):
        T, H, V, N, G = h.shape[0], m["heads"], m["vdim"], m["state"], m["groups"]
        inner = H * V
        z, xbc, dt = self.lin(h, p + "in").split([inner, inner + 2 * G * N, H], 1)
        xbc = silu(short_filter(xbc, self.w(p + "conv"), self.w(p + "conv.b")))
        x = xbc[:, :inner].reshape(T, H, V)
        b, c = (t.reshape(T, G, N).repeat_interleave(H // G, 1) for t in xbc[:, inner:].split(G * N, 1))
        dt = softplus(dt + self.w(p + "dt_bias"))[:, :, None]
        y = recur(c, b * dt, x, torch.exp(-torch.exp(self.w(p + "A_log"))[None, :, None] * dt)) + self.w(p + "D")[None, :, None] * x
        y = y.reshape(T, inner) * silu(z)
        y = rms(y.view(T, m["norm_groups"], -1), None, eps).reshape(T, inner) * self.w(p + "norm")
        return self.lin(y, p + "o")

    def parallel(self, h, p, m, eps):
        left, T = m["left"], h.shape[0]
        at, rot = torch.arange(T, device=DEVICE), left["rot"]
        q, k, v = (self.lin(h, f"{p}left.{n}").view(T, -1, 128) for n in "qkv")
        q, k = (turn(rms(x, self.w(f"{p}left.{n}.norm"), eps), at, rot["base"], rot["dims"], rot["scaling"]["factor"]) for x, n in ((q, "q"), (k, "k")))
        size = left["mask"]["size"]
        o = torch.cat([attend(q[s:s + size], k[s:s + size], v[s:s + size], left["scale"]) for s in range(0, T, size)])
        o = self.lin(o.reshape(T, -1), p + "left.o")
        right = self.delta(h, p + "right.", m["right"], eps)
        return 0.5 * (rms(o, self.w(p + "left.out"), eps) + rms(right, self.w(p + "right.out"), eps))

    def unit(self, h, p, limit=None):
        gate, up = self.lin(h, p + "gate"), self.lin(h, p + "up")
        if limit is None:
            return self.lin(silu(gate) * up, p + "down")
        gate, up = gate.clamp(max=limit), up.clamp(-limit, limit)
        return self.lin(gate * torch.sigmoid(1.702 * gate) * (up + 1.0), p + "down")

    def experts(self, h, ids, p, mlp):
        out = self.unit(h, p + "shared.")
        chosen = self.w(p + "table")[torch.tensor(ids, device=DEVICE)]
        for e in range(mlp["router"]["experts"]):
            rows = (chosen == e).any(1).nonzero()[:, 0]
            if len(rows):
                out[rows] += self.unit(h[rows], f"{p}e{e}.") / mlp["router"]["top"]
        return out

    def sequences(self, sequences, wanted):
        """Logits at the `wanted` places of every sequence.  Row-wise parts run all sequences' rows together, mixers one by one."""
        cfg, eps = self.cfg, self.cfg["norm"]["eps"]
        ids = [t for s in sequences for t in s]
        cuts = [len(s) for s in sequences]
        buzetar = cfg["architecture"] == "Buzetar"

        def norm(x, name):
            return rms(x - x.mean(-1, keepdim=True), self.w(name), eps) if buzetar else rms(x, 1.0 + self.w(name), eps)

        x = self.embed("embed", ids)
        for i, layer in enumerate(cfg["layers"]):
            h = norm(x, f"l{i}.norm1")
            mixer = getattr(self, layer["type"])
            y = torch.cat([mixer(part, f"l{i}.mix.", layer["mixer"], eps) for part in h.split(cuts)])
            mlp = layer["mlp"]
            y = y + (self.unit(h, f"l{i}.mlp.", mlp["limit"]) if buzetar else self.experts(h, ids, f"l{i}.mlp.", mlp))
            x = x + y
        rows = torch.cat([part[torch.tensor(want, device=DEVICE)] for part, want in zip(x.split(cuts), wanted)])
        return self.lin(norm(rows, "final.norm"), "head" if buzetar else "embed")


class ExactQwen3(Exact64):
    def sequences(self, sequences, past=None):
        """Logits of every sequence's last place; `past(layer)` gives [2, requests, context, kv heads, width] seen before."""
        cfg, eps = self.cfg, self.cfg["rms_norm_eps"]
        D, base = cfg["head_dim"], cfg["rope_theta"]
        cuts = [len(s) for s in sequences]
        x = self.embed("model.embed_tokens.weight", [t for s in sequences for t in s])
        for i in range(cfg["num_hidden_layers"]):
            p, T = f"model.layers.{i}.", x.shape[0]
            h = rms(x, self.w(p + "input_layernorm.weight"), eps)
            q, k, v = (self.lin(h, f"{p}self_attn.{n}_proj.weight").view(T, -1, D) for n in "qkv")
            q, k = rms(q, self.w(p + "self_attn.q_norm.weight"), eps), rms(k, self.w(p + "self_attn.k_norm.weight"), eps)
            kept = past(i) if past is not None else None
            before = kept.shape[2] if kept is not None else 0
            out = []
            for r, (qr, kr, vr) in enumerate(zip(q.split(cuts), k.split(cuts), v.split(cuts))):
                at = torch.arange(before, before + len(qr), device=DEVICE)
                qr, kr = turn(qr, at, base, D), turn(kr, at, base, D)
                if kept is not None:
                    kr, vr = torch.cat([kept[0, r].to(D64), kr]), torch.cat([kept[1, r].to(D64), vr])
                out.append(attend(qr, kr, vr, D ** -0.5))
            x = x + self.lin(torch.cat(out).reshape(T, -1), p + "self_attn.o_proj.weight")
            h = rms(x, self.w(p + "post_attention_layernorm.weight"), eps)
            x = x + self.lin(silu(self.lin(h, p + "mlp.gate_proj.weight")) * self.lin(h, p + "mlp.up_proj.weight"), p + "mlp.down_proj.weight")
        last = torch.tensor(cuts, device=DEVICE).cumsum(0) - 1
        x = rms(x[last], self.w("model.norm.weight"), eps)
        return self.lin(x, "model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight")


def _rows_by_step(case):
    """How many requests' logits each of a prompt pass's steps returns (a step without any returns nothing)."""
    counts, used, here = [], 0, 0
    for n in lengths(case):
        while used + n > PORTION:           # the step is full: the rest of this prompt is the next step's
            n -= PORTION - used
            counts.append(here)
            used = here = 0
        used, here = used + n, here + 1
        if used == PORTION:
            counts.append(here)
            used = here = 0
    return [c for c in counts + [here] if c]


@torch.no_grad()
def exact(case, seed):
    if case["kind"] == "sample":
        return None                         # token ids
    cfg = config_of(case)
    vocab = cfg["vocab_size"] if case["family"] == "qwen3" else cfg["vocab"]
    if case["kind"] == "decode":
        tokens = token_ids(vocab, seed, "tokens", case["batch"])
        return [ExactQwen3(cfg, seed).sequences([[t] for t in tokens], lambda layer: history(cfg, case, seed, layer))]
    prompts = [token_ids(vocab, seed, f"prompt {r}", n) for r, n in enumerate(lengths(case))]
    if case["family"] == "qwen3":
        last = ExactQwen3(cfg, seed).sequences(prompts)
        return list(last.split(_rows_by_step(case)))
    steps = case.get("steps", 0)
    replies = [token_ids(vocab, seed, f"reply {s}", case["batch"]) for s in range(steps)]
    whole = [prompt + [reply[r] for reply in replies] for r, prompt in enumerate(prompts)]
    wanted = [[len(prompt) - 1 + s for s in range(steps + 1)] for prompt in prompts]
    logits = ExactDesign(cfg, seed).sequences(whole, wanted).view(case["batch"], steps + 1, -1)
    return list(logits[:, 0].split(_rows_by_step(case))) + [logits[:, 1 + s].contiguous() for s in range(steps)]
