"""Timed workloads of the framework: what a serving program has it do, called the way such a program calls it.

Every case names a model shape of `tilemega_b200.synthetic` (cut to a few layers: every layer of a kind runs the same
kernels) and one pass over it:

  llama     one decoded token of `batch` sequences at `context` positions through a decode plan, logits read by the host
            (a server that samples on the CPU)
  encoder   one forward pass of `batch` sequences of 128 tokens through a forward plan
  ragged    one step of a ragged plan: `decode` sequences at about `context` positions take one token each, and a portion
            of `rows` prompt tokens behind `history` positions already run joins them; logits of every decoded token and
            of `wanted` places of the portion

Weights are N(0, 0.02) draws (an embedding of unit size for ragged plans), token ids uniform; where there are experts, a token's
embedding leans towards some of them, as it does in trained models, so that few choices are close calls. A step is run again from the
same lengths, the way speculative decoding takes steps back; recurrent states move on from pass to pass.
"""
from __future__ import annotations

import math
import zlib

import torch
import torch.nn.functional as F

from tilemega_b200 import synthetic
from tilemega_b200.planbuild import emit_plan

SHAPES = {
    "llama-8b": (synthetic.LLAMA_3_1_8B, 8), "llama-1b": (synthetic.LLAMA_3_2_1B, 8), "bert-base": (synthetic.BERT_BASE, 12),
    "nadilorn-8b": (synthetic.NADILORN_8B, (0, 2)), "nadilorn-1b": (synthetic.NADILORN_1B, (0, 4)),
    "nadilorn-7b-a1b": (synthetic.NADILORN_7B_A1B, (1, 5)), "nadilorn-30b-a3b": (synthetic.NADILORN_30B_A3B, (1, 3)),
    "benarax-7b-a1b": (synthetic.BENARAX_7B_A1B, (0, 6)), "benarax-30b-a3b": (synthetic.BENARAX_30B_A3B, (0, 3)),
}
RAGGED = {"decode": 0, "context": 0, "rows": 0, "history": 0, "wanted": 0}


def ragged(shape: str, **sizes) -> dict:
    return {"kind": "ragged", "shape": shape} | RAGGED | sizes


def listed() -> list[dict]:
    return [
        # one user's answer being written, the benchmark's headline shape and context; mostly weights streamed from memory
        {"name": "llama decode 1", "kind": "llama", "shape": "llama-8b", "batch": 1, "context": 2646},
        # one query embedded while its user waits: the smallest call, nothing but latency
        {"name": "encode 1", "kind": "encoder", "shape": "bert-base", "batch": 1},
        # documents embedded in bulk
        {"name": "encode 32", "kind": "encoder", "shape": "bert-base", "batch": 32},
        # an ordinary prompt, all in one step
        {"name": "prompt 2048"} | ragged("nadilorn-8b", rows=2048, wanted=16),
        # a chat prompt of no round size on a small model
        {"name": "prompt 431 small"} | ragged("nadilorn-1b", rows=431, wanted=5),
        # continuous batching: running answers and the middle of a long prompt in the same step
        {"name": "mixed 24 + 999"} | ragged("nadilorn-8b", decode=24, context=1500, rows=999, history=2500, wanted=1),
        # one user's answer from a mixture of experts
        {"name": "experts decode 1"} | ragged("nadilorn-7b-a1b", decode=1, context=2646),
        # a full batch on the same model
        {"name": "experts decode 64"} | ragged("nadilorn-7b-a1b", decode=64, context=1100),
        # a prompt through a larger mixture of experts
        {"name": "experts prompt 2048"} | ragged("nadilorn-30b-a3b", rows=2048, wanted=16),
        # a few users at a time on latent attention, delta rule and short convolutions
        {"name": "latent decode 8"} | ragged("benarax-7b-a1b", decode=8, context=2646),
        # the third portion of a long document on the same kind of model, the largest step here
        {"name": "latent prompt 2048 at 4096"} | ragged("benarax-30b-a3b", rows=2048, history=4096, wanted=16),
    ]


def draw(rng) -> dict:
    def size(low: int, high: int) -> int:
        return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))

    kind = rng.choice(("llama", "encoder", "prompt", "prompt", "mixed", "decode", "decode"))
    if kind == "llama":
        return {"kind": "llama", "shape": rng.choice(("llama-8b", "llama-1b")), "batch": rng.choice((1, 1, 2, 4, 8)), "context": size(16, 6000)}
    if kind == "encoder":
        return {"kind": "encoder", "shape": "bert-base", "batch": size(1, 32)}
    if kind == "prompt":
        shape = rng.choice(("nadilorn-8b", "nadilorn-1b", "nadilorn-7b-a1b", "benarax-7b-a1b", "benarax-30b-a3b"))
        return ragged(shape, rows=size(17, 2048), history=rng.choice((0, 0, size(1, 4000))), wanted=rng.randint(1, 16))
    if kind == "mixed":
        shape = rng.choice(("nadilorn-8b", "nadilorn-1b", "nadilorn-7b-a1b", "benarax-7b-a1b"))
        return ragged(shape, decode=size(1, 48), context=size(16, 2500), rows=size(17, 1800), history=size(1, 2500), wanted=1)
    shape = rng.choice(("nadilorn-8b", "nadilorn-1b", "nadilorn-7b-a1b", "benarax-7b-a1b"))
    batch = size(1, 64)
    return ragged(shape, decode=batch, context=size(16, 6000 if batch <= 8 else 2000))


# -- the models ------------------------------------------------------------------------------------------------------------
def config_of(case: dict) -> dict:
    config, cut = SHAPES[case["shape"]]
    config = dict(config)
    if case["kind"] == "ragged":
        config["layers"] = config["layers"][cut[0]:cut[1]]
    else:
        config["num_hidden_layers"] = cut
    return config


def shapes_of(case: dict) -> dict[str, tuple[int, ...]]:
    if case["kind"] == "ragged":
        from tilemega_b200.registry import tensor_shapes
        return tensor_shapes(config_of(case))
    if case["kind"] == "encoder":
        return dict(synthetic.encoder_parameter_shapes(config_of(case)))
    return dict(synthetic.parameter_shapes(config_of(case)))


class Drawn:
    """A checkpoint whose tensors are drawn on the device when asked for, each from a generator of its own."""

    def __init__(self, case: dict, seed: int, dtype: torch.dtype):
        self.shapes, self.seed, self.dtype = shapes_of(case), seed, dtype
        mixtures = [layer["mlp"] for layer in config_of(case).get("layers", ()) if layer["mlp"]["kind"] == "moe"]
        self.top = mixtures[0]["router"]["top"] if mixtures else 0

    def tensor(self, name: str) -> torch.Tensor:
        if name == "lm_head.weight" and name not in self.shapes:
            name = "model.embed_tokens.weight"
        shape, last = self.shapes[name], name.rsplit(".", 1)[-1]
        label = "router" if last == "router" else name
        generator = torch.Generator(device="cuda").manual_seed((self.seed << 32) ^ zlib.crc32(label.encode()))
        value = torch.empty(shape, device="cuda").normal_(0.0, 0.02, generator=generator)
        if name == "embed":
            value *= 50.0
            routers = [other for other in self.shapes if other.endswith("mlp.router")]
            if routers:
                direction = F.normalize(self.tensor(routers[0]).float(), dim=-1)
                likes = torch.rand((shape[0], len(direction)), device="cuda", generator=generator).topk(self.top, dim=-1).indices
                value += torch.zeros((shape[0], len(direction)), device="cuda").scatter_(1, likes, 14.0) @ direction
        elif name.endswith("canon1"):
            value *= 15.0
        elif last.startswith("norm") or "norm" in name.lower() and name.endswith(".weight"):
            value += 1.0
        return value.to(self.dtype)


def tokens_of(case: dict, seed: int, count: int, vocab: int) -> list[int]:
    generator = torch.Generator().manual_seed(seed * 7919 + count)
    return torch.randint(0, vocab, (count,), generator=generator).tolist()


def sequences_of(case: dict, seed: int) -> tuple[list[list[int]], list[int], list[int]]:
    """Of a ragged case: tokens of every sequence, how many of them have run before the step, and the wanted places."""
    vocab, sequences, done = config_of(case)["vocab"], [], []
    for index in range(case["decode"]):
        length = max(1, case["context"] - (37 * index) % max(1, case["context"] // 4))
        sequences.append(tokens_of(case, seed + index, length + 1, vocab))
        done.append(length)
    wanted = []
    if case["rows"]:
        sequences.append(tokens_of(case, seed + 1000, case["history"] + case["rows"], vocab))
        done.append(case["history"])
        wanted = sorted({case["rows"] - 1 - index * case["rows"] // case["wanted"] for index in range(case["wanted"])})
    return sequences, done, wanted


class Program:
    """What a program holds: something to close when it lets go of it."""

    def __init__(self, **held):
        self.__dict__.update(held)

    def __del__(self):
        self.engine.close()


def prepare(case: dict, seed: int) -> Program:
    return {"llama": prepare_llama, "encoder": prepare_encoder, "ragged": prepare_ragged}[case["kind"]](case, seed)


def prepare_llama(case: dict, seed: int) -> Program:
    from tilemega_b200.serving.plan import PlanLibrary
    from tilemega_b200.serving.state import allocate_state
    from tilemega_b200.serving.weights import load_weights
    config, batch, context = config_of(case), case["batch"], case["context"]
    capacity = (context + 32) // 16 * 16
    blocks = capacity // 16
    library = PlanLibrary(emit_plan(config, batch_lo=batch, batch_hi=batch, capacity=capacity, kv_layout="paged", num_blocks=batch * blocks + 1))
    weights = load_weights(Drawn(case, seed, torch.bfloat16), library, device="cuda")
    state = allocate_state(config, batch, library, "cuda", context_base=torch.full((batch,), context, dtype=torch.int32))
    state.kv_storage.normal_(0.0, 0.5, generator=torch.Generator(device="cuda").manual_seed(seed))
    state.tokens[:, context] = torch.tensor(tokens_of(case, seed, batch, config["vocab_size"]), dtype=torch.int32)
    engine = library.create(batch, {name: tensor.data_ptr() for name, tensor in weights.items()} | state.pointers, 0)
    engine.set_prompt_len(0)
    engine.set_steps([0])
    logits = torch.empty((batch, config["vocab_size"]))
    return Program(kind="llama", engine=engine, weights=weights, state=state, logits=logits, stream=torch.cuda.current_stream().cuda_stream)


def prepare_encoder(case: dict, seed: int) -> Program:
    from tilemega_b200.serving.encoder import EncoderEngine
    library = emit_plan(config_of(case), phase="forward", batch_lo=case["batch"], dtype="f16")
    engine = EncoderEngine(Drawn(case, seed, torch.float16), library, case["batch"])
    ids, types = encoder_inputs(case, seed)
    return Program(kind="encoder", engine=engine, ids=ids, types=types)


def encoder_inputs(case: dict, seed: int) -> tuple[torch.Tensor, torch.Tensor]:
    ids, types = synthetic.encoder_inputs(config_of(case), case["batch"], seed=seed)
    return ids.cuda(), types.cuda()


def prepare_ragged(case: dict, seed: int) -> Program:
    from tilemega_b200.serving.ragged import Portion, RaggedExecutor
    sequences, done, wanted = sequences_of(case, seed)
    capacity = (max(len(tokens) for tokens in sequences) + 31) // 16 * 16
    blocks = sum((len(tokens) + 31) // 16 for tokens in sequences)
    library = emit_plan(config_of(case), phase="ragged", slots=len(sequences), capacity=capacity, num_blocks=blocks + 2, max_rows=2048, max_wanted=64)
    engine = RaggedExecutor(Drawn(case, seed, torch.bfloat16), library)
    slots = [engine.open() for _ in sequences]
    engine.run([Portion(slot, tokens[:count]) for slot, tokens, count in zip(slots, sequences, done) if count])
    step = []
    for index, (slot, tokens, count) in enumerate(zip(slots, sequences, done)):
        step.append(Portion(slot, tokens[count:], [0] if index < case["decode"] else wanted))
    keep = [engine.state[name] for name in sorted(engine.state) if name.startswith(("kv_pool", "delta")) and name.endswith(f".{len(config_of(case)['layers']) - 1}")]
    return Program(kind="ragged", engine=engine, step=step, lengths=dict(zip(slots, done)), count=case["decode"] + len(wanted), keep=keep)


def run(state: Program):
    engine = state.engine
    if state.kind == "llama":
        engine.launch(0, 2, state.stream)
        engine.read_buffer("serving.logits", state.logits.data_ptr(), state.logits.numel() * 4)
        return state.logits
    if state.kind == "encoder":
        return list(engine(state.ids, state.types))
    engine.sequences.length.update(state.lengths)
    engine.step(state.step)
    return {"logits": engine.logits(state.count), "caches": state.keep}


# -- what a pass cannot do without -----------------------------------------------------------------------------------------
def work(case: dict) -> dict:
    config = config_of(case)
    if case["kind"] == "encoder":
        hidden, inter, layers, rows = config["hidden_size"], config["intermediate_size"], config["num_hidden_layers"], case["batch"] * 128
        matrices = layers * (4 * hidden * hidden + 2 * hidden * inter)
        return {"bytes": 2 * matrices + rows * (16 + 4 * hidden), "flops": 2 * matrices * rows + 4 * layers * rows * 128 * hidden}
    if case["kind"] == "llama":
        dim, hidden, batch, context = synthetic.head_dim_of(config), config["hidden_size"], case["batch"], case["context"] + 1
        heads, kv_heads = config["num_attention_heads"], config["num_key_value_heads"]
        matrices = config["num_hidden_layers"] * hidden * (dim * (2 * heads + 2 * kv_heads) + 3 * config["intermediate_size"]) + hidden * config["vocab_size"]
        cached = config["num_hidden_layers"] * batch * context * 2 * kv_heads * dim
        return {"bytes": 2 * (matrices + cached) + 4 * batch * config["vocab_size"], "flops": 2 * matrices * batch + 4 * config["num_hidden_layers"] * batch * context * heads * dim}
    sequences, done, wanted = sequences_of(case, 0)
    width, scored = config["width"], case["decode"] + len(wanted)
    rows = case["decode"] + case["rows"]
    moved, flops = 2 * config["vocab"] * width + 4 * scored * config["vocab"] + 2 * rows * width, 2 * config["vocab"] * width * scored
    for layer in config["layers"]:
        m, mlp = layer["mixer"], layer["mlp"]
        heads, dim = m["heads"], m["dim"]
        if layer["type"] == "general_delta":
            every = width * (6 * width + m["decay_rank"]) + width * m["decay_rank"]
            state = heads * dim * dim
            moved += len(sequences) * 8 * state
            flops += rows * 8 * state
        else:
            if "kv_rank" in m:
                key, value, cached = dim + m["rot_dim"], m["vdim"], m["kv_rank"] + m["rot_dim"]
                every = width * (m["q_rank"] + cached) + heads * key * m["q_rank"] + heads * (dim + value) * m["kv_rank"] + width * heads * value
            else:
                key, value, cached = dim, m["vdim"], m["kv_heads"] * (dim + m["vdim"])
                every = width * (heads * dim + m["kv_heads"] * (dim + value) + 2 * heads * value)
            size = (m.get("mask") or {}).get("size", 1 << 30)
            for tokens, count in zip(sequences, done):
                moved += 2 * cached * (min(len(tokens), size + len(tokens) - count - 1) + len(tokens) - count)
                flops += 2 * heads * (key + value) * sum(min(position + 1, size) for position in range(count, len(tokens)))
        if mlp["kind"] == "moe":
            experts, top = mlp["router"]["experts"], mlp["router"]["top"]
            matrix = width * mlp["expert"]["ff"] * (2 if config["architecture"] == "Nadilorn" else 3)
            every += width * experts
            moved += 2 * matrix * experts * (1.0 - (1.0 - top / experts) ** rows)      # (rows that spread evenly)
            flops += 2 * matrix * top * rows
        else:
            every += 3 * width * mlp["ff"]
        moved += 2 * every
        flops += 2 * every * rows
    return {"bytes": moved, "flops": flops}


def tolerance(case: dict):
    """Four times the error against 64 bits that was measured (encoder 0.001 in 16 bits, 8 layers of the decode plan 0.022,
    ragged steps 0.003 to 0.0055; with experts one close call more or less is allowed for)."""
    if case["kind"] == "encoder":
        return {"rel": 4e-3}
    if case["kind"] == "llama":
        return {"rel": 8e-2}
    return {"rel": 4e-2 if "-a" in case["shape"] else 2e-2}


# -- the same results in 64 bits -------------------------------------------------------------------------------------------
def exact(case: dict, seed: int):
    return {"llama": exact_llama, "encoder": exact_encoder, "ragged": exact_ragged}[case["kind"]](case, seed)


def rms(x: torch.Tensor, eps: float) -> torch.Tensor:
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def turned(x: torch.Tensor, positions: torch.Tensor, frequencies: torch.Tensor, size: float = 1.0, neighbours: bool = False) -> torch.Tensor:
    """Rotary positions on the first 2 x len(frequencies) columns of x [rows, heads, dim]."""
    half = len(frequencies)
    angle = positions[:, None, None].double() * frequencies
    cos, sin = size * angle.cos(), size * angle.sin()
    if neighbours:
        u, v = x[..., 0:2 * half:2], x[..., 1:2 * half:2]
        return torch.cat((torch.stack((u * cos - v * sin, v * cos + u * sin), dim=-1).flatten(-2), x[..., 2 * half:]), dim=-1)
    u, v = x[..., :half], x[..., half:2 * half]
    return torch.cat((u * cos - v * sin, v * cos + u * sin, x[..., 2 * half:]), dim=-1)


def powers(base: float, dims: int) -> torch.Tensor:
    return base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device="cuda") / dims)


def exact_encoder(case: dict, seed: int):
    config, drawn = config_of(case), Drawn(case, seed, torch.float16)
    w = lambda name: drawn.tensor(name).double()
    ids, types = encoder_inputs(case, seed)
    hidden, heads, batch = config["hidden_size"], config["num_attention_heads"], case["batch"]
    norm = lambda x, name: F.layer_norm(x, (hidden,), w(name + ".weight"), w(name + ".bias"), config["layer_norm_eps"])
    linear = lambda x, name: F.linear(x, w(name + ".weight"), w(name + ".bias"))
    split = lambda x: x.view(batch, 128, heads, hidden // heads).transpose(1, 2)
    x = w("embeddings.word_embeddings.weight")[ids] + w("embeddings.token_type_embeddings.weight")[types] + w("embeddings.position_embeddings.weight")[:128]
    x = norm(x, "embeddings.LayerNorm")
    for layer in range(config["num_hidden_layers"]):
        p = f"encoder.layer.{layer}."
        q, k, v = (split(linear(x, p + f"attention.self.{part}")) for part in ("query", "key", "value"))
        mixed = torch.softmax(q @ k.transpose(-1, -2) * (hidden // heads) ** -0.5, dim=-1) @ v
        x = norm(linear(mixed.transpose(1, 2).reshape(batch, 128, hidden), p + "attention.output.dense") + x, p + "attention.output.LayerNorm")
        x = norm(linear(F.gelu(linear(x, p + "intermediate.dense")), p + "output.dense") + x, p + "output.LayerNorm")
    return [x, torch.tanh(linear(x[:, 0], "pooler.dense"))]


def exact_llama(case: dict, seed: int):
    config, drawn, batch, context = config_of(case), Drawn(case, seed, torch.bfloat16), case["batch"], case["context"]
    w = lambda name: drawn.tensor(name).double()
    dim, heads, kv_heads, eps = synthetic.head_dim_of(config), config["num_attention_heads"], config["num_key_value_heads"], config["rms_norm_eps"]
    blocks = (context + 32) // 16
    pool = torch.empty((config["num_hidden_layers"], 2, batch * blocks + 1, kv_heads, 16, dim), dtype=torch.bfloat16, device="cuda")
    pool.normal_(0.0, 0.5, generator=torch.Generator(device="cuda").manual_seed(seed))
    # (cached rows keep their pieces of eight numbers in an order that depends on the position)
    piece = torch.arange(dim // 8, device="cuda")[None, :] ^ (torch.arange(16, device="cuda")[:, None] % 8)
    index = (8 * piece[:, :, None] + torch.arange(8, device="cuda")).reshape(16, dim)
    x = w("model.embed_tokens.weight")[torch.tensor(tokens_of(case, seed, batch, config["vocab_size"]), device="cuda")]
    position, turn = torch.full((batch,), context, device="cuda"), powers(config["rope_theta"], dim)
    for layer in range(config["num_hidden_layers"]):
        p = f"model.layers.{layer}."
        h = rms(x, eps) * w(p + "input_layernorm.weight")
        q = turned((h @ w(p + "self_attn.q_proj.weight").T).view(batch, heads, dim), position, turn)
        k = turned((h @ w(p + "self_attn.k_proj.weight").T).view(batch, kv_heads, dim), position, turn)
        v = (h @ w(p + "self_attn.v_proj.weight").T).view(batch, kv_heads, dim)
        mixed = torch.empty_like(q)
        for b in range(batch):
            rows = [pool[layer, part, b * blocks:(b + 1) * blocks].gather(-1, index.expand(blocks, kv_heads, 16, dim)) for part in (0, 1)]
            keys, values = (torch.cat((row.double().transpose(0, 1).reshape(kv_heads, -1, dim)[:, :context], new[b][:, None]), dim=1) for row, new in zip(rows, (k, v)))
            score = q[b].view(kv_heads, -1, dim) @ keys.transpose(1, 2) * dim ** -0.5
            mixed[b] = (torch.softmax(score, dim=-1) @ values).view(heads, dim)
        x = x + mixed.reshape(batch, -1) @ w(p + "self_attn.o_proj.weight").T
        h = rms(x, eps) * w(p + "post_attention_layernorm.weight")
        x = x + (F.silu(h @ w(p + "mlp.gate_proj.weight").T) * (h @ w(p + "mlp.up_proj.weight").T)) @ w(p + "mlp.down_proj.weight").T
    return (rms(x, eps) * w("model.norm.weight")) @ w("lm_head.weight").T


def exact_ragged(case: dict, seed: int):
    if work(case)["flops"] > 9e12 or case["decode"] * case["context"] + case["history"] + case["rows"] > 24000:
        return None                                    # (too long in 64 bits)
    config, drawn = config_of(case), Drawn(case, seed, torch.bfloat16)
    cast: dict[str, torch.Tensor] = {}

    def w(name: str) -> torch.Tensor:
        if ".e" in name or name == "head":
            return drawn.tensor(name).double()
        if name not in cast:
            cast[name] = drawn.tensor(name).double()
        return cast[name]

    sequences, done, wanted = sequences_of(case, seed)
    forward = exact_nadilorn if config["architecture"] == "Nadilorn" else exact_benarax
    rows = forward(config, w, sequences)
    head, scored = w("head"), []
    for index, (x, count) in enumerate(zip(rows, done)):
        scored.append(x[[count]] if index < case["decode"] else x[torch.tensor(wanted, device="cuda") + count])
    caches = {"general_delta": 1, "attention": 2}.get(config["layers"][-1]["type"], 1)
    return {"logits": torch.cat(scored) @ head.T, "caches": [None] * caches}


def attend(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, scale: float, size: int | None, null_key: bool) -> torch.Tensor:
    """q [T, heads, dim], k and v [T, kv_heads, ...] -> [T, heads * vdim], every position seeing the last `size` ones."""
    count, heads = q.shape[:2]
    places = torch.arange(count, device="cuda")
    gap = places[:, None] - places[None, :]
    hidden = (gap < 0) | (gap >= size) if size else gap < 0
    out = []
    for head in range(heads):
        kv = head // (heads // k.shape[1])
        score = (q[:, head] @ k[:, kv].T * scale).masked_fill(hidden, -math.inf)
        if null_key:
            score = torch.cat((score, torch.zeros_like(score[:, :1])), dim=1)
        out.append(torch.softmax(score, dim=-1)[:, :count] @ v[:, kv])
    return torch.stack(out, dim=1).flatten(1)


def mixture(h: torch.Tensor, chosen: torch.Tensor, expert) -> torch.Tensor:
    """Sum over a row's chosen experts of expert(number, rows, their place among the chosen)."""
    out = torch.zeros_like(h)
    for number in chosen.unique().tolist():
        rows, place = (chosen == number).nonzero(as_tuple=True)
        out.index_add_(0, rows, expert(number, rows, place))
    return out


def exact_nadilorn(config: dict, w, sequences: list[list[int]]) -> list[torch.Tensor]:
    eps, lengths = config["norm"]["eps"], [len(tokens) for tokens in sequences]
    x = w("embed")[torch.tensor(sum(sequences, []), device="cuda")]
    positions = torch.cat([torch.arange(length, device="cuda") for length in lengths])
    for index, layer in enumerate(config["layers"]):
        m, p = layer["mixer"], f"l{index}.mix."
        turn = powers(m["rot"]["base"], m["rot"]["dims"]) / m["rot"]["scaling"]["factor"]
        q = turned((rms(x @ w(p + "q").T, eps) * w(p + "q.norm")).view(-1, m["heads"], m["dim"]), positions, turn)
        k = turned((rms(x @ w(p + "k").T, eps) * w(p + "k.norm")).view(-1, m["kv_heads"], m["dim"]), positions, turn)
        v = (x @ w(p + "v").T).view(-1, m["kv_heads"], m["vdim"])
        mixed = torch.cat([attend(*parts, m["scale"], m["mask"]["size"], True) for parts in zip(*(t.split(lengths) for t in (q, k, v)))])
        x = x + rms((mixed * torch.sigmoid(x @ w(p + "g").T)) @ w(p + "o").T, eps) * w(f"l{index}.norm1")
        p, mlp = f"l{index}.mlp.", layer["mlp"]
        if mlp["kind"] == "dense":
            y = (F.gelu(x @ w(p + "gate").T, approximate="tanh") * (x @ w(p + "up").T)) @ w(p + "down").T
        else:
            score, chosen = torch.sigmoid(x @ w(p + "router").T).topk(mlp["router"]["top"], dim=-1)
            y = mixture(x, chosen, lambda e, rows, place: F.relu((score[rows, place][:, None] * x[rows]) @ w(f"{p}e{e}.up").T) ** 2 @ w(f"{p}e{e}.down").T)
        x = x + rms(y, eps) * w(f"l{index}.norm2")
    return list((rms(x, eps) * w("final.norm")).split(lengths))


def stretched(rot: dict) -> tuple[torch.Tensor, float]:
    plain, scaling = powers(rot["base"], rot["dims"]), rot.get("scaling")
    if not scaling:
        return plain, 1.0
    at = lambda turns: rot["dims"] * math.log(scaling["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(rot["base"]))
    low, high = max(math.floor(at(scaling["fast"])), 0), min(math.ceil(at(scaling["slow"])), rot["dims"] - 1)
    ramp = ((torch.arange(rot["dims"] // 2, device="cuda").double() - low) / max(high - low, 0.001)).clamp(0.0, 1.0)
    return plain / scaling["factor"] * ramp + plain * (1.0 - ramp), 0.1 * math.log(scaling["factor"]) + 1.0


def exact_delta(h: torch.Tensor, lengths: list[int], m: dict, w, p: str, eps: float) -> torch.Tensor:
    heads, dim = m["heads"], m["dim"]
    split = lambda t: [part.view(-1, heads, dim) for part in t.split(lengths)]
    r, k, v = (split(h @ w(p + name).T) for name in ("r", "k", "v"))
    decay = split(torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ w(p + "w1").T) @ w(p + "w2").T + w(p + "w0"))))
    removal = split(torch.sigmoid(h @ w(p + "a").T + w(p + "a.b")))
    longest = max(lengths)
    padded = [torch.stack([F.pad(t, (0, 0, 0, 0, 0, longest - len(t))) for t in part]) for part in (r, k, v, decay, removal)]
    unit = padded[1] / torch.sqrt((padded[1] ** 2).sum(-1, keepdim=True) + 1e-6)
    state, out = torch.zeros(len(lengths), heads, dim, dim, dtype=torch.float64, device="cuda"), []
    for t in range(longest):
        rt, kt, vt, wt, at = (part[:, t] for part in padded)
        ut = unit[:, t]
        seen = torch.einsum("bhd,bhde->bhe", ut, state)
        state = wt[..., None] * state - (at * ut)[..., None] * seen[..., None, :] + kt[..., None] * vt[..., None, :]
        out.append(torch.einsum("bhd,bhde->bhe", rt, state))
    out = torch.stack(out, dim=1)
    o = torch.cat([out[b, :length] for b, length in enumerate(lengths)])
    return (rms(o, eps).flatten(1) * w(p + "norm") * torch.sigmoid(h @ w(p + "g").T)) @ w(p + "o").T


def exact_benarax(config: dict, w, sequences: list[list[int]]) -> list[torch.Tensor]:
    eps, groups, part = config["norm"]["eps"], config["norm"]["groups"], config["token_side"]["dim"]
    lengths, ids = [len(tokens) for tokens in sequences], torch.tensor(sum(sequences, []), device="cuda")
    positions = torch.cat([torch.arange(length, device="cuda") for length in lengths])
    grouped = lambda x, name: rms(x.view(len(x), groups, -1), eps).flatten(1) * w(name)
    x = w("embed")[ids]
    for index, layer in enumerate(config["layers"]):
        m, p = layer["mixer"], f"l{index}.mix."
        h = grouped(x, f"l{index}.norm1")
        kernel = w(f"l{index}.canon1")
        read = h + torch.cat([F.conv1d(F.pad(t.T, (kernel.shape[1] - 1, 0))[None], kernel[:, None], groups=len(kernel))[0].T for t in h.split(lengths)])
        if layer["type"] == "general_delta":
            added = exact_delta(read, lengths, m, w, p, eps)
        else:
            (turn, size), near, rank = stretched(m["rot"]), layer["type"] == "latent_attention", m["kv_rank"]
            q = ((rms(read @ w(p + "dq").T, eps) * w(p + "dq.norm")) @ w(p + "uq").T).view(len(x), m["heads"], -1)
            down = read @ w(p + "dkv").T
            c = rms(down[:, :rank], eps) * w(p + "dkv.norm")
            k = torch.cat(((c @ w(p + "uk").T).view(len(x), m["heads"], -1), turned(down[:, None, rank:], positions, turn, size, near).expand(-1, m["heads"], -1)), dim=-1)
            q = torch.cat((q[..., :m["dim"]], turned(q[..., m["dim"]:], positions, turn, size, near)), dim=-1)
            v = (c @ w(p + "uv").T).view(len(x), m["heads"], -1)
            added = torch.cat([attend(*parts, m["scale"], None, False) for parts in zip(*(t.split(lengths) for t in (q, k, v)))]) @ w(p + "o").T
        p, mlp = f"l{index}.mlp.", layer["mlp"]
        logits, chosen = (h @ w(p + "router").T).topk(mlp["router"]["top"], dim=-1)
        weight, limit = torch.softmax(logits, dim=-1), mlp["expert"]["limit"]

        def expert(e, rows, place):
            g, u = (h[rows] @ w(f"{p}e{e}.gate").T).clamp(max=limit), (h[rows] @ w(f"{p}e{e}.up").T).clamp(-limit, limit)
            return weight[rows, place][:, None] * ((g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(f"{p}e{e}.down").T)

        x = x + added + mixture(h, chosen, expert)
        p = f"l{index}.side."
        e = w("side.embed")[ids][:, index * part:(index + 1) * part]
        x = x + rms((F.gelu(x @ w(p + "gate").T, approximate="tanh") * e) @ w(p + "proj").T, eps) * w(p + "norm")
    return list(grouped(x, "final.norm").split(lengths))
