"""Performance cases: what the engine is run for, through the runner that the engine, the servers and the trace replay drive.

A pass is one of

* ``prefill``: the next ``tokens`` tokens of a chat on one lane, from a cache that is already ``depth`` tokens deep (0: a new request),
  with the logits at ``want`` places of them (1: the last one, as when an answer is to follow; more: a given text is scored);
* ``decode``: the next ``tokens`` tokens of ``lanes`` chats that are about ``depth`` tokens deep, chosen greedily: the captured step with the
  feed of the token before and the read of the token it made, as the engine drives it, and the logits of the last one.

Models have the sizes of this repository's configurations: GLM-5.3 (``glm53_geometry``, four of its layers: one dense, three of 256 FP8
experts, two with their own indexer) and the benchmark's small, medium and routed sizes of the other two families.  Weights are
random, with what a trained model has and random numbers have not: an update is small beside the residual, the router is
sure of its experts (tokens belong to topics, and a topic has experts of its own) and the next token is clear.
"""

from __future__ import annotations

import dataclasses
import math
import zlib
from collections.abc import Mapping

import torch

CAPACITY = 32768  # the benchmark's context
ANSWER = 16  # tokens of a decode pass
CHUNK_ROWS = {"glm": 2048, "namizen": 4096, "zikevik": 4096}  # rows per prefill pass, as the benchmarks have them
SIZES = {
    "small": dict(width=2048, heads=16, kv_heads=4, head_dim=128, ff=8192, vocab=65536, layers=6),
    "medium": dict(width=4096, heads=32, kv_heads=8, head_dim=128, ff=14336, vocab=131072, layers=6),
    "routed": dict(width=4096, heads=32, kv_heads=8, head_dim=128, ff=1536, experts=64, top=4, vocab=131072, layers=6),
}
TOPICS = 64
TOPIC_SHARE = 0.45  # of a token's embedding that its topic explains
UPDATE = {"mixer": 0.6, "ff": 0.25}  # scale of what a layer's parts add to the residual
QUERY = 2.0  # scale of the queries: a row attends to some tens of its keys, not to all of them alike


def listed() -> list[dict]:
    def case(name, model, size, call, tokens, depth, lanes=1, want=1, chunk=8192):
        return dict(name=name, model=model, size=size, call=call, tokens=tokens, depth=depth, lanes=lanes, want=want, chunk=chunk)

    return [
        # a short question to the flagship: the benchmark's prompt, few rows per expert
        case("glm_prompt_200", "glm", "glm53", "prefill", 200, 0),
        # a document: whole passes of 2,048 rows, tensor-core experts and attention over up to 2,048 keys a row
        case("glm_prompt_4096", "glm", "glm53", "prefill", 4096, 0),
        # the next turn of a long chat: a ragged stretch whose rows choose among more keys than they may attend to
        case("glm_turn_777_at_6000", "glm", "glm53", "prefill", 777, 6000, want=8),
        # the headline: one chat answers
        case("glm_decode_1", "glm", "glm53", "decode", ANSWER, 200),
        # four concurrent chats deep in their contexts
        case("glm_decode_4_at_5000", "glm", "glm53", "decode", ANSWER, 5000, lanes=4),
        # the smallest call: one short chat of a small model, latency and launches
        case("namizen_small_decode_1", "namizen", "small", "decode", ANSWER, 300),
        # a long prompt, two passes that see the same chunk
        case("namizen_prompt_8192", "namizen", "medium", "prefill", 8192, 0),
        # a full server
        case("namizen_decode_8_at_3000", "namizen", "medium", "decode", ANSWER, 3000, lanes=8),
        # a ragged prompt through the recurrence and the expanded latent attention
        case("zikevik_prompt_5003", "zikevik", "medium", "prefill", 5003, 0),
        # scoring a given text with routed experts
        case("zikevik_routed_score_1777", "zikevik", "routed", "prefill", 1777, 0, want=8),
        case("zikevik_decode_1_at_2000", "zikevik", "medium", "decode", ANSWER, 2000),
        case("zikevik_routed_decode_8", "zikevik", "routed", "decode", ANSWER, 700, lanes=8),
    ]


def draw(rng) -> dict:
    def spread(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    model = rng.choice(("glm", "namizen", "zikevik"))
    size = {"glm": ("glm53",), "namizen": ("small", "medium"), "zikevik": ("small", "medium", "routed")}[model]
    case = dict(model=model, size=rng.choice(size), call=rng.choice(("prefill", "decode")), tokens=ANSWER, depth=0, lanes=1, want=1,
                chunk=rng.choice((2048, 4096, 8192)))
    if case["call"] == "decode":
        case["lanes"] = rng.randint(1, 4 if model == "glm" else 8)
        case["depth"] = spread(400, 6000 if model == "glm" else 3000)
        case["chunk"] = 8192  # an answer that begins a new chunk leaves less of the old one than a second answer would need
        return case
    case["want"] = rng.choice((1, 8))
    case["tokens"] = spread(24, 4096 if model == "glm" else 8192)
    if rng.random() < 0.4:  # a later turn: within one chunk
        case["tokens"] = spread(24, 2000)
        case["depth"] = spread(100, 6000)
        case["chunk"] = 8192
    return case


# ---------------------------------------------------------------------------------------------------- models
def geometry(case: dict):
    if case["model"] == "glm":
        from glm_tpu_b200.config.model import glm53_geometry

        return dataclasses.replace(glm53_geometry(), num_layers=4, indexer_types=("full", "shared", "full", "shared"),
                                   mlp_layer_types=("dense", "sparse", "sparse", "sparse"))
    s = SIZES[case["size"]]
    if case["model"] == "namizen":
        from glm_tpu_b200.config.namizen import bench_namizen

        return bench_namizen(s["layers"], width=s["width"], heads=s["heads"], kv_heads=s["kv_heads"], head_dim=s["head_dim"], ff=s["ff"],
                             vocab=s["vocab"], chunk=case["chunk"])
    from glm_tpu_b200.config.zikevik import RoutedSpec, bench_zikevik

    routed = RoutedSpec(s["experts"], s["top"], s["ff"]) if "experts" in s else None
    return bench_zikevik(s["layers"], width=s["width"], heads=s["heads"], head_dim=s["head_dim"], ff=s["ff"], vocab=s["vocab"], routed=routed)


class Tensors(Mapping):
    """A checkpoint made on the GPU, a tensor at a time when it is looked up; each depends on the seed and its name alone."""

    def __init__(self, g, seed: int):
        self.seed, self.device = int(seed), torch.device("cuda", torch.cuda.current_device())
        self.vocab, self.width = g.vocab_size, g.hidden_size
        if hasattr(g, "tensor_shapes"):
            self.embed, self.head = "embed", "head"
            self.shapes = dict(g.tensor_shapes())
        else:
            self.embed, self.head = "model.embed_tokens.weight", "lm_head.weight"
            self.shapes = {self.embed: (g.vocab_size, g.hidden_size), self.head: (g.vocab_size, g.hidden_size), "model.norm.weight": (g.hidden_size,)}
            for layer in range(g.num_layers):
                self.shapes.update(_glm_shapes(g, layer))
        experts = getattr(g, "num_routed_experts", None) or 0
        top = getattr(g, "routed_top_k", None) or 0
        for layer in getattr(g, "layers", ()):
            mlp = getattr(layer, "mlp", None)
            experts, top = max(experts, getattr(mlp, "experts", 0)), max(top, getattr(mlp, "top", 0))
        self.experts, self.top = experts, top

    def __iter__(self):
        return iter(self.shapes)

    def __len__(self) -> int:
        return len(self.shapes)

    def __contains__(self, name) -> bool:
        return name in self.shapes

    def _rng(self, name: str) -> torch.Generator:
        return torch.Generator(self.device).manual_seed((self.seed * 1000003 + zlib.crc32(name.encode())) % (1 << 62))

    def _normal(self, name: str, shape, mean: float = 0.0, std: float = 1.0, dtype=torch.bfloat16) -> torch.Tensor:
        return torch.empty(shape, dtype=dtype, device=self.device).normal_(mean, std, generator=self._rng(name))

    def topics(self) -> torch.Tensor:
        return self._normal("topics", (TOPICS, self.width), dtype=torch.float32)

    def topic_of(self) -> torch.Tensor:
        return torch.randint(0, TOPICS, (self.vocab,), device=self.device, generator=self._rng("topic_of"))

    def follows(self) -> torch.Tensor:
        """``[vocab]``: the token that follows a token."""
        return torch.randperm(self.vocab, device=self.device, generator=self._rng("follows"))

    def __getitem__(self, name: str) -> torch.Tensor:
        shape = self.shapes[name]
        leaf = name.rsplit(".", 1)[-1]
        if name == self.embed:
            topic = self.topics().to(torch.bfloat16)[self.topic_of()]
            return topic.mul_(TOPIC_SHARE).add_(self._normal(name, shape, std=math.sqrt(1 - TOPIC_SHARE**2)))
        if name == self.head:
            out = torch.empty(shape, dtype=torch.bfloat16, device=self.device)
            out[self.follows()] = self[self.embed] * shape[1] ** -0.5
            return out
        if leaf == "router" or name.endswith("mlp.gate.weight"):
            # the experts of a topic: their rows point at it (and a little elsewhere, so that scores differ)
            rng = self._rng(name)
            chosen = torch.rand((TOPICS, self.experts), device=self.device, generator=rng).argsort(dim=1)[:, : self.top]
            member = torch.zeros((TOPICS, self.experts), device=self.device).scatter_(1, chosen, 1.0)
            rows = member.T @ self.topics() * (5.0 / self.width) + self._normal(name + ".spread", shape, std=0.2 * self.width**-0.5, dtype=torch.float32)
            return rows.to(torch.bfloat16)
        if leaf == "e_score_correction_bias":
            return self._normal(name, shape, std=0.02, dtype=torch.float32)
        if leaf == "scale_inv":  # of e4m3 codes of standard deviation 64
            scale = torch.empty(shape, device=self.device).uniform_(0.7, 1.4, generator=self._rng(name))
            columns = self.shapes[name[: -len("scale_inv")] + "weight_bits"][-1]
            return scale * (columns**-0.5 / 64.0 * (UPDATE["ff"] if "down_proj" in name else 1.0))
        if leaf == "weight_bits":
            out = torch.empty(shape, dtype=torch.uint8, device=self.device)
            rng = self._rng(name)
            for part in out.split(16):
                z = torch.empty(part.shape, dtype=torch.bfloat16, device=self.device).normal_(0.0, 64.0, generator=rng)
                part.copy_(z.clamp_(-448.0, 448.0).to(torch.float8_e4m3fn).view(torch.uint8))
            return out
        if "layernorm" in name or name.endswith(("model.norm.weight", "k_norm.weight", ".norm", "dq.norm", "dkv.norm")) and name != "final.norm":
            return self._normal(name, shape, 1.0, 0.1)
        if leaf in ("norm1", "norm2") or name == "final.norm":
            return self._normal(name, shape, 0.0 if "l0.mix.A_log" in self.shapes or "l0.mix.dkv" in self.shapes else 1.0, 0.1)
        if name.endswith("k_norm.bias"):
            return self._normal(name, shape, 0.0, 0.05)
        if leaf == "conv":
            out = self._normal(name, shape, 0.0, 0.3)
            out[:, -1] += 0.8
            return out
        if leaf == "vmix":
            return torch.tensor(0.4, dtype=torch.bfloat16, device=self.device)
        if leaf in ("A_log", "dt_bias", "sink"):
            mean, std = {"A_log": (0.0, 0.7), "dt_bias": (-3.0, 1.0), "sink": (0.5, 1.0)}[leaf]
            return self._normal(name, shape, mean, std)
        scale = 1.0
        if leaf == "o" or "o_proj" in name:
            scale = UPDATE["mixer"]
        elif leaf == "down" or "down_proj" in name:
            scale = UPDATE["ff"]
        elif leaf in ("q", "uq") or "q_b_proj" in name:
            scale = QUERY
        return self._normal(name, shape, 0.0, shape[-1] ** -0.5 * scale)


def _glm_shapes(g, layer: int) -> dict:
    """Tensors of a GLM layer: routed experts as FP8 codes and block scales, every other table in bf16."""
    p, H = f"model.layers.{layer}.", g.hidden_size
    a, m = p + "self_attn.", p + "mlp."
    out = {
        p + "input_layernorm.weight": (H,), p + "post_attention_layernorm.weight": (H,), a + "q_a_layernorm.weight": (g.q_lora_rank,),
        a + "kv_a_layernorm.weight": (g.kv_lora_rank,), a + "q_a_proj.weight": (g.q_lora_rank, H),
        a + "kv_a_proj_with_mqa.weight": (g.kv_lora_rank + g.qk_rope_head_dim, H),
        a + "q_b_proj.weight": (g.attention_heads * (g.qk_nope_head_dim + g.qk_rope_head_dim), g.q_lora_rank),
        a + "kv_b_proj.weight": (g.attention_heads * (g.qk_nope_head_dim + g.v_head_dim), g.kv_lora_rank),
        a + "o_proj.weight": (H, g.attention_heads * g.v_head_dim),
    }
    if g.indexer_types[layer] == "full":
        out |= {a + "indexer.wq_b.weight": (g.index_heads * g.index_head_dim, g.q_lora_rank), a + "indexer.wk.weight": (g.index_head_dim, H),
                a + "indexer.k_norm.weight": (g.index_head_dim,), a + "indexer.k_norm.bias": (g.index_head_dim,),
                a + "indexer.weights_proj.weight": (g.index_heads, H)}

    def ff(prefix: str, n: int) -> dict:
        return {prefix + "gate_proj.weight": (n, H), prefix + "up_proj.weight": (n, H), prefix + "down_proj.weight": (H, n)}

    if g.mlp_layer_types[layer] == "dense":
        return out | ff(m, g.dense_intermediate_size)
    out |= {m + "gate.weight": (g.num_routed_experts, H), m + "gate.e_score_correction_bias": (g.num_routed_experts,)}
    out |= ff(m + "shared_experts.", g.moe_intermediate_size * g.num_shared_experts)
    for name, (_, (n, k)) in zip(("gate_proj", "up_proj", "down_proj"), ff("", g.moe_intermediate_size).items()):
        out[f"{m}experts.{name}.weight_bits"] = (g.num_routed_experts, n, k)
        out[f"{m}experts.{name}.scale_inv"] = (g.num_routed_experts, -(-n // 128), -(-k // 128))
    return out


# ---------------------------------------------------------------------------------------------------- a pass
def _depths(case: dict) -> list[int]:
    return [max(1, case["depth"] - 37 * lane) if case["call"] == "decode" else case["depth"] for lane in range(case["lanes"])]


def _texts(case: dict, vocab: int, seed: int) -> list[list[int]]:
    """Per lane, the tokens before the pass and, for a prefill, the pass's own."""
    own = case["tokens"] if case["call"] == "prefill" else 1
    gen = torch.Generator().manual_seed(int(seed) * 7919 + 17)
    return [torch.randint(0, vocab, (depth + own,), generator=gen).tolist() for depth in _depths(case)]


def _places(case: dict) -> list[int]:
    return [(i + 1) * case["tokens"] // case["want"] - 1 for i in range(case["want"])]


def prepare(case: dict, seed: int) -> dict:
    from glm_tpu_b200.runner.gpu_runner import build_runner

    g = geometry(case)
    runner = build_runner(g, device=f"cuda:{torch.cuda.current_device()}", checkpoint=Tensors(g, seed), context_capacity=CAPACITY, lanes=case["lanes"],
                          prefill_chunk=CHUNK_ROWS[case["model"]])
    depths, texts = _depths(case), _texts(case, g.vocab_size, seed)
    for lane, (depth, text) in enumerate(zip(depths, texts)):
        runner.open_lane(lane)
        if depth:
            runner.extend(lane, text[:depth])
    state = dict(case=case, runner=runner, depths=depths, texts=texts, device_depths=torch.tensor(depths, dtype=torch.int32, device=runner.device))
    # what a step overwrites and a position does not bound: the short histories of the convolutions, the recurrent states
    live = [t for name in ("conv", "state") for t in getattr(runner.state, name, []) if t is not None]
    state["saved"] = [(t, t.clone()) for t in live] if any(depths) else []
    if case["call"] == "decode":
        runner.build_decode_program()
    return state


def _back_to_the_question(state: dict) -> None:
    """The lanes as they were when the context had been read: another answer to the same question begins here."""
    runner = state["runner"]
    for tensor, saved in state["saved"]:
        tensor.copy_(saved)
    runner.state.positions.copy_(state["device_depths"])
    runner.lengths[:] = state["depths"]
    if state["case"]["call"] == "decode":
        runner.state.active.fill_(1)


def run(state: dict):
    case, runner = state["case"], state["runner"]
    if case["call"] == "prefill":
        if case["depth"]:
            _back_to_the_question(state)
        else:
            runner.open_lane(0)
        return runner.extend(0, state["texts"][0][case["depth"] :], want=_places(case))
    _back_to_the_question(state)
    tokens = [text[-1] for text in state["texts"]]
    answer = []
    for _ in range(case["tokens"] - 1):
        runner.feed_tokens(dict(enumerate(tokens)))
        runner.decode_step()
        tokens = runner.read_last_tokens()
        answer.append(tokens)
        runner.lengths = [n + 1 for n in runner.lengths]
    logits = runner.decode_logits(dict(enumerate(tokens)))
    return {"tokens": torch.tensor(answer, dtype=torch.int32), "logits": torch.stack([logits[lane] for lane in range(case["lanes"])])}


# ---------------------------------------------------------------------------------------------------- what a pass cannot do without
def work(case: dict) -> dict:
    g = geometry(case)
    decode = case["call"] == "decode"
    steps = case["tokens"] if decode else 1
    rows = case["lanes"] if decode else case["tokens"]  # of a step
    heads_rows = case["lanes"] if decode else case["want"]
    starts = [d + s for d in _depths(case) for s in range(steps)] if decode else list(range(case["depth"], case["depth"] + case["tokens"]))
    weights, macs, cache, attention = 0.0, 0.0, 0.0, 0.0  # bytes a step reads; multiply-adds a row needs; bytes of cache; flops of attention, all in the pass

    def experts(total: int, top: int) -> float:
        return total * (1 - (1 - top / total) ** rows)

    for i in range(g.num_layers):
        if case["model"] == "glm":
            mla = sum(math.prod(s) for n, s in _glm_shapes(g, i).items() if ".self_attn." in n and len(s) == 2)
            weights, macs = weights + 2 * mla, macs + mla
            if g.mlp_layer_types[i] == "dense":
                n = 3 * g.dense_intermediate_size * g.hidden_size
                weights, macs = weights + 2 * n, macs + n
            else:
                n = 3 * g.moe_intermediate_size * g.hidden_size
                weights += 2 * n + experts(g.num_routed_experts, g.routed_top_k) * n + 2 * g.num_routed_experts * g.hidden_size
                macs += (g.routed_top_k + 1) * n + g.num_routed_experts * g.hidden_size
            keys = sum(min(p + 1, g.index_top_k) for p in starts)
            attention += 2 * keys * g.attention_heads * (g.qk_nope_head_dim + g.qk_rope_head_dim + g.v_head_dim)
            row = 2 * (g.kv_lora_rank + g.qk_rope_head_dim)
            cache += row * (keys if decode else starts[-1] + 1 + rows)
            if g.indexer_types[i] == "full":
                every = sum(p + 1 for p in starts)
                attention += 2 * every * g.index_heads * g.index_head_dim
                cache += 2 * g.index_head_dim * (every if decode else starts[-1] + 1)
            continue
        layer = g.layers[i]
        m = layer.mixer
        if case["model"] == "namizen":
            mix = (m.qkv_width + m.out_width) * g.hidden_size
            keys = sum(p % m.chunk + 1 for p in starts)
            attention += 2 * keys * m.heads * (m.dim + m.vdim)
            row = 2 * m.kv_heads * (m.dim + m.vdim)
            cache += row * (keys if decode else rows)
        elif hasattr(m, "kv_rank"):
            mix = sum(math.prod(s) for s in m.tensors(g.hidden_size).values() if len(s) == 2)
            keys = sum(p + 1 for p in starts)
            attention += 2 * keys * m.heads * (m.dim + m.rot_dim + m.vdim)
            row = 2 * (m.kv_rank + m.rot_dim)
            cache += row * (keys if decode else starts[-1] + 1 + rows)
        else:
            mix = sum(math.prod(s) for n, s in m.tensors(g.hidden_size).items() if len(s) == 2 and not n.endswith("conv"))
            attention += 8 * rows * steps * m.heads * m.dim * m.vdim
            cache += 2 * 4 * m.heads * m.dim * m.vdim * (rows * steps if decode else 1)
        weights, macs = weights + 2 * mix, macs + mix
        ff = layer.ff if case["model"] == "namizen" else layer.mlp.ff
        n = 3 * ff * g.hidden_size
        if case["model"] == "zikevik" and hasattr(layer.mlp, "experts"):
            router = layer.mlp.experts * g.hidden_size
            weights += 2 * (experts(layer.mlp.experts, layer.mlp.top) * n + router)
            macs += layer.mlp.top * n + router
        else:
            weights, macs = weights + 2 * n, macs + n
    head = g.vocab_size * g.hidden_size
    io = steps * rows * 2 * g.hidden_size + heads_rows * g.vocab_size * 4
    return {"bytes": steps * (weights + 2 * head) + cache + io, "flops": 2 * steps * (rows * macs + heads_rows * head) + attention}


def tolerance(case: dict):
    # against ``exact`` the GLM model (bf16 residual and updates) is up to 0.008 off, the others (fp32 residual) up to 0.0023
    return {"rel": 0.025 if case["model"] == "glm" else 0.008}


# ---------------------------------------------------------------------------------------------------- in 64 bits
F64 = torch.float64


def exact(case: dict, seed: int):
    g = geometry(case)
    tensors = Tensors(g, seed)
    forward = {"glm": _glm, "namizen": _namizen, "zikevik": _zikevik}[case["model"]]
    texts = _texts(case, g.vocab_size, seed)
    if case["call"] == "prefill":
        at = [[case["depth"] + place for place in _places(case)]]
    else:
        # greedily: the next token is the clear one, which the answer's own tokens below confirm
        after = tensors.follows().cpu()
        for text in texts:
            for _ in range(case["tokens"] - 1):
                text.append(int(after[text[-1]]))
        at = [list(range(len(text) - case["tokens"], len(text))) for text in texts]
    hidden = forward(g, tensors, texts, at)
    head = tensors[tensors.head]
    logits = [torch.cat([h @ part.to(F64).T for part in head.split(16384)], dim=1) for h in hidden]
    if case["call"] == "prefill":
        return logits[0].cpu()
    tokens = torch.stack([x[:-1].argmax(dim=1) for x in logits], dim=1).to(torch.int32)
    return {"tokens": tokens.cpu(), "logits": torch.stack([x[-1] for x in logits]).cpu()}


def _mm(x: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
    return x @ w.to(F64).T


def _rms(x: torch.Tensor, weight: torch.Tensor, eps: float) -> torch.Tensor:
    return x * torch.rsqrt(x.square().mean(dim=-1, keepdim=True) + eps) * weight.to(F64)


def _turn(x: torch.Tensor, dims: int, base: float, pairs: bool) -> torch.Tensor:
    """Rotary positions of ``x [T, heads, dim]`` on its first ``dims`` features: neighbours are a pair, or a feature and the one half way on."""
    j = torch.arange(dims // 2, dtype=F64, device=x.device)
    angle = torch.arange(x.shape[0], dtype=F64, device=x.device)[:, None] * base ** (-2.0 * j / dims)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    u, v = (x[..., 0:dims:2], x[..., 1:dims:2]) if pairs else (x[..., : dims // 2], x[..., dims // 2 : dims])
    a, b = u * cos - v * sin, v * cos + u * sin
    turned = torch.stack([a, b], dim=-1).flatten(-2) if pairs else torch.cat([a, b], dim=-1)
    return torch.cat([turned, x[..., dims:]], dim=-1)


def _attend(q, k, v, visible, scale: float, sink=None) -> torch.Tensor:
    """One head: ``q [T, d]``, ``k [T, d]``, ``v [T, e]``; a sink takes part in the denominator only."""
    s = (q @ k.T).mul_(scale).masked_fill_(~visible, -math.inf)
    top = s.amax(dim=1, keepdim=True)
    if sink is not None:
        top = torch.maximum(top, sink.to(F64))
    p = s.sub_(top).exp_()
    total = p.sum(dim=1, keepdim=True)
    return p @ v / (total if sink is None else total + torch.exp(sink.to(F64) - top))


def _conv(u: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    taps = weight.shape[1]
    padded = torch.cat([torch.zeros((taps - 1, u.shape[1]), dtype=F64, device=u.device), u])
    return sum(weight[:, j].to(F64) * padded[j : j + u.shape[0]] for j in range(taps))


def _causal(total: int, device) -> torch.Tensor:
    return torch.ones((total, total), dtype=torch.bool, device=device).tril_()


def _silu(z: torch.Tensor) -> torch.Tensor:
    return z * torch.sigmoid(z)


def _gated(h: torch.Tensor, gate, up, down, act=_silu) -> torch.Tensor:
    return _mm(act(_mm(h, gate)) * _mm(h, up), down)


def _glm(g, t: Tensors, texts, at) -> list[torch.Tensor]:
    table = t[t.embed]
    xs = [table[torch.tensor(text, device=t.device)].to(F64) for text in texts]
    del table
    L, dn, dv, rd, dh, eps = g.kv_lora_rank, g.qk_nope_head_dim, g.v_head_dim, g.qk_rope_head_dim, g.index_head_dim, g.rms_norm_eps
    visible: list = [None] * len(xs)
    for i in range(g.num_layers):
        w = lambda name, i=i: t[f"model.layers.{i}.{name}.weight"]  # noqa: E731
        kv_b = w("self_attn.kv_b_proj").view(g.attention_heads, dn + dv, L)
        for lane, x in enumerate(xs):
            total = x.shape[0]
            h = _rms(x, w("input_layernorm"), eps)
            resid = _rms(_mm(h, w("self_attn.q_a_proj")), w("self_attn.q_a_layernorm"), eps)
            joint = _mm(h, w("self_attn.kv_a_proj_with_mqa"))
            latent = _rms(joint[:, :L], w("self_attn.kv_a_layernorm"), eps)
            turned = _turn(joint[:, None, L:], rd, g.rope_theta, True)[:, 0]
            if g.indexer_types[i] == "full":
                visible[lane] = _causal(total, x.device)
                if total > g.index_top_k:
                    key = _mm(h, w("self_attn.indexer.wk"))
                    key = torch.nn.functional.layer_norm(key, (dh,), w("self_attn.indexer.k_norm").to(F64), t[f"model.layers.{i}.self_attn.indexer.k_norm.bias"].to(F64), 1e-6)
                    key = _turn(key[:, None], rd, g.rope_theta, True)[:, 0]
                    query = _turn(_mm(resid, w("self_attn.indexer.wq_b")).view(total, g.index_heads, dh), rd, g.rope_theta, True)
                    share = _mm(h, w("self_attn.indexer.weights_proj"))
                    scores = torch.zeros((total, total), dtype=F64, device=x.device)
                    for head in range(g.index_heads):
                        scores.addcmul_((query[:, head] @ key.T).relu_(), share[:, head, None])
                    scores.masked_fill_(~visible[lane], -math.inf)
                    chosen = scores.topk(g.index_top_k, dim=1).indices
                    visible[lane] &= torch.zeros_like(visible[lane]).scatter_(1, chosen, True)
                    del scores, chosen
            q_b, out = w("self_attn.q_b_proj").view(g.attention_heads, dn + rd, -1), []
            for head in range(g.attention_heads):
                q = _mm(resid, q_b[head])
                q = torch.cat([q[:, :dn], _turn(q[:, None, dn:], rd, g.rope_theta, True)[:, 0]], dim=1)
                k = torch.cat([_mm(latent, kv_b[head, :dn]), turned], dim=1)
                out.append(_attend(q, k, _mm(latent, kv_b[head, dn:]), visible[lane], (dn + rd) ** -0.5))
            xs[lane] = x + _mm(torch.cat(out, dim=1), w("self_attn.o_proj"))
        x = torch.cat(xs)
        h = _rms(x, w("post_attention_layernorm"), eps)
        if g.mlp_layer_types[i] == "dense":
            x = x + _gated(h, w("mlp.gate_proj"), w("mlp.up_proj"), w("mlp.down_proj"))
        else:
            scores = torch.sigmoid(_mm(h, w("mlp.gate")))
            chosen = (scores + t[f"model.layers.{i}.mlp.gate.e_score_correction_bias"].to(F64)).topk(g.routed_top_k, dim=1).indices
            share = scores.gather(1, chosen)
            share = share / share.sum(dim=1, keepdim=True)
            x = x + _gated(h, *(w(f"mlp.shared_experts.{n}_proj") for n in ("gate", "up", "down")))
            tables = {n: tuple(t[f"model.layers.{i}.mlp.experts.{n}_proj.{part}"] for part in ("weight_bits", "scale_inv")) for n in ("gate", "up", "down")}
            for e in range(g.num_routed_experts):
                rows, slot = (chosen == e).nonzero(as_tuple=True)
                if len(rows):
                    y = _gated(h[rows], *(_decoded(bits[e], scale[e]) for bits, scale in tables.values()))
                    x.index_add_(0, rows, y * (share[rows, slot] * g.routed_scaling_factor)[:, None])
        xs = list(x.split([len(text) for text in texts]))
    return [_rms(x[places], t["model.norm.weight"], eps) for x, places in zip(xs, at)]


def _decoded(bits: torch.Tensor, scale: torch.Tensor) -> torch.Tensor:
    """The bf16 table that e4m3 codes with a scale per 128 x 128 block stand for."""
    n, k = bits.shape
    full = scale.repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)[:, :k]
    return (bits.view(torch.float8_e4m3fn).float() * full).to(torch.bfloat16)


def _gelu(z: torch.Tensor) -> torch.Tensor:
    return torch.nn.functional.gelu(z, approximate="tanh")


def _namizen(g, t: Tensors, texts, at) -> list[torch.Tensor]:
    out, table = [], t["embed"]
    for text, places in zip(texts, at):
        x, first = table[torch.tensor(text, device=t.device)].to(F64), None
        total = x.shape[0]
        for i, layer in enumerate(g.layers):
            m, w = layer.mixer, lambda name, i=i: t[f"l{i}.{name}"]
            h = _rms(x, w("norm1"), g.norm_eps)
            q, k, v = (_conv(_mm(h, w("mix." + n)), w(f"mix.{n}.conv")) for n in "qkv")
            q = _turn(q.view(total, m.heads, m.dim), m.rot_dims, m.rot_base, False)
            k = _turn(k.view(total, m.kv_heads, m.dim), m.rot_dims, m.rot_base, False)
            v = v.view(total, m.kv_heads, m.vdim)
            if first is None:
                first = v
            else:
                amount = w("mix.vmix").to(F64)
                v = (1 - amount) * v + amount * first
            sink, per, mixed = w("mix.sink"), m.heads // m.kv_heads, torch.empty((total, m.heads, m.vdim), dtype=F64, device=x.device)
            for low in range(0, total, m.chunk):
                part = slice(low, min(total, low + m.chunk))
                seen = _causal(part.stop - low, x.device)
                for head in range(m.heads):
                    mixed[part, head] = _attend(q[part, head], k[part, head // per], v[part, head // per], seen, m.scale, sink[head])
            update = _mm(mixed.flatten(1), w("mix.o"))
            h = _rms(x, w("norm2"), g.norm_eps)
            x = x + update + _gated(h, w("mlp.gate"), w("mlp.up"), w("mlp.down"), _gelu)
        out.append(_rms(x[places], t["final.norm"], g.norm_eps))
    return out


def _unit(x: torch.Tensor) -> torch.Tensor:
    return x * torch.rsqrt(x.square().sum(dim=-1, keepdim=True) + 1e-6)


def _delta_rule(m, h: list[torch.Tensor], w, eps: float) -> list[torch.Tensor]:
    """The gated delta rule, token by token; sequences of different lengths side by side (what follows a shorter one's end is cut off)."""
    parts, longest = [], max(x.shape[0] for x in h)
    for x in h:
        total = x.shape[0]
        q, k, v = (_silu(_conv(_mm(x, w(n)), w(n + ".conv"))) for n in "qkv")
        q, k = (_unit(y.view(total, m.kv_heads, m.dim)).repeat_interleave(m.heads // m.kv_heads, dim=1) for y in (q, k))
        step = torch.nn.functional.softplus(_mm(_mm(x, w("a1")), w("a2")) + w("dt_bias").to(F64)).view(total, m.heads, m.dim)
        decay = torch.exp(-torch.exp(w("A_log").to(F64))[:, None] * step)
        beta = torch.sigmoid(_mm(x, w("b")))[..., None]
        rows = (q * m.dim**-0.5, k, v.view(total, m.heads, m.vdim), decay, beta)
        parts.append([torch.nn.functional.pad(y, (0, 0, 0, 0, 0, longest - total)) for y in rows])
    q, k, v, decay, beta = (torch.stack(p, dim=1).flatten(1, 2) for p in zip(*parts))  # [T, lanes * heads, .]
    state = torch.zeros((q.shape[1], m.dim, m.vdim), dtype=F64, device=q.device)
    read = torch.empty_like(v)
    q, k, v, decay, read = q[:, :, None], k[:, :, None], v[:, :, None], decay[..., None], read[:, :, None]
    for i in range(longest):
        state.mul_(decay[i])
        wrong = torch.baddbmm(v[i], k[i], state, alpha=-1).mul_(beta[i][:, None])
        state.baddbmm_(k[i].transpose(1, 2), wrong)
        torch.bmm(q[i], state, out=read[i])
    read = read.view(longest, len(h), m.heads, m.vdim)
    out = []
    for lane, x in enumerate(h):
        o = _rms(read[: x.shape[0], lane], w("norm"), eps)
        gate = torch.sigmoid(_mm(_mm(x, w("g1")), w("g2"))).view(o.shape)
        out.append(_mm((o * gate).flatten(1), w("o")))
    return out


def _latent(m, h: torch.Tensor, w, eps: float) -> torch.Tensor:
    total, out = h.shape[0], []
    q = _mm(_rms(_mm(h, w("dq")), w("dq.norm"), eps), w("uq")).view(total, m.heads, m.dim + m.rot_dim)
    joint = _mm(h, w("dkv"))
    latent = _rms(joint[:, : m.kv_rank], w("dkv.norm"), eps)
    turned = _turn(joint[:, None, m.kv_rank :], m.rot_dim, m.rot_base, True)[:, 0]
    q_turned = _turn(q[..., m.dim :], m.rot_dim, m.rot_base, True)
    k, v = _mm(latent, w("uk")).view(total, m.heads, m.dim), _mm(latent, w("uv")).view(total, m.heads, m.vdim)
    seen, sink = _causal(total, h.device), w("sink")
    for head in range(m.heads):
        out.append(_attend(torch.cat([q[:, head, : m.dim], q_turned[:, head]], dim=1), torch.cat([k[:, head], turned], dim=1), v[:, head], seen, m.scale, sink[head]))
    mixed = torch.stack(out, dim=1) * torch.sigmoid(_mm(h, w("g")))[..., None]
    return _mm(mixed.flatten(1), w("o"))


def _zikevik(g, t: Tensors, texts, at) -> list[torch.Tensor]:
    table = t["embed"]
    x = torch.cat([table[torch.tensor(text, device=t.device)].to(F64) * g.embedding_scale for text in texts])
    lengths = [len(text) for text in texts]
    for i, layer in enumerate(g.layers):
        w = lambda name, i=i: t[f"l{i}.mix.{name}"]  # noqa: E731
        h = _rms(x, 1 + t[f"l{i}.norm1"].to(F64), g.norm_eps).split(lengths)
        x = x + torch.cat([_latent(layer.mixer, y, w, g.norm_eps) for y in h] if hasattr(layer.mixer, "kv_rank") else _delta_rule(layer.mixer, h, w, g.norm_eps))
        h = _rms(x, 1 + t[f"l{i}.norm2"].to(F64), g.norm_eps)
        if not hasattr(layer.mlp, "experts"):
            x = x + _gated(h, *(t[f"l{i}.mlp.{n}"] for n in ("gate", "up", "down")))
            continue
        share, chosen = torch.sigmoid(_mm(h, t[f"l{i}.mlp.router"])).topk(layer.mlp.top, dim=1)
        for e in range(layer.mlp.experts):
            rows, slot = (chosen == e).nonzero(as_tuple=True)
            if len(rows):
                x.index_add_(0, rows, _gated(h[rows] * share[rows, slot][:, None], *(t[f"l{i}.mlp.e{e}.{n}"] for n in ("gate", "up", "down"))))
    return [_rms(y[places], 1 + t["final.norm"].to(F64), g.norm_eps) for y, places in zip(x.split(lengths), at)]
