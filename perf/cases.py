"""The work that users of this framework have it do, as cases that can be timed and compared.

Every case runs on the seeded synthetic models of ``bobcat_b200.synth`` (the shapes of the benchmark
configurations) through the public classes: prompts, decoded tokens, host-stepped turns, several
sequences at once, cached prefixes, scored labels, sampled replies, and the mixture-of-experts block
through the op calls. A model's weights are loaded once per process, as a serving program does; the
inputs (tokens, activations, draws) come from the seed alone.

Contexts of the cases that return token ids are taken token by token (float32 operands), so that the
tokens that follow do not hang on the rounding of a half-precision prefill.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from bobcat_b200 import Q4_0, BatchCuda, Cuda, Engine, Model, Norm, SeqCuda, synth
from bobcat_b200._lib import Sampling

# ---------------------------------------------------------------------------------------- the cases


def listed() -> list[dict]:
    return [
        # A first chat message of a few words on the smallest model: time to its first logits.
        dict(name="prompt 350m 11", kind="prompt", model="lfm2-350m", tokens=11, chunk=0, kv_half=True),
        # The headline prompt: 512 tokens of the 2.6B shape, in one call.
        dict(name="prompt 2.6b 512", kind="prompt", model="lfm2-2.6b", tokens=512, chunk=0, kv_half=True),
        # A document fed to the DeltaNet model in the 64-token chunks of its benchmark configuration.
        dict(name="prompt qwen-2b 64s", kind="prompt", model="qwen35-2b", tokens=2048, chunk=64, kv_half=True),
        # A request of its own behind a cached 4096-token prefix (shared pages) on the largest model.
        dict(name="suffix qwen-9b", kind="suffix", model="qwen35-9b", context=4096, tokens=1501, kv_half=True),
        # Greedy replies, one sequence: small model with an f32 cache, headline model, mixture of experts.
        dict(name="decode 350m", kind="decode", model="lfm2-350m", context=128, steps=32, kv_half=False),
        dict(name="decode 2.6b", kind="decode", model="lfm2-2.6b", context=512, steps=32, kv_half=True),
        dict(name="decode moe-8b", kind="decode", model="lfm2moe-8b-a1b", context=256, steps=16, kv_half=True),
        # A handful of users served together, one token each per pass.
        dict(name="batch 2.6b x6", kind="batch", model="lfm2-2.6b", seqs=6, context=40, steps=8, kv_half=True),
        # The next turn of a conversation: back to the checkpoint, the new message, then tokens whose
        # logits the host's own sampler reads.
        dict(name="turn qwen-2b", kind="turn", model="qwen35-2b", context=700, tokens=37, steps=8, kv_half=True),
        # A short question answered by the engine with device-side sampling.
        dict(name="reply 2.6b", kind="reply", model="lfm2-2.6b", tokens=13, steps=16, sampled=True, kv_half=True),
        # Label scoring (classification): prompts that share their beginning.
        dict(name="score 2.6b", kind="score", model="lfm2-2.6b", context=200, prompts=5, tokens=23, labels=4, kv_half=True),
        # One mixture-of-experts block of a prefill chunk, through the op calls.
        dict(name="experts 8b", kind="experts", tokens=203),
    ]


def _log_int(rng, low: int, high: int) -> int:
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high + 1)))))))


def draw(rng) -> dict:
    kind = rng.choice(["prompt", "prompt", "prompt", "suffix", "decode", "decode", "batch", "turn", "reply", "score", "experts"])
    kv_half = rng.random() < 0.8
    if kind == "prompt":
        return dict(kind=kind, model=rng.choice(["lfm2-350m", "lfm2-2.6b", "qwen35-2b"]), tokens=_log_int(rng, 1, 2048),
                    chunk=rng.choice([0, 0, 0, 64, 100, 256]), kv_half=kv_half)
    if kind == "suffix":
        return dict(kind=kind, model=rng.choice(["lfm2-2.6b", "qwen35-2b", "qwen35-9b"]), context=_log_int(rng, 300, 4096),
                    tokens=_log_int(rng, 20, 1500), kv_half=True)
    if kind == "decode":
        return dict(kind=kind, model=rng.choice(["lfm2-350m", "lfm2-2.6b", "qwen35-2b", "lfm2moe-8b-a1b"]), context=_log_int(rng, 16, 700),
                    steps=_log_int(rng, 4, 48), kv_half=kv_half)
    if kind == "batch":
        return dict(kind=kind, model=rng.choice(["lfm2-350m", "lfm2-2.6b", "lfm2moe-8b-a1b"]), seqs=rng.randint(2, 15),
                    context=_log_int(rng, 16, 48), steps=rng.randint(2, 8), kv_half=kv_half)
    if kind == "turn":
        return dict(kind=kind, model=rng.choice(["lfm2-2.6b", "qwen35-2b", "qwen35-9b"]), context=_log_int(rng, 100, 3000),
                    tokens=_log_int(rng, 1, 128), steps=rng.randint(2, 12), kv_half=kv_half)
    if kind == "reply":
        return dict(kind=kind, model=rng.choice(["lfm2-350m", "lfm2-2.6b", "qwen35-2b"]), tokens=rng.randint(2, 15), steps=_log_int(rng, 4, 24),
                    sampled=rng.random() < 0.6, kv_half=kv_half)
    if kind == "score":
        return dict(kind=kind, model=rng.choice(["lfm2-350m", "lfm2-2.6b", "qwen35-2b"]), context=_log_int(rng, 40, 600), prompts=rng.randint(2, 6),
                    tokens=_log_int(rng, 4, 64), labels=rng.randint(2, 8), kv_half=kv_half)
    return dict(kind=kind, tokens=_log_int(rng, 2, 512))


# --------------------------------------------------------------------------------- what a program keeps

_kept: dict = {}


def _cuda() -> Cuda:
    if "cuda" not in _kept:
        _kept["cuda"] = Cuda.open(0)
    return _kept["cuda"]


def _model(name: str) -> Model:
    if name not in _kept:
        _kept[name] = Model.load(synth.cached_model(name))
    return _kept[name]


EXPERTS = synth.CONFIGS["lfm2moe-8b-a1b"]


def _expert_weights() -> dict:
    """One layer's experts, router and norm of the 8B-A1B shape: Q4_0 blocks with scales of
    N(0, 0.02) weights (0.02 * 4 / 8, spread by a quarter)."""
    if "experts" not in _kept:
        cuda, c = _cuda(), EXPERTS
        rng = np.random.default_rng(7)

        def matrix(n_rows, n_cols):
            blocks = rng.integers(0, 256, (n_rows * n_cols // 32, 18), dtype=np.uint8)
            blocks[:, :2] = (rng.uniform(0.0075, 0.0125, blocks.shape[0]).astype(np.float16)).view(np.uint8).reshape(-1, 2)
            return cuda.upload_matrix(Q4_0, blocks.reshape(-1), n_rows, n_cols)

        h, ff, e = c["hidden"], c["ff_expert"], c["experts"]
        _kept["experts"] = dict(
            gate=matrix(e * ff, h), up=matrix(e * ff, h), down=matrix(e * h, ff),
            router=cuda.buffer_from((rng.standard_normal((e, h)) * 0.02).astype(np.float32)),
            bias=cuda.buffer_from((rng.standard_normal(e) * 0.02).astype(np.float32)), norm=cuda.buffer_from(np.ones(h, dtype=np.float32)))
    return _kept["experts"]


class _OnDevice:
    """A buffer of the backend seen as an array on the device."""

    def __init__(self, buffer, shape):
        self.buffer = buffer  # lives as long as the array
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f4", data=(buffer.device_ptr, False), version=2)


def _tokens(rng, model: Model, n: int) -> np.ndarray:
    return rng.integers(0, model.hp.n_vocab, size=n).astype(np.uint32)


def _step_all(seq: SeqCuda, tokens: np.ndarray) -> None:
    for t in tokens[:-1]:
        seq.step(int(t))
    seq.step(int(tokens[-1]), np.empty(seq.model.hp.n_vocab, dtype=np.float32))


def prepare(case: dict, seed: int) -> dict:
    kind, cuda = case["kind"], _cuda()
    rng = np.random.default_rng(seed)
    if kind == "experts":
        w, c, n = _expert_weights(), EXPERTS, case["tokens"]
        h, ff, used = c["hidden"], c["ff_expert"], c["experts_used"]
        x = rng.standard_normal((n, h)).astype(np.float32)
        y = cuda.new_buffer(x.nbytes)
        return dict(case=case, w=w, x=cuda.buffer_from(x), y=y, normed=cuda.new_buffer(x.nbytes), route=cuda.new_buffer(cuda.route_bytes(used, n)),
                    offsets=cuda.new_buffer((c["experts"] + 1) * 4), entries=cuda.new_buffer(n * used * 4), ffn=cuda.new_buffer(n * used * ff * 4),
                    out=cuda.new_buffer(n * used * h * 4), y_array=torch.as_tensor(_OnDevice(y, (n, h)), device="cuda"))
    model = _model(case["model"])
    half = case["kv_half"]
    if kind == "prompt":
        seq = SeqCuda(model, cuda, max(64, case["tokens"] + 32), half)
        return dict(case=case, seq=seq, tokens=_tokens(rng, model, case["tokens"]), logits=np.zeros(model.hp.n_vocab, dtype=np.float32))
    if kind == "suffix":
        n_ctx = case["context"] + case["tokens"] + 32
        source = SeqCuda(model, cuda, n_ctx, half, paged=True)
        source.prefill(_tokens(rng, model, case["context"]))
        prefix = source.save_prefix()
        source.close()
        return dict(case=case, seq=SeqCuda(model, cuda, n_ctx, half, paged=True), prefix=prefix, tokens=_tokens(rng, model, case["tokens"]),
                    logits=np.zeros(model.hp.n_vocab, dtype=np.float32))
    if kind == "decode":
        seq = SeqCuda(model, cuda, case["context"] + case["steps"] + 32, half)
        _step_all(seq, _tokens(rng, model, case["context"]))
        return dict(case=case, seq=seq, start=seq.checkpoint())
    if kind == "batch":
        batch = BatchCuda(model, cuda, case["seqs"], case["context"] + case["steps"] + 32, half)
        for i in range(case["seqs"]):  # the sequences stand at different positions
            _step_all(batch.seq(i), _tokens(rng, model, case["context"] - (3 * i) % 14))
        return dict(case=case, batch=batch, starts=[batch.seq(i).checkpoint() for i in range(case["seqs"])])
    if kind == "turn":
        seq = SeqCuda(model, cuda, case["context"] + case["tokens"] + case["steps"] + 32, half)
        seq.prefill(_tokens(rng, model, case["context"]))
        return dict(case=case, seq=seq, start=seq.checkpoint(), tokens=_tokens(rng, model, case["tokens"]),
                    picked=[int(t) for t in _tokens(rng, model, case["steps"])],
                    logits=np.zeros((1 + case["steps"], model.hp.n_vocab), dtype=np.float32))
    if kind == "reply":
        settings = Sampling(0.8, 40, 0.95, 0.05, 1.1) if case["sampled"] else None
        return dict(case=case, engine=Engine(model, cuda, case["tokens"] + case["steps"] + 64, half, seed=seed), settings=settings,
                    tokens=_tokens(rng, model, case["tokens"]))
    shared = _tokens(rng, model, case["context"])
    prompts = [np.concatenate([shared, _tokens(rng, model, case["tokens"] + i % 3)]) for i in range(case["prompts"])]
    return dict(case=case, engine=Engine(model, cuda, case["context"] + case["tokens"] + 64, half), prompts=prompts,
                labels=[_tokens(rng, model, case["labels"]) for _ in prompts])


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "prompt":
        seq, tokens, logits = state["seq"], state["tokens"], state["logits"]
        seq.reset()
        chunk = case["chunk"] or len(tokens)
        for at in range(0, len(tokens), chunk):
            seq.prefill(tokens[at:at + chunk], logits if at + chunk >= len(tokens) else None)
        return logits
    if kind == "suffix":
        state["seq"].load_prefix(state["prefix"])
        state["seq"].prefill(state["tokens"], state["logits"])
        return state["logits"]
    if kind == "decode":
        state["seq"].restore(state["start"])
        return state["seq"].generate(case["steps"])
    if kind == "batch":
        for i, start in enumerate(state["starts"]):
            state["batch"].seq(i).restore(start)
        return state["batch"].generate(case["steps"])
    if kind == "turn":
        seq, logits = state["seq"], state["logits"]
        seq.restore(state["start"])
        seq.prefill(state["tokens"], logits[0])
        for i, token in enumerate(state["picked"]):
            seq.step(token, logits[1 + i])
        return logits
    if kind == "reply":
        return np.array(state["engine"].generate(state["tokens"], case["steps"], sampling=state["settings"])[0], dtype=np.uint32)
    if kind == "score":
        return np.array(state["engine"].score(state["prompts"], state["labels"]), dtype=np.float64)
    cuda, w, c, n = _cuda(), state["w"], EXPERTS, case["tokens"]
    h, ff, e, used = c["hidden"], c["ff_expert"], c["experts"], c["experts_used"]
    cuda.begin()
    cuda.copy(state["x"], state["y"], n * h)
    cuda.moe_route(state["x"], (Norm(w["norm"].at(0), c["eps"]), state["normed"].at(0)), w["router"], w["bias"], state["route"], h, e, used, n)
    cuda.moe_group(state["route"], state["offsets"], state["entries"], e, used, n)
    cuda.matmul_experts(Q4_0, w["gate"], w["up"], ff, h, e, state["normed"], True, state["offsets"], state["entries"], used, state["ffn"], n)
    cuda.matmul_experts(Q4_0, w["down"], None, h, ff, e, state["ffn"], False, state["offsets"], state["entries"], used, state["out"], n)
    cuda.moe_combine(state["out"], state["route"], state["y"], h, used, n)
    cuda.end()
    return state["y_array"]


# ------------------------------------------------------------------------------- what it cannot do without


def _shape(name: str) -> dict:
    """Weights of the linears a token multiplies, bytes of cache and state, by the model's shape."""
    c = synth.CONFIGS[name]
    h, layers = c["hidden"], c["layers"]
    if c["arch"] == "qwen35":
        n_attn = layers // 4
        q, kv = c["heads"] * c["head_dim"], c["kv_heads"] * c["head_dim"]
        key, value = c["k_heads"] * c["k_dim"], c["v_heads"] * c["v_dim"]
        linears = n_attn * h * (3 * q + 2 * kv) + (layers - n_attn) * h * (2 * key + 3 * value + 2 * c["v_heads"]) + layers * 3 * h * c["ff"]
        state = (layers - n_attn) * c["v_heads"] * c["k_dim"] * c["v_dim"] * 4
        experts = 0
    else:
        n_attn, q, kv = len(c["attention"]), h, c["kv_heads"] * (h // c["heads"])
        dense = c.get("dense_layers", layers)
        linears = n_attn * h * (2 * q + 2 * kv) + (layers - n_attn) * 4 * h * h + dense * 3 * h * c["ff"]
        state = (layers - n_attn) * (c["conv_kernel"] - 1) * h * 4
        experts = (layers - dense) * 3 * h * c.get("ff_expert", 0)  # weights of one expert in every such layer
    return dict(linears=linears, experts=experts, n_experts=c.get("experts", 0), used=c.get("experts_used", 0), output=h * c["vocab"],
                attention=n_attn, q=q, kv=kv, state=state)


def _forward(name: str, n: int, start: int, kv_bytes: int, logits: int, rows: int = 1) -> tuple[float, float]:
    """(bytes, flops) of one pass over n tokens of each of `rows` sequences from position `start`, with `logits` rows of logits."""
    s = _shape(name)
    tokens = n * rows
    picked = min(s["n_experts"], tokens * s["used"])
    b = (s["linears"] + picked * s["experts"]) * 18 / 32 + 2 * s["state"] * rows
    b += s["attention"] * s["kv"] * 2 * kv_bytes * (start + n) * rows + (s["output"] * 4 if logits else 0)
    f = 2.0 * tokens * (s["linears"] + s["used"] * s["experts"]) + 2.0 * logits * s["output"]
    f += 4.0 * s["attention"] * s["q"] * rows * (n * start + n * (n + 1) / 2)
    return b, f


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "experts":
        c, n = EXPERTS, case["tokens"]
        one = 3 * c["hidden"] * c["ff_expert"]
        return dict(bytes=min(c["experts"], n * c["experts_used"]) * one * 18 / 32 + 3 * n * c["hidden"] * 4, flops=2.0 * n * c["experts_used"] * one)
    name, kv_bytes = case["model"], 2 if case["kv_half"] else 4
    passes = []  # (tokens, start, logits, rows)
    if kind == "prompt":
        chunk = case["chunk"] or case["tokens"]
        passes = [(min(chunk, case["tokens"] - at), at, int(at + chunk >= case["tokens"]), 1) for at in range(0, case["tokens"], chunk)]
    elif kind == "suffix":
        passes = [(case["tokens"], case["context"], 1, 1)]
    elif kind == "decode":
        passes = [(1, case["context"] + i, 1, 1) for i in range(case["steps"])]
    elif kind == "batch":
        passes = [(1, case["context"] + i, case["seqs"], case["seqs"]) for i in range(case["steps"])]
    elif kind == "turn":
        passes = [(case["tokens"], case["context"], 1, 1)] + [(1, case["context"] + case["tokens"] + i, 1, 1) for i in range(case["steps"])]
    elif kind == "reply":
        passes = [(case["tokens"], 0, 1, 1)] + [(1, case["tokens"] + i, 1, 1) for i in range(case["steps"] - 1)]
    elif kind == "score":
        passes = [(case["context"], 0, 0, 1)] + [(case["tokens"] + i % 3, case["context"], 1, 1) for i in range(case["prompts"])]
    total = [_forward(name, n, start, kv_bytes, logits, rows) for n, start, logits, rows in passes]
    return dict(bytes=sum(b for b, _ in total), flops=sum(f for _, f in total))


def tolerance(case: dict):
    kind = case["kind"]
    if kind in ("decode", "batch", "reply"):
        return {"rel": 0.0, "differ": 0.01}  # token ids, from float32 operands
    if kind == "experts":
        return {"rel": 2e-3}  # half-precision operands, one block
    if kind == "score":
        return {"rel": 3e-3}  # log-probabilities near -11 from logits of half-precision operands
    if kind == "prompt" and case["tokens"] < 16 and not case["chunk"]:
        return {"rel": 1e-3}  # float32 operands, half-precision cache rows
    return {"rel": 1.5e-2}  # half-precision operands through 16 to 32 layers
