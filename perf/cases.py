"""The work that is measured: what a run of reinforcement-learning post-training has this framework do on one GPU.

Four paths, each over packed sequences of many lengths:

* ``train``: one micro-batch of the trainer: ``GPTModel`` forward, the fused policy loss on the response tokens, backward into
  the fp32 gradient buffer. Mixture models replay the experts that the rollout chose, as ``--use-rollout-routing-replay`` does.
* ``score``: log-probs of given responses without gradients (old policy, reference policy, teacher).
* ``prefill``: the rollout engine takes in prompts (``Engine.feed``), fresh or behind a context that is in the cache already.
* ``decode``: one token for each running request (``Engine.feed`` on the captured decode step, sampling included).
* ``fp8``: the four projections of a layer with block-fp8 resident weights, as an engine with ``--sglang-quantization fp8`` runs them.

The models are the ones the launch recipes and the benchmark name, Qwen2.5-0.5B, Qwen3-4B and Qwen3-30B-A3B, with the embedding,
the head and so many of their equal layers that bf16 outputs of two correct programs can still be compared. Weights and tokens are
random. Lengths are spread evenly from ``shortest`` to ``longest`` and then shuffled; multiples of a tile are met only by chance.
"""

import math
import os
import random

import torch

#: width, heads, key heads, head width, feed-forward width, vocabulary, tied head, biased qkv, q / k norms, experts, their width, chosen
MODELS = {
    "qwen2.5-0.5b": dict(h=896, hq=14, hkv=2, d=64, f=4864, v=151936, tied=True, bias=True, qk=False, e=0, fe=0, k=0),
    "qwen3-4b": dict(h=2560, hq=32, hkv=8, d=128, f=9728, v=151936, tied=True, bias=False, qk=True, e=0, fe=0, k=0),
    "qwen3-30b-a3b": dict(h=2048, hq=32, hkv=4, d=128, f=0, v=151936, tied=False, bias=False, qk=True, e=128, fe=768, k=8),
}
EPS, BASE = 1e-6, 1e6
LAYERS = {"qwen2.5-0.5b": (8, 12), "qwen3-4b": (3, 6), "qwen3-30b-a3b": (2, 3)}  # of the trainer's cases, of the engine's


def _case(name, path, model, layers, sequences, shortest, longest, cached=0):
    c = dict(path=path, model=model, layers=layers, sequences=sequences, shortest=shortest, longest=longest, cached=cached)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one short conversation: a first trial of a recipe, the tail of a step; launches and latency count
        _case("train-short", "train", "qwen2.5-0.5b", 8, 1, 397, 397),
        # the micro-batch of the benchmark's step: prompts of 256 tokens, answers of 128 to 1024
        _case("train-batch", "train", "qwen2.5-0.5b", 8, 19, 384, 1280),
        # reasoning traces: one of about eight thousand tokens with a shorter one, the 9216 tokens of the Qwen3-4B recipe
        _case("train-long", "train", "qwen3-4b", 3, 2, 1187, 8011),
        # the mixture model's micro-batch, experts replayed from the rollout
        _case("train-experts", "train", "qwen3-30b-a3b", 2, 6, 700, 2047),
        # log-probs under the reference policy
        _case("score-batch", "score", "qwen2.5-0.5b", 8, 12, 301, 1100),
        # a single chat turn: time to the first token
        _case("prefill-one", "prefill", "qwen2.5-0.5b", 12, 1, 301, 301),
        # a step's prompts as the scheduler packs them, up to its budget of tokens
        _case("prefill-batch", "prefill", "qwen3-4b", 6, 9, 517, 1531),
        # next turns of tool-using conversations: new tokens behind what is cached
        _case("prefill-turns", "prefill", "qwen3-4b", 6, 4, 333, 1400, cached=3100),
        # the benchmark's rollout in full swing
        _case("decode-many", "decode", "qwen2.5-0.5b", 12, 256, 257, 1279),
        # long reasoning rollouts of the Qwen3-4B recipe
        _case("decode-long", "decode", "qwen3-4b", 6, 64, 1025, 5111),
        # the mixture model's rollout near its end: few requests, and their experts
        _case("decode-experts", "decode", "qwen3-30b-a3b", 3, 12, 600, 2400),
        # prompts or a large decode batch of an engine that keeps its weights in block fp8
        _case("fp8-layer", "fp8", "qwen3-4b", 1, 1, 3465, 3465),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """One more case: a path, a model and lengths from the ranges of the listed ones, at most as much work as the largest of its path and model."""
    while True:
        path = rng.choice(["train", "train", "score", "prefill", "prefill", "decode", "decode", "fp8"])
        model = "qwen3-4b" if path == "fp8" else rng.choice(sorted(MODELS))
        most = {"qwen2.5-0.5b": 15800, "qwen3-4b": 9200, "qwen3-30b-a3b": 8200}[model]
        layers, cached = LAYERS[model][path in ("prefill", "decode")], 0
        if path == "fp8":
            tokens = _log(rng, 16, 4000)
            return _case("", path, model, 1, 1, tokens, tokens)
        if path == "decode":
            sequences = _log(rng, 2, 256 if model == "qwen2.5-0.5b" else 64)
            shortest = _log(rng, 200, 2000)
            longest = shortest + _log(rng, 10, 3000)
            if sequences * (shortest + longest) > 390000:
                continue
        else:
            sequences = _log(rng, 1, 20)
            shortest = _log(rng, 200, 4000)
            longest = shortest + (_log(rng, 10, 4000) if sequences > 1 else 0)
            if sequences * (shortest + longest) // 2 > most:
                continue
        if path == "prefill" and rng.random() < 0.4:
            cached = _log(rng, 64, 3100)
            if sequences * cached > 12400:
                continue
        return _case("", path, model, layers, sequences, shortest, longest, cached)


# ------------------------------------------------------------------------------------------------------ sizes
def _lengths(case):
    n, lo, hi = case["sequences"], case["shortest"], case["longest"]
    out = [lo + (hi - lo) * i // max(n - 1, 1) for i in range(n)]
    random.Random(n * 7919 + lo).shuffle(out)
    return out


def _prompt(length):
    """The part of a training sample that carries no loss."""
    return min(256, length // 3)


def _params(m, layers):
    """(weights of the layers that a token is multiplied with, all weights of the layers, of one vocabulary matrix)"""
    attn = m["h"] * m["d"] * (2 * m["hq"] + 2 * m["hkv"])
    if m["e"]:
        return layers * (attn + m["e"] * m["h"] + 3 * m["h"] * m["fe"] * m["k"]), layers * (attn + m["e"] * m["h"] + 3 * m["h"] * m["fe"] * m["e"]), m["h"] * m["v"]
    dense = layers * (attn + 3 * m["h"] * m["f"])
    return dense, dense, m["h"] * m["v"]


def work(case):
    """Each weight and each cached key and value read once, gradients, logits and new keys and values written once; products and attention."""
    m, L, lens = MODELS[case["model"]], case["layers"], _lengths(case)
    active, held, vocab = _params(m, L)
    kv = 4 * m["hkv"] * m["d"] * L  # bytes of a cached token
    if case["path"] == "fp8":
        t = sum(lens)
        return {"bytes": sum(n * k + 2 * t * (n + k) for n, k in _projections(m)), "flops": 2 * t * sum(n * k for n, k in _projections(m))}
    pairs = sum(n * (n + 1) / 2 + n * case["cached"] for n in lens) if case["path"] != "decode" else sum(n + 1 for n in lens)
    attention = 4 * m["hq"] * m["d"] * L * pairs
    tokens = sum(lens) if case["path"] != "decode" else len(lens)
    if case["path"] in ("train", "score"):
        rows = sum(n - _prompt(n) for n in lens)
        matrices = held + vocab * (1 if m["tied"] else 2)
        forward = 2 * active * tokens + 2 * vocab * rows
        if case["path"] == "score":
            return {"bytes": 2 * matrices + 8 * tokens + 4 * rows, "flops": forward + attention}
        return {"bytes": 2 * matrices + 4 * matrices + 8 * tokens + 8 * rows, "flops": 3 * forward + 3.5 * attention}
    if m["e"]:
        one = 3 * m["h"] * m["fe"]
        held -= L * one * (m["e"] - min(m["e"], tokens * m["k"]))
    read = kv * (sum(lens) if case["path"] == "decode" else case["cached"] * len(lens))
    return {"bytes": 2 * held + 2 * vocab + read + kv * tokens + 4 * m["v"] * len(lens), "flops": 2 * active * tokens + 2 * vocab * len(lens) + attention}


def tolerance(case):
    """bf16 operands, activations and residual stream. Through all the layers of a case two orders of the same sums come to 0.5 to 2 %
    apart (a product that is split along K adds its parts in any order, and so shows it by itself); one product rounds its output once."""
    if case["path"] == "fp8":
        return {"rel": 0.01, "max": 0.1}
    return {"rel": 0.03, "max": 0.9}


# ------------------------------------------------------------------------------------------------------ inputs
def _names(m, layers):
    """(name, shape, how it is drawn) of every weight, in the order of the gradient buffer."""
    h, d = m["h"], m["d"]
    rows, std, out = (m["hq"] + 2 * m["hkv"]) * d, 0.02, 0.02 / math.sqrt(2 * layers)
    yield "embedding.word_embeddings.weight", (m["v"], h), std
    for i in range(layers):
        a, f = f"decoder.layers.{i}.self_attention.", f"decoder.layers.{i}.mlp."
        yield a + "linear_qkv.weight", (rows, h), std
        yield a + "linear_qkv.layer_norm_weight", (h,), 1.0
        if m["bias"]:
            yield a + "linear_qkv.bias", (rows,), std
        if m["qk"]:
            yield a + "q_layernorm.weight", (d,), 1.0
            yield a + "k_layernorm.weight", (d,), 1.0
        yield a + "linear_proj.weight", (h, m["hq"] * d), out
        if m["e"]:
            yield f + "pre_mlp_layernorm.weight", (h,), 1.0
            yield f + "router.weight", (m["e"], h), std
            for e in range(m["e"]):
                yield f + f"experts.linear_fc1.weight{e}", (2 * m["fe"], h), std
            for e in range(m["e"]):
                yield f + f"experts.linear_fc2.weight{e}", (h, m["fe"]), out
        else:
            yield f + "linear_fc1.weight", (2 * m["f"], h), std
            yield f + "linear_fc1.layer_norm_weight", (h,), 1.0
            yield f + "linear_fc2.weight", (h, m["f"]), out
    yield "decoder.final_layernorm.weight", (h,), 3.0  # logits as spread out as a trained model's
    if not m["tied"]:
        yield "output_layer.weight", (m["v"], h), std


def _weights(case, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    out = {}
    for name, shape, draw_ in _names(MODELS[case["model"]], case["layers"]):
        t = torch.empty(shape, dtype=torch.bfloat16, device="cuda")
        out[name] = t.normal_(draw_, 0.1 * draw_, generator=g) if draw_ >= 1 else t.normal_(0.0, draw_, generator=g)
    return out


def _projections(m):
    """(rows, columns) of a dense layer's fused matrices."""
    return [((m["hq"] + 2 * m["hkv"]) * m["d"], m["h"]), (m["h"], m["hq"] * m["d"]), (2 * m["f"], m["h"]), (m["h"], m["f"])]


def _quantised_inputs(case, seed):
    """Activations in bf16, some columns ten times as large as the others, and the matrices before they are quantised."""
    g = torch.Generator("cuda").manual_seed(seed)
    bf16 = lambda n, k, std: torch.empty(n, k, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=g)  # noqa: E731
    out = []
    for n, k in _projections(MODELS[case["model"]]):
        x = bf16(sum(_lengths(case)), k, 1.0)
        x[:, ::97] *= 10
        out.append((x, bf16(n, k, 0.02)))
    return out


def _tokens(case, seed):
    """Per sequence: cached context, then the new tokens (decode: the context, then one token)."""
    r = random.Random(seed)
    extra = 1 if case["path"] == "decode" else case["cached"]
    return [[r.randrange(MODELS[case["model"]]["v"]) for _ in range(n + extra)] for n in _lengths(case)]


def _samples(case, seed):
    """What the trainer gets besides the tokens: loss weight and advantage of every response token, experts chosen by the rollout."""
    m, lens = MODELS[case["model"]], _lengths(case)
    g = torch.Generator("cuda").manual_seed(seed + 1)
    adv = torch.empty(len(lens), device="cuda").normal_(0.3, 1.0, generator=g)
    n = torch.tensor([x - _prompt(x) for x in lens], device="cuda")
    rows, starts = [], 0
    for x in lens:
        rows.append(torch.arange(starts + _prompt(x) - 1, starts + x - 1, device="cuda"))
        starts += x
    experts = None
    if m["e"]:
        score = torch.empty(sum(lens), case["layers"], m["e"], device="cuda").normal_(generator=g)
        experts = (score + 0.5 * torch.linspace(-1, 1, m["e"], device="cuda")).topk(m["k"], dim=-1).indices  # some are asked for more often
    return dict(weight=(1.0 / (n * len(lens))).repeat_interleave(n), advantage=adv.repeat_interleave(n), rows=torch.cat(rows), experts=experts)


def _targets(tokens):
    return [t for s in tokens for t in s[_prompt(len(s)) :]]


# ------------------------------------------------------------------------------------------------------ the framework's side
def _config(case):
    from slime_b200.models.config import get_preset

    cfg = get_preset(case["model"])
    cfg.num_layers = case["layers"]
    return cfg


def _trainer(case, seed):
    from slime_b200.backends.train.buffers import FlatBuffer
    from slime_b200.models.gpt import GPTModel, PackedSeqParams
    from slime_b200.parallel import state as mpu

    if not mpu.model_parallel_is_initialized():
        mpu.initialize_model_parallel()
    model = GPTModel(_config(case), device="cuda", seed=seed)
    held = dict(model.named_parameters())
    weights = _weights(case, seed)
    assert set(held) == set(weights)
    for name, w in weights.items():
        held[name].data.copy_(w)
    names = list(weights)
    del weights
    grads = FlatBuffer([held[n] for n in names], names, None, 1, 0, torch.device("cuda")) if case["path"] == "train" else None
    tokens, lens = _tokens(case, seed), _lengths(case)
    cu = torch.tensor([0] + lens).cumsum(0).to("cuda", torch.int32)
    positions = torch.cat([torch.arange(n) for n in lens]).to("cuda", torch.int32)
    ids = torch.tensor([t for s in tokens for t in s], device="cuda")
    targets = torch.tensor(_targets(tokens), dtype=torch.int32, device="cuda")
    return dict(_samples(case, seed), case=case, model=model, grads=grads, packed=lambda: PackedSeqParams(cu, max(lens)), ids=ids, positions=positions, targets=targets)


def _engine(case, seed):
    from slime_b200.engine.engine import Engine
    from slime_b200.engine.server_args import ServerArgs

    m, lens, tokens = MODELS[case["model"]], _lengths(case), _tokens(case, seed)
    held = max(len(t) for t in tokens)
    args = ServerArgs(page_size=64, context_length=held + 64, max_running_requests=len(lens), disable_radix_cache=True)
    engine = Engine(_config(case), args, device="cuda", num_pages=sum(-(-len(t) // 64) for t in tokens) + 2)
    q, kv = m["hq"] * m["d"], m["hkv"] * m["d"]
    parts = []  # under the names of a checkpoint
    for name, w in _weights(case, seed).items():
        own = name.split(".")
        p = f"model.layers.{own[2]}." if own[1] == "layers" else ""
        if name == "embedding.word_embeddings.weight":
            parts.append(("model.embed_tokens.weight", w))
        elif name == "output_layer.weight":
            parts.append(("lm_head.weight", w))
        elif name == "decoder.final_layernorm.weight":
            parts.append(("model.norm.weight", w))
        elif "linear_qkv." in name and "norm" not in name:
            parts += [(f"{p}self_attn.{x}_proj.{own[-1]}", t) for x, t in zip("qkv", w.split([q, kv, kv]))]
        elif "experts" in name:
            e = own[-1][len("weight") :]
            two = [("gate", w[: m["fe"]]), ("up", w[m["fe"] :])] if "linear_fc1" in name else [("down", w)]
            parts += [(f"{p}mlp.experts.{e}.{x}_proj.weight", t) for x, t in two]
        elif name.endswith("linear_fc1.weight"):
            parts += [(f"{p}mlp.{x}_proj.weight", t) for x, t in zip(("gate", "up"), w.split(m["f"]))]
        else:
            table = {"linear_qkv.layer_norm_weight": "input_layernorm", "q_layernorm.weight": "self_attn.q_norm", "k_layernorm.weight": "self_attn.k_norm",
                     "linear_proj.weight": "self_attn.o_proj", "linear_fc1.layer_norm_weight": "post_attention_layernorm", "linear_fc2.weight": "mlp.down_proj",
                     "pre_mlp_layernorm.weight": "post_attention_layernorm", "router.weight": "mlp.gate"}  # fmt: skip
            parts.append((f"{p}{table['.'.join(own[-2:])]}.weight", w))
    assert not engine.update_weights(parts)
    del parts
    state = dict(case=case, engine=engine, tokens=tokens, requests=None)
    kept = [t[:-1] if case["path"] == "decode" else t[: case["cached"]] for t in tokens]
    if kept[0]:
        state["requests"] = [engine.open_stream(str(i)) for i in range(len(tokens))]
        batch = []
        for r, k in zip(state["requests"], kept):
            if sum(len(t) for _, t, _ in batch) + len(k) > 16384:
                engine.feed(batch)
                batch = []
            batch.append((r, k, []))
        engine.feed(batch)
        if case["path"] == "decode":
            run(state)  # the decode step is captured once, when a server starts
    return state


def _quantised(case, seed):
    from slime_b200.engine.quant import Fp8Weight

    pairs = []
    for x, w in _quantised_inputs(case, seed):
        held = Fp8Weight(*w.shape, device="cuda")
        held.load_rows(0, w)
        pairs.append((x, held))
    return dict(case=case, pairs=pairs)


def prepare(case, seed):
    if case["path"] == "fp8":
        return _quantised(case, seed)
    return _trainer(case, seed) if case["path"] in ("train", "score") else _engine(case, seed)


def run(state):
    path = state["case"]["path"]
    if path == "train":
        return _train(state)
    if path == "score":
        return _score(state)
    if path == "fp8":
        from slime_b200.engine import quant

        return [quant.linear(x, w) for x, w in state["pairs"]]
    return _feed(state)


def _replay(s):
    """The experts that the rollout chose go to the routers, in the order in which the pass will ask for them."""
    from slime_b200.utils import routing_replay

    if s["experts"] is None:
        return
    os.environ["ENABLE_ROUTING_REPLAY"] = "1"
    routing_replay.set_stage("replay_forward")
    for layer in s["model"].decoder.layers:
        layer.mlp.router.replay.clear()
        layer.mlp.router.replay.top_indices_list.append(s["experts"][:, layer.layer_number])


def _train(s):
    from slime_b200.backends.train import fused_loss

    model, grads = s["model"], s["grads"]
    grads.zero_grad()
    _replay(s)
    hidden = model(s["ids"], s["positions"], packed_seq_params=s["packed"](), return_hidden=True)
    loss, logp, entropy, _ = fused_loss.fused_policy_loss(hidden.index_select(0, s["rows"]), model.output_weight(), s["targets"], None, s["advantage"], s["weight"],
                                                          eps_clip=0.2, eps_clip_high=0.28)  # fmt: skip
    loss.backward()
    grads.fold_autograd_grads()
    return {"loss": loss.detach(), "logp": logp, "entropy": entropy, "gradients": grads.grad_data}


@torch.no_grad()
def _score(s):
    from slime_b200.backends.train import fused_loss

    model = s["model"]
    _replay(s)
    hidden = model(s["ids"], s["positions"], packed_seq_params=s["packed"](), return_hidden=True)
    logp, _ = fused_loss.logprob_entropy_rows(hidden.index_select(0, s["rows"]), model.output_weight(), s["targets"], with_entropy=False)
    return {"logp": logp}


def _feed(s):
    engine, tokens, kept = s["engine"], s["tokens"], s["requests"]
    requests = kept or [engine.open_stream(str(i)) for i in range(len(tokens))]
    before = [r.num_computed for r in requests]
    logits = engine.feed([(r, t[n:], [len(t) - n - 1]) for r, t, n in zip(requests, tokens, before)])
    for r, n in zip(requests, before):
        if kept:  # another continuation of the same context may follow
            r.num_computed = n
            del r.input_ids[n:]
        else:
            engine.close_stream(r)
    return {"logits": logits}


# ------------------------------------------------------------------------------------------------------ the same in 64 bits
def _norm(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w


def _rotate(x):
    """x: [n, heads, d], positions 0 .. n - 1"""
    half = x.shape[-1] // 2
    angle = torch.arange(x.shape[0], device=x.device, dtype=torch.float64)[:, None] * BASE ** (-torch.arange(half, device=x.device, dtype=torch.float64) / half)
    c, s = angle.cos()[:, None], angle.sin()[:, None]
    return torch.cat([x[..., :half] * c - x[..., half:] * s, x[..., half:] * c + x[..., :half] * s], -1)


def _attend(q, k, v):
    """One sequence, one key head: q [n, g, d], k and v [n, d]; causal."""
    n = q.shape[0]
    out = []
    for a in range(0, n, 2048):  # rows of a part see the keys up to its end
        b = min(n, a + 2048)
        z = torch.einsum("igd,jd->gij", q[a:b], k[:b]) / math.sqrt(q.shape[-1])
        z = z.masked_fill(torch.ones(b - a, b, dtype=torch.bool, device=q.device).triu(a + 1), -math.inf)
        out.append(torch.einsum("gij,jd->igd", z.softmax(-1), v[:b]))
    return torch.cat(out)


def _layer(x, w, i, m, lens, experts):
    a, f = f"decoder.layers.{i}.self_attention.", f"decoder.layers.{i}.mlp."
    t, d, g = x.shape[0], m["d"], m["hq"] // m["hkv"]
    y = _norm(x, w[a + "linear_qkv.layer_norm_weight"]) @ w[a + "linear_qkv.weight"].t()
    y = y + w[a + "linear_qkv.bias"] if m["bias"] else y
    q, k, v = y.view(t, -1, d).split([m["hq"], m["hkv"], m["hkv"]], 1)
    if m["qk"]:
        q, k = _norm(q, w[a + "q_layernorm.weight"]), _norm(k, w[a + "k_layernorm.weight"])
    out, at = [], 0
    for n in lens:
        qs, ks = _rotate(q[at : at + n]), _rotate(k[at : at + n])
        out.append(torch.cat([torch.utils.checkpoint.checkpoint(_attend, qs[:, j * g : (j + 1) * g], ks[:, j], v[at : at + n, j], use_reentrant=False)
                              for j in range(m["hkv"])], 1))  # fmt: skip
        at += n
    x = x + torch.cat(out).reshape(t, -1) @ w[a + "linear_proj.weight"].t()
    glu = lambda y, up, down: (lambda z: torch.nn.functional.silu(z[:, : z.shape[1] // 2]) * z[:, z.shape[1] // 2 :])(y @ up.t()) @ down.t()  # noqa: E731
    if not m["e"]:
        y = _norm(x, w[f + "linear_fc1.layer_norm_weight"])
        return x + torch.cat([glu(p, w[f + "linear_fc1.weight"], w[f + "linear_fc2.weight"]) for p in y.split(16384)])
    y = _norm(x, w[f + "pre_mlp_layernorm.weight"])
    score = y @ w[f + "router.weight"].t()
    chosen = score.topk(m["k"], dim=-1).indices if experts is None else experts[:, i]
    share = score.gather(1, chosen).softmax(-1)
    z = torch.zeros_like(x)
    for e in range(m["e"]):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        z = z.index_add(0, rows, glu(y[rows], w[f + f"experts.linear_fc1.weight{e}"], w[f + f"experts.linear_fc2.weight{e}"]) * share[rows, place][:, None])
    return x + z


def _hidden(case, w, tokens, experts=None):
    m, lens = MODELS[case["model"]], [len(t) for t in tokens]
    x = w["embedding.word_embeddings.weight"][torch.tensor([t for s in tokens for t in s], device="cuda")]
    for i in range(case["layers"]):
        x = torch.utils.checkpoint.checkpoint(_layer, x, w, i, m, lens, experts, use_reentrant=False)
    return _norm(x, w["decoder.final_layernorm.weight"])


def _scored(h, head, targets):
    z = h @ head.t()
    lse = z.logsumexp(-1)
    return z.gather(1, targets[:, None])[:, 0] - lse, lse - ((z - lse[:, None]).exp() * z).sum(-1)


def _blocks(x, rows):
    """x rounded to e4m3 in blocks of ``rows`` x 128 whose largest value becomes 448."""
    n, k = x.shape
    pad = torch.nn.functional.pad(x.float(), (0, 0, 0, -n % rows)).view(-1, rows, k // 128, 128)
    scale = pad.abs().amax((1, 3), keepdim=True) / 448
    return ((pad / scale).to(torch.float8_e4m3fn).double() * scale.double()).reshape(-1, k)[:n]


def exact(case, seed):
    if case["path"] == "fp8":  # of the values that the quantised operands have
        out = []
        for x, w in _quantised_inputs(case, seed):
            out.append(_blocks(x, 1) @ _blocks(w, 128).t())
        return out
    train = case["path"] == "train"
    w = {n: t.double().requires_grad_(train) for n, t in _weights(case, seed).items()}
    head = w.get("output_layer.weight", w["embedding.word_embeddings.weight"])
    tokens = _tokens(case, seed)
    with torch.set_grad_enabled(train):
        if case["path"] in ("prefill", "decode"):
            out = []
            for a in range(0, len(tokens), 16):  # a few sequences at a time
                part = tokens[a : a + 16]
                last = torch.tensor([len(t) for t in part], device="cuda").cumsum(0) - 1
                out.append(_hidden(case, w, part)[last] @ head.t())
            return {"logits": torch.cat(out)}
        s = _samples(case, seed)
        h = _hidden(case, w, tokens, s["experts"])[s["rows"]]
        targets = torch.tensor(_targets(tokens), device="cuda")
        parts = [torch.utils.checkpoint.checkpoint(_scored, p, head, t, use_reentrant=False) for p, t in zip(h.split(1024), targets.split(1024))]
        logp, entropy = (torch.cat(x) for x in zip(*parts))
        if not train:
            return {"logp": logp}
        # the ratio to the policy itself is one, and so nothing is clipped
        loss = -(s["weight"].double() * s["advantage"].double() * (logp - logp.detach()).exp()).sum()
        loss.backward()
    pad = lambda t: torch.nn.functional.pad(t.reshape(-1), (0, -t.numel() % 128))  # noqa: E731
    return {"loss": loss.detach(), "logp": logp.detach(), "entropy": entropy.detach(), "gradients": torch.cat([pad(t.grad) for t in w.values()])}
