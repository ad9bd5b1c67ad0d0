"""Workloads of the GRPO loop: what a training run asks of the framework, at the sizes of its benchmark configurations.

A step of the loop samples completions (prefill of the prompts, one decode step and one draw per token), scores them and
updates the adapters (forward and backward of a micro-batch).  Every case is one of these passes on a slice of a decoder:
the width, heads, feed-forward, window and expert sizes of a configuration with fewer layers and a vocabulary that shrinks
with them, so that the head keeps about the share of a pass that it has in the whole model.

    train    ``LmPolicy.token_logprobs`` with gradients, the GRPO loss, its backward: log-probs and every adapter gradient
    score    ``LmPolicy.token_logprobs_detached``: the pass over a frozen reference for the KL term
    prefill  a decoder's ``prefill`` of right-padded prompts: last logits and the filled caches
    decode   one token for every row, replayed from a CUDA graph as a rollout replays it: logits and recurrent state
    sample   one top-p draw for every row: tokens and their log-probs

Weights and inputs are random, drawn on the device from the seed.  ``exact`` restates every pass in float64.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

PAGE = 64
DEPTH = 64          # layers of the whole models, which scales what one layer adds to the stream


# ----------------------------------------------------------------------------------------------------------- the cases
def _dense(width=4096, heads=32, kv=8, dim=128, ff=12288, vocab=32768, layers=4, lora=16, remat=False):
    return dict(family="dense", width=width, heads=heads, kv=kv, dim=dim, ff=ff, vocab=vocab, layers=layers, lora=lora, remat=remat)


def _gemma(width=5376, heads=32, kv=16, dim=128, ff=21504, vocab=32768, window=1024, every=3, layers=3, lora=16, remat=True):
    return dict(family="gemma", width=width, heads=heads, kv=kv, dim=dim, ff=ff, vocab=vocab, window=window, every=every,
                layers=layers, lora=lora, remat=remat)


def _hybrid(width=5120, heads=24, kv=4, dim=256, ff=17408, vocab=32768, kh=16, vh=48, layers=4, lora=32, gdn="io", experts=0, top=0,
            remat=True):
    """``experts``: routed experts of width ``ff`` beside one shared expert of the same width (0: a dense feed-forward)."""
    return dict(family="hybrid", width=width, heads=heads, kv=kv, dim=dim, ff=ff, vocab=vocab, kh=kh, vh=vh, layers=layers, lora=lora,
                gdn=gdn, experts=experts, top=top, remat=remat)


def _moe(width=2048, heads=16, kv=2, dim=256, ff=768, kh=16, vh=16, experts=128, top=8, lora=8, **kw):
    return _hybrid(width=width, heads=heads, kv=kv, dim=dim, ff=ff, kh=kh, vh=vh, experts=experts, top=top, lora=lora, gdn="", **kw)


def listed():
    return [
        # update of the headline configuration (8B-class dense decoder, LoRA on all projections): one micro-batch of 8 rows
        dict(name="train dense", kind="train", **_dense(), prompts=1, group=8, lo=400, hi=400, new=1024),
        # update of a small model in a few short rows of odd lengths: launches and host work count
        dict(name="train dense small", kind="train", **_dense(1024, 8, 2, 128, 3072), prompts=3, group=1, lo=61, hi=97, new=203),
        # update of a sliding-window decoder (5:1 there, 2:1 in this slice) with rematerialisation, two rows
        dict(name="train window", kind="train", **_gemma(), prompts=1, group=2, lo=256, hi=256, new=2048),
        # update of a 27B-class hybrid on one long completion, rematerialised
        dict(name="train hybrid long", kind="train", **_hybrid(), prompts=1, group=1, lo=1024, hi=1024, new=4096),
        # update of the hybrid mixture of experts, four rows
        dict(name="train hybrid moe", kind="train", **_moe(), prompts=2, group=2, lo=512, hi=512, new=1024),
        # KL reference pass of the hybrid over ragged rows
        dict(name="score hybrid", kind="score", **_hybrid(), prompts=2, group=2, lo=501, hi=1024, new=1024),
        # prompts of a rollout of the headline configuration: 16 ragged prompts, groups of 8 behind each
        dict(name="prefill dense", kind="prefill", **_dense(), prompts=16, group=8, lo=128, hi=512),
        # decode step of that rollout, half way: 16 groups of 8 that share their prompt
        dict(name="decode dense rollout", kind="decode", **_dense(), prompts=16, group=8, lo=128, hi=512, done=512),
        # a single sequence of a small model: latency
        dict(name="decode dense one", kind="decode", **_dense(1024, 8, 2, 128, 3072, layers=8), prompts=1, group=1, lo=333, hi=333, done=444),
        # decode step of the sliding-window decoder past its window
        dict(name="decode window", kind="decode", **_gemma(every=6, layers=6), prompts=8, group=8, lo=256, hi=256, done=1300),
        # decode step of the hybrid mixture of experts: 128 rows, recurrent states and one cache in four layers
        dict(name="decode hybrid moe", kind="decode", **_moe(), prompts=16, group=8, lo=512, hi=512, done=512),
        # the draw of a rollout over the headline configuration's whole vocabulary
        dict(name="sample", kind="sample", family="none", rows=128, vocab=151936, dtype="bf16", top_p=0.95, temperature=1.0),
    ]


def _log(rng, lo, hi, step=1):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step) * step)))


def draw(rng):
    """One more case: kinds and families as often as they are listed, sizes over their whole range."""
    kind = rng.choice(["train", "train", "train", "score", "prefill", "decode", "decode", "decode", "sample"])
    if kind == "sample":
        return dict(kind=kind, family="none", rows=_log(rng, 1, 256), vocab=_log(rng, 8192, 262144, 64), dtype=rng.choice(["bf16", "f32"]),
                    top_p=rng.choice([0.95, 0.9, 0.8, 1.0]), temperature=rng.choice([1.0, 0.7, 1.2]))
    family = rng.choice(["dense", "dense", "gemma", "hybrid", "moe"])
    if kind == "prefill" and family in ("hybrid", "moe"):
        family = "dense"
    if kind == "score" and family == "gemma":
        family = "hybrid"
    dim = rng.choice([128, 128, 64]) if family == "dense" else 128 if family == "gemma" else 256
    kv = rng.choice([2, 4, 8] if dim < 256 else [2, 4])
    heads = kv * rng.choice([2, 4, 8] if family in ("hybrid", "moe") else [2, 4])
    layers = rng.choice([2, 3, 4])
    if family == "moe":
        ff, kh = _log(rng, 256, 1024, 64), rng.choice([8, 16])
        m = _moe(_log(rng, 1024, 3072, 128), heads, kv, dim, ff, kh, kh * rng.choice([1, 2]), rng.choice([32, 64, 128]), rng.choice([4, 6, 8]), layers=4)
    else:
        width = _log(rng, 1024, 5120, 128)
        ff = _log(rng, 2 * width, min(4 * width, 17408), 128)
        if family == "dense":
            m = _dense(width, heads, kv, dim, ff, rng.choice([32000, 32768, 49152]), layers, rng.choice([8, 16, 32]), rng.random() < 0.3)
        elif family == "gemma":
            m = _gemma(width, heads, kv, dim, ff, 32768, rng.choice([512, 1024]), 3, layers)
        else:
            kh = rng.choice([8, 16])
            m = _hybrid(width, heads, kv, dim, ff, 32768, kh, kh * rng.choice([1, 2, 3]), 4, rng.choice([8, 16, 32]))
    if kind in ("train", "score"):
        rows = _log(rng, 1, 8)
        group = rng.choice([g for g in (1, 2, 4, 8) if rows % g == 0])
        hi = _log(rng, 32, 512)
        new = _log(rng, 64, min(4096, 8192 // rows))
        return dict(kind=kind, **m, prompts=rows // group, group=group, lo=max(1, hi // 2), hi=hi, new=new)
    if kind == "prefill":
        hi = _log(rng, 16, 1024)
        return dict(kind=kind, **m, prompts=_log(rng, 1, max(1, min(16, 8192 // hi))), group=rng.choice([1, 4, 8]), lo=max(1, hi // 4), hi=hi)
    group = rng.choice([1, 4, 8])
    hi = _log(rng, 32, 512)
    return dict(kind=kind, **m, prompts=_log(rng, 1, 128 // group), group=group, lo=max(1, hi // 2), hi=hi, done=_log(rng, 16, 700))


# ------------------------------------------------------------------------------------------------------------- weights
def _types(c):
    if c["family"] == "gemma":
        return ["full_attention" if i % c["every"] == c["every"] - 1 else "sliding_attention" for i in range(c["layers"])]
    if c["family"] == "hybrid":
        return ["full_attention" if i % 4 == 3 else "linear_attention" for i in range(c["layers"])]
    return ["full_attention"] * c["layers"]


def _projections(c, kind):
    """``{projection: (input width, {part: output width}, adapted parts)}`` of one layer, in the fused order."""
    W, D, hq, hkv, ff = c["width"], c["dim"], c["heads"], c["kv"], c["ff"]
    if c["family"] == "hybrid":
        if kind == "full_attention":
            p = {"inp": (W, {"q": 2 * hq * D, "k": hkv * D, "v": hkv * D}, "q k v"), "out": (hq * D, {"o": W}, "o")}
        else:
            kd, vd = c["kh"] * 128, c["vh"] * 128
            p = {"inp": (W, {"qkv": 2 * kd + vd, "z": vd, "b": c["vh"], "a": c["vh"]}, "qkv z" if "i" in c["gdn"] else ""),
                 "out": (vd, {"out": W}, "out" if "o" in c["gdn"] else "")}
        mlp = "shared" if c["experts"] else "mlp"
        p[f"{mlp}.gate_up"] = (W, {"gate": ff, "up": ff}, "gate up")
        p[f"{mlp}.down"] = (ff, {"down": W}, "down")
        return p
    parts = {"q": hq * D, "k": hkv * D, "v": hkv * D}
    if c["family"] == "gemma" and kind == "full_attention":
        del parts["v"]          # keys are the values there
    return {"qkv": (W, parts, "q k v"), "o": (hq * D, {"o": W}, "o"), "gate_up": (W, {"gate": ff, "up": ff}, "gate up"),
            "down": (ff, {"down": W}, "down")}


def _norms(c, kind):
    """``{norm: (width, mean of its stored weight)}``; scores of unit keys and queries stay near one in size."""
    W, D = c["width"], c["dim"]
    if c["family"] == "gemma":
        return {"input_norm": (W, 1.0), "post_attn_norm": (W, 1.0), "pre_ffn_norm": (W, 1.0), "post_ffn_norm": (W, 1.0),
                "q_norm": (D, D ** -0.5), "k_norm": (D, 1.0)}
    n = {"input_norm": (W, 0.0 if c["family"] == "hybrid" else 1.0)}
    n["post_norm"] = n["input_norm"]
    if kind == "full_attention":
        n["q_norm"] = n["k_norm"] = (D, n["input_norm"][1])
    else:
        n["gdn_norm"] = (128, 1.0)
    return n


def _weights(c, seed):
    """``{name: tensor}``: bf16 weights, float32 adapters and recurrence constants, drawn from the seed.  As in a trained
    decoder the stream carries more than one layer adds to it (unit embedding rows, projections back onto the stream
    scaled down) and the router decides (the least chosen expert has a small weight)."""
    g = torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)
    rnd = lambda std, *shape: torch.randn(shape, generator=g, device="cuda") * std  # noqa: E731
    b16 = lambda std, *shape: rnd(std, *shape).bfloat16()  # noqa: E731
    W = c["width"]
    tied = c["family"] == "gemma"
    w = {"embed": b16(0.02 if tied else 1.0, c["vocab"], W), "final_norm": (rnd(0.1, W) + (0.0 if c["family"] == "hybrid" else 1.0)).bfloat16()}
    if not tied:
        w["head"] = b16(0.02, c["vocab"], W)
    back = 0.02 * (2 * DEPTH) ** -0.5
    train = c["kind"] == "train"
    for i, kind in enumerate(_types(c)):
        for name, (n, mean) in _norms(c, kind).items():
            w[f"{i}.{name}"] = (rnd(0.1 * (mean or 1.0), n) + mean).bfloat16()
        for name, (inn, parts, adapted) in _projections(c, kind).items():
            w[f"{i}.{name}"] = b16(back if name.split(".")[-1] in ("o", "out", "down") else 0.02, sum(parts.values()), inn)
            for part in parts:
                if train and part in adapted.split():
                    w[f"{i}.{name}.{part}.A"] = rnd(0.02, c["lora"], inn)
                    w[f"{i}.{name}.{part}.B"] = rnd(0.01, parts[part], c["lora"])
        if kind == "linear_attention":
            w[f"{i}.conv_w"] = b16(0.3, (2 * c["kh"] + c["vh"]) * 128, 4)
            w[f"{i}.A_log"] = torch.log(torch.rand(c["vh"], generator=g, device="cuda") * 15 + 1)
            w[f"{i}.dt_bias"] = rnd(0.5, c["vh"]) - 2.0
        if c["family"] == "hybrid" and c["experts"]:
            E, ff = c["experts"], c["ff"]
            w[f"{i}.router"] = b16(4 * W ** -0.5, E, W)
            w[f"{i}.experts_gate_up"] = b16(0.02, E, 2 * ff, W)
            w[f"{i}.experts_down"] = b16(back, E, W, ff)
            w[f"{i}.shared_gate"] = b16(0.02, 1, W)
    return w


def _resolve(obj, path):
    for p in path.split("."):
        obj = getattr(obj, p)
    return obj


def _model(c, w):
    """The framework's model of a case with the weights ``w``; ``{parameter name: parameter}`` of its adapters."""
    from ferrl_b200.models import DenseGradModel, DenseSpec, LoraSpec
    length = (c["hi"] + c.get("new", c.get("done", 0)) + 127) // 128 * 128 + 128
    lora = LoraSpec(c["lora"], 2.0 * c["lora"]) if c["kind"] == "train" else None
    kw = dict(dtype=torch.bfloat16, device="cuda", remat=c["remat"])
    if c["family"] == "dense":
        m = DenseGradModel(DenseSpec(c["vocab"], c["width"], c["layers"], c["heads"], c["kv"], c["dim"], c["ff"],
                                     max_position_embeddings=length), lora, **kw)
    elif c["family"] == "gemma":
        from ferrl_b200.models.gemma4 import Gemma4GradModel, Gemma4Spec
        m = Gemma4GradModel(Gemma4Spec(c["vocab"], c["width"], c["layers"], c["heads"], c["kv"], c["dim"], c["dim"], c["kv"], c["ff"],
                                       _types(c), c["window"], max_position_embeddings=length), lora, keep_transpose=False, **kw)
    else:
        from ferrl_b200.models.qwen35 import MoeDims, Qwen35GradModel, Qwen35LoraTargets, Qwen35Spec
        moe = MoeDims(c["experts"], c["top"], c["ff"], c["ff"]) if c["experts"] else None
        m = Qwen35GradModel(Qwen35Spec(c["vocab"], c["width"], c["layers"], c["heads"], c["kv"], c["dim"], c["ff"], _types(c),
                                       max_position_embeddings=length, tie_word_embeddings=False, lin_k_heads=c["kh"], lin_v_heads=c["vh"], moe=moe), lora,
                            Qwen35LoraTargets("qkvo", "gud", c["gdn"]), **dict(kw, **({} if moe else {"keep_transpose": False})))
    params = {}
    with torch.no_grad():
        m.embed.copy_(w["embed"])
        m.final_norm.copy_(w["final_norm"])
        if "head" in w:
            m.lm_head.copy_(w["head"])
        for i, kind in enumerate(_types(c)):
            layer = m.layers[i]
            mine = _projections(c, kind)
            for name in mine:
                p = _resolve(layer, name)
                p.set_weight(w[f"{i}.{name}"])
                for j, k in enumerate(p.adapted_idx if lora else ()):
                    for letter, bank in (("A", p.lora_A), ("B", p.lora_B)):
                        key = f"{i}.{name}.{p.names[k]}.{letter}"
                        bank[j].copy_(w[key])
                        params[key] = bank[j]
            for key, t in w.items():
                if key.startswith(f"{i}.") and key.count(".") == 1 and key.split(".")[1] not in mine:
                    getattr(layer, key.split(".")[1]).copy_(t)
        m.refresh_head()
    return m, params


# -------------------------------------------------------------------------------------------------------------- inputs
def _spread(lo, hi, n):
    """``n`` lengths from ``hi`` down to ``lo``."""
    return [hi - (hi - lo) * i // max(1, n - 1) for i in range(n)]


def _rng(c, seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * seed + 29)


def _ids(c, g, *shape):
    return torch.randint(0, c["vocab"], shape, generator=g, device="cuda")


def _rows(c, seed):
    """Completions of a scoring pass: ``(token ids per prompt on the host, prompt lengths, advantages, mask)``."""
    g = _rng(c, seed)
    lens, G, N = _spread(c["lo"], c["hi"], c["prompts"]), c["group"], c["new"]
    toks = [torch.cat([_ids(c, g, 1, L).expand(G, L), _ids(c, g, G, N)], 1).cpu() for L in lens]
    R = G * len(lens)
    adv = torch.randn(R, generator=g, device="cuda")
    done = torch.randint(N // 4, N + 1, (R, 1), generator=g, device="cuda")
    mask = (torch.arange(N, device="cuda")[None, :] < done).float()
    return toks, lens, adv, mask


def _cache(c, seed):
    """A decode step in the middle of a rollout: prompt lengths and cached lengths of the rows, tokens to feed, and the
    cached keys, values and states of every layer (rows of a group share their prompt's keys and values)."""
    g = _rng(c, seed)
    P, G = c["prompts"], c["group"]
    B = P * G
    lens = torch.tensor(_spread(c["lo"], c["hi"], P), device="cuda")
    kv_len = lens.repeat_interleave(G) + c["done"]
    top = int(c["hi"] + c["done"])
    tokens = _ids(c, g, B)
    layers = []
    for kind in _types(c):
        if kind == "linear_attention":
            layers.append((torch.randn(B, (2 * c["kh"] + c["vh"]) * 128, 3, generator=g, device="cuda").bfloat16(),
                           torch.randn(B, c["vh"], 128, 128, generator=g, device="cuda") * 0.1))
            continue
        # a full window is a ring of slots in any order
        slots = min(top, c["window"]) if kind == "sliding_attention" else top
        kv = []
        for _ in range(2):
            x = torch.randn(B, slots, c["kv"], c["dim"], generator=g, device="cuda").bfloat16()
            if kind != "sliding_attention":
                x = x.view(P, G, slots, c["kv"], c["dim"])
                shared = torch.arange(slots, device="cuda")[None, None, :, None, None] < lens.view(P, 1, 1, 1, 1)
                x = torch.where(shared, x[:, :1], x).reshape(B, slots, c["kv"], c["dim"])
            kv.append(x)
        layers.append(tuple(kv))
    return lens, kv_len.int(), tokens, layers


# ------------------------------------------------------------------------------------------------------------- prepare
def _prepare_rows(c, seed):
    from ferrl_b200.lm_policy import LmPolicy
    from ferrl_b200.policy import Rollout
    from ferrl_b200.sampler import GrpoSampler
    model, params = _model(c, _weights(c, seed))
    toks, lens, adv, mask = _rows(c, seed)
    rollouts = [Rollout.rectangular(t, L) for t, L in zip(toks, lens)]
    s = SimpleNamespace(case=c, policy=LmPolicy(model, GrpoSampler(seed, 1.0)), rollouts=rollouts, params=params, adv=adv, mask=mask)
    if c["kind"] == "train":
        from ferrl_b200.grpo import LossConfig
        s.loss = LossConfig(dapo_norm=float(mask.sum()))
    return s


def _prepare_prefill(c, seed):
    model, _ = _model(c, _weights(c, seed))
    model.merge_adapters()
    g = _rng(c, seed)
    P, G = c["prompts"], c["group"]
    ids = _ids(c, g, P, c["hi"])
    lens = torch.tensor(_spread(c["lo"], c["hi"], P), device="cuda")
    ids[torch.arange(c["hi"], device="cuda")[None, :] >= lens[:, None]] = 0
    grouped = c["family"] == "dense"
    dec = model.new_decoder(P * G, c["hi"] + 128, group=G) if grouped else model.new_decoder(P, c["hi"] + 128)
    return SimpleNamespace(case=c, dec=dec, ids=ids, lens=lens)


def _prepare_decode(c, seed):
    model, _ = _model(c, _weights(c, seed))
    model.merge_adapters()
    lens, kv_len, tokens, layers = _cache(c, seed)
    P, G = c["prompts"], c["group"]
    B, top = P * G, int(c["hi"] + c["done"])
    if c["family"] == "dense":
        dec = model.new_decoder(B, top + 64, group=G)
        with torch.no_grad():
            rows = P if G > 1 else B
            dec.prefill(torch.zeros(rows, c["hi"], dtype=torch.int64, device="cuda"), lens)      # lays out the rows' caches
    else:
        dec = model.new_decoder(B, top + 64)
    for i, kind in enumerate(_types(c)):
        mine = (dec.state[i][0], dec.state[i][1]) if c["family"] == "hybrid" else (dec.k[i], dec.v[i])
        for at, x in zip(mine, layers[i]):
            if kind == "linear_attention":
                at.copy_(x)
            elif hasattr(dec, "table"):
                t = torch.arange(x.shape[1], device="cuda")
                at[dec.table[:, t // PAGE].long(), (t % PAGE)[None, :].expand(B, -1)] = x
            else:
                at[:, :x.shape[1]] = x
    live = torch.ones(B, dtype=torch.bool, device="cuda")
    step = getattr(dec, "decode_native", None) or dec.decode
    feed = (lambda: step(tokens, live)) if getattr(dec, "supports_retirement", False) else (lambda: step(tokens))

    def once():
        dec.kv_len.copy_(kv_len)            # every pass at the same context
        return feed()
    advanced = dec.step_state() if hasattr(dec, "step_state") else []
    kept = [t.clone() for t in advanced]
    once()
    torch.cuda.synchronize()
    for t, k in zip(advanced, kept):
        t.copy_(k)
    del kept
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        logits = once()
    states = [dec.state[i][1] for i, k in enumerate(_types(c)) if k == "linear_attention"]
    return SimpleNamespace(case=c, graph=graph, out=[logits, *states], keep=(dec, kv_len, tokens, live))


def _sample_inputs(c, seed):
    g = _rng(c, seed)
    logits = torch.randn(c["rows"], c["vocab"], generator=g, device="cuda") * 2.5
    rows = torch.randint(0, 1 << 40, (c["rows"],), generator=g, device="cuda")
    return (logits.bfloat16() if c["dtype"] == "bf16" else logits), rows, seed % 1000


def prepare(case, seed):
    if case["kind"] == "sample":
        from ferrl_b200.sampler import GrpoSampler
        logits, rows, at = _sample_inputs(case, seed)
        return SimpleNamespace(case=case, sampler=GrpoSampler(seed, case["temperature"]), logits=logits, rows=rows, at=at)
    return {"prefill": _prepare_prefill, "decode": _prepare_decode}.get(case["kind"], _prepare_rows)(case, seed)


def run(state):
    c = state.case
    if c["kind"] == "train":
        from ferrl_b200.grpo import grpo_loss
        for p in state.params.values():
            p.grad = None
        logp = state.policy.token_logprobs(state.rollouts)
        loss = grpo_loss(logp, logp.detach(), None, state.adv, state.mask, state.loss)
        state.policy.backward(loss)
        return {"logp": logp.detach(), **{k: p.grad for k, p in state.params.items()}}
    if c["kind"] == "score":
        return state.policy.token_logprobs_detached(state.rollouts)
    if c["kind"] == "prefill":
        return [state.dec.prefill(state.ids, state.lens), state.dec.k, state.dec.v]
    if c["kind"] == "decode":
        state.graph.replay()
        return state.out
    return state.sampler.sample(state.logits, state.rows, state.at, None, c["top_p"])


# ---------------------------------------------------------------------------------------------------------------- work
def _layer_weights(c, kind, tokens):
    """``(entries of a layer's weights that a pass over ``tokens`` reads, multiply-adds per token)``."""
    n = sum(inn * sum(parts.values()) for inn, parts, _ in _projections(c, kind).values())
    if c["family"] != "hybrid" or not c["experts"]:
        return n, n
    one = 3 * c["width"] * c["ff"]
    return (n + c["experts"] * c["width"] + one * min(c["experts"], tokens * c["top"]),
            n + c["experts"] * c["width"] + one * c["top"])


def work(case):
    c = case
    if c["kind"] == "sample":
        return {"bytes": c["rows"] * c["vocab"] * (2 if c["dtype"] == "bf16" else 4), "flops": 0}
    head = c["vocab"] * c["width"]
    if c["kind"] == "decode":
        lens = _spread(c["lo"], c["hi"], c["prompts"])
        B = c["prompts"] * c["group"]
        read, flops = head, 2 * B * head
        for kind in _types(c):
            n, per = _layer_weights(c, kind, B)
            read += n
            flops += 2 * B * per
            row = 2 * c["kv"] * c["dim"]
            if kind == "linear_attention":
                read += B * c["vh"] * 128 * 128 * 4           # float32 state, read and written: twice two entries
                flops += B * c["vh"] * 128 * 128 * 6
            elif kind == "sliding_attention":
                read += row * sum(min(L + c["done"], c["window"]) for L in lens) * c["group"]
                flops += 4 * c["heads"] * c["dim"] * B * min(c["hi"] + c["done"], c["window"])
            else:
                shared = [L for L in lens] if c["family"] == "dense" else [L * c["group"] for L in lens]
                read += row * (sum(shared) + B * c["done"])
                flops += 4 * c["heads"] * c["dim"] * sum((L + c["done"]) * c["group"] for L in lens)
        return {"bytes": 2 * read + 4 * B * c["vocab"], "flops": flops}
    lens = _spread(c["lo"], c["hi"], c["prompts"])
    if c["kind"] == "prefill":
        rows, scored = lens, len(lens)
    else:
        rows = [L + c["new"] - 1 for L in lens for _ in range(c["group"])]
        scored = c["new"] * len(rows)
    T = sum(rows)
    flops, read = 2 * scored * head, (1 if c["family"] == "gemma" else 2) * head
    for kind in _types(c):
        n, per = _layer_weights(c, kind, T)
        read += n
        flops += 2 * T * per
        if kind == "linear_attention":
            flops += T * c["vh"] * 128 * 128 * 6
        else:
            far = c["window"] if kind == "sliding_attention" else 1 << 30
            flops += 4 * c["heads"] * c["dim"] * sum(sum(min(t + 1, far) for t in range(S)) for S in rows)
    hidden = 2 * T * c["width"] * (2 * c["layers"] + 1)
    if c["kind"] == "train":
        return {"bytes": 2 * (2 * read) + 2 * hidden, "flops": 2 * flops}       # the gradient of every input once more
    if c["kind"] == "prefill":
        hidden += 2 * 2 * T * c["kv"] * c["dim"] * c["layers"]
    return {"bytes": 2 * read + hidden, "flops": flops}


def tolerance(case):
    """bf16 operands and activations through a few layers: logits and log-probs are up to 0.011 off float64, gradients (which
    a backward through the same roundings reaches) up to 0.02, this framework's kernels and library kernels alike; float32
    probabilities in the draw."""
    if case["kind"] == "sample":
        return {"rel": 1e-4, "max": 1e-3, "differ": 0.01}
    return {"rel": 0.03 if case["kind"] in ("train", "decode") else 0.02, "max": 0.9}


# --------------------------------------------------------------------------------------------------------------- exact
def _rms(x, w=None, zero=False, eps=1e-6):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)
    return y if w is None else y * (1 + w if zero else w)


def _rope(x, pos, freq):
    """Rotates the leading ``2 * len(freq)`` entries of ``x`` ``[B,S,H,D]`` at positions ``[B,S]``."""
    n = freq.shape[0]
    a = (pos[..., None].float() * freq.float()).double()[:, :, None]
    u, v = x[..., :n], x[..., n:2 * n]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin(), x[..., 2 * n:]], -1)


def _freq(width, theta):
    return (theta ** -(torch.arange(0, width, 2, dtype=torch.float64, device="cuda") / width)).float()


def _act(c, g):
    return F.gelu(g, approximate="tanh") if c["family"] == "gemma" else F.silu(g)


class _Exact:
    """The decoder of a case in float64; ``w`` holds its weights and, when training, the adapters' leaves."""

    def __init__(self, c, w):
        self.c, self.w = c, {k: v.double() for k, v in w.items()}
        rot = {"hybrid": c["dim"] // 4}.get(c["family"], c["dim"])
        self.freq = _freq(rot, {"dense": 1e6, "hybrid": 1e7, "gemma": 1e6}[c["family"]])
        self.freq_sliding = _freq(rot, 1e4)

    def lin(self, i, kind, name, x):
        inn, parts, adapted = _projections(self.c, kind)[name]
        y = x @ self.w[f"{i}.{name}"].T
        outs = list(y.split(list(parts.values()), -1))
        for j, part in enumerate(parts):
            a = self.w.get(f"{i}.{name}.{part}.A")
            if a is not None:
                outs[j] = outs[j] + (x @ a.T) @ self.w[f"{i}.{name}.{part}.B"].T * 2.0
        return outs

    def attend(self, q, k, v, mask, scale):
        """``q`` ``[B,S,H,D]``, ``k``, ``v`` ``[B,T,G,D]``, ``mask`` ``[B or 1,S,T]``."""
        B, S, H, D = q.shape
        q = q.transpose(1, 2).reshape(B, k.shape[2], -1, S, D)
        s = torch.einsum("bgrsd,btgd->bgrst", q, k) * scale
        p = torch.softmax(s.masked_fill(~mask[:, None, None], float("-inf")), -1)
        return torch.einsum("bgrst,btgd->bgrsd", p, v).reshape(B, H, S, D).transpose(1, 2)

    def attention(self, i, kind, x, pos, mask, cached):
        c, w, gemma, zero = self.c, self.w, self.c["family"] == "gemma", self.c["family"] == "hybrid"
        B, S, _ = x.shape
        name = "inp" if zero else "qkv"
        parts = self.lin(i, kind, name, x)
        q, k = parts[0], parts[1]
        gate = None
        if zero:
            q, gate = q.chunk(2, -1)
        k = k.reshape(B, S, c["kv"], c["dim"])
        v = k if len(parts) == 2 else parts[2].reshape(k.shape)
        if gemma:
            v = _rms(v)
        f = self.freq_sliding if kind == "sliding_attention" else self.freq
        q = _rope(_rms(q.reshape(B, S, c["heads"], -1), w[f"{i}.q_norm"], zero), pos, f)
        k = _rope(_rms(k, w[f"{i}.k_norm"], zero), pos, f)
        own = (k, v)
        if cached is not None:
            k, v = (torch.cat([t.double(), n], 1) for t, n in zip(cached, own))
        a = self.attend(q, k, v, mask, 1.0 if gemma else c["dim"] ** -0.5).reshape(B, S, -1)
        if zero:
            a = a * torch.sigmoid(gate)
        return self.lin(i, kind, "out" if zero else "o", a)[0], own

    def gdn(self, i, x, state):
        """Gated delta rule over chunks; ``state`` = (convolution inputs ``[B,C,3]``, ``S``) or ``None``."""
        c, w = self.c, self.w
        B, T, _ = x.shape
        kh, vh = c["kh"], c["vh"]
        mixed, z, b, a = self.lin(i, "linear_attention", "inp", x)
        left = mixed.new_zeros(B, mixed.shape[-1], 3) if state is None else state[0].double()
        ctx = torch.cat([left, mixed.transpose(1, 2)], -1)
        y = F.silu(sum(ctx[..., j:j + T] * w[f"{i}.conv_w"][:, j, None] for j in range(4))).transpose(1, 2)
        q, k, v = (t.reshape(B, T, -1, 128) for t in y.split([kh * 128, kh * 128, vh * 128], -1))
        unit = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        q, k = (unit(t).repeat_interleave(vh // kh, 2) for t in (q, k))
        q = q * 128 ** -0.5
        beta, g = torch.sigmoid(b), -torch.exp(w[f"{i}.A_log"]) * F.softplus(a + w[f"{i}.dt_bias"])
        q, k, v, beta, g = (t.transpose(1, 2) for t in (q, k, v, beta, g))                 # [B, vh, T, ..]
        S = v.new_zeros(B, vh, 128, 128) if state is None else state[1].double()
        outs = []
        for s in range(0, T, 64):
            qc, kc, vc, bc, gc = (t[:, :, s:s + 64] for t in (q, k, v, beta, g))
            n = qc.shape[2]
            G = gc.cumsum(-1)
            low = torch.ones(n, n, dtype=torch.bool, device=x.device).tril()
            decay = (G[..., :, None] - G[..., None, :]).masked_fill(~low, float("-inf")).exp()
            eye = torch.eye(n, dtype=x.dtype, device=x.device)
            M = eye + (kc @ kc.transpose(-1, -2) * decay).tril(-1) * bc[..., None]
            rhs = bc[..., None] * (vc - G.exp()[..., None] * (kc @ S))
            new = torch.linalg.solve_triangular(M, rhs, upper=False)
            outs.append(G.exp()[..., None] * (qc @ S) + (qc @ kc.transpose(-1, -2) * decay) @ new)
            last = G[..., -1:]
            S = last.exp()[..., None] * S + (kc * (last - G).exp()[..., None]).transpose(-1, -2) @ new
        o = torch.cat(outs, 2).transpose(1, 2)
        o = _rms(o, w[f"{i}.gdn_norm"]) * F.silu(z.reshape(B, T, vh, 128))
        return self.lin(i, "linear_attention", "out", o.reshape(B, T, -1))[0], S

    def ffn(self, i, kind, x):
        c, w = self.c, self.w
        name = {"hybrid": "shared." if c.get("experts") else "mlp."}.get(c["family"], "")
        g, u = self.lin(i, kind, name + "gate_up", x)
        y = self.lin(i, kind, name + "down", _act(c, g) * u)[0]
        if not c.get("experts"):
            return y
        y = y * torch.sigmoid(x @ w[f"{i}.shared_gate"].T)
        flat = x.reshape(-1, x.shape[-1])
        p, idx = torch.softmax(flat @ w[f"{i}.router"].T, -1).topk(c["top"], -1)
        p = p / p.sum(-1, keepdim=True)
        out = torch.zeros_like(flat)
        for e in range(c["experts"]):
            t, slot = (idx == e).nonzero(as_tuple=True)
            g, u = (flat[t] @ w[f"{i}.experts_gate_up"][e].T).chunk(2, -1)
            out = out.index_add(0, t, (F.silu(g) * u) @ w[f"{i}.experts_down"][e].T * p[t, slot, None])
        return y + out.reshape(x.shape)

    def layer(self, i, kind, h, pos, masks, cached=None):
        c, w, zero = self.c, self.w, self.c["family"] == "hybrid"
        x = _rms(h, w[f"{i}.input_norm"], zero)
        if kind == "linear_attention":
            o, kept = self.gdn(i, x, cached)
        else:
            o, kept = self.attention(i, kind, x, pos, masks[kind], cached)
        if c["family"] == "gemma":
            h = h + _rms(o, w[f"{i}.post_attn_norm"])
            return h + _rms(self.ffn(i, kind, _rms(h, w[f"{i}.pre_ffn_norm"])), w[f"{i}.post_ffn_norm"]), kept
        h = h + o
        return h + self.ffn(i, kind, _rms(h, w[f"{i}.post_norm"], zero)), kept

    def embed(self, ids):
        return self.w["embed"][ids] * (self.c["width"] ** 0.5 if self.c["family"] == "gemma" else 1.0)

    def logits(self, h):
        z = _rms(h, self.w["final_norm"], self.c["family"] == "hybrid") @ self.w.get("head", self.w["embed"]).T
        return 30 * torch.tanh(z / 30) if self.c["family"] == "gemma" else z

    def sequence(self, ids):
        """Hidden states of whole rows ``ids`` ``[B,S]`` and what every layer would cache."""
        S = ids.shape[1]
        pos = torch.arange(S, device=ids.device)[None, :]
        far = pos[0][:, None] - pos[0][None, :]
        masks = {"full_attention": (far >= 0)[None], "sliding_attention": ((far >= 0) & (far < self.c.get("window", 1)))[None]}
        h, kept = self.embed(ids), []
        for i, kind in enumerate(_types(self.c)):
            h, k = checkpoint(self.layer, i, kind, h, pos, masks, use_reentrant=False)
            kept.append(k)
        return h, kept


def _exact_rows(c, seed):
    w = _weights(c, seed)
    m = _Exact(c, w)
    leaves = {k: v.requires_grad_() for k, v in m.w.items() if k.count(".") > 1 and k[-2:] in (".A", ".B")}
    toks, lens, adv, mask = _rows(c, seed)
    N, parts, at = c["new"], [], 0
    total = mask.sum().double()
    for t, L in zip(toks, lens):                # rows of a prompt one by one: the float64 intermediates are large
        for r in range(t.shape[0]):
            with torch.set_grad_enabled(c["kind"] == "train"):
                ids = t[r:r + 1].cuda()
                h, _ = m.sequence(ids[:, :-1])
                z = torch.log_softmax(m.logits(h[:, L - 1:L - 1 + N]), -1)
                logp = z.gather(-1, ids[:, L:, None])[..., 0]
                if c["kind"] == "train":
                    (-(logp * mask[at:at + 1]).sum() * adv[at].double() / total).backward()
            parts.append(logp.detach())
            at += 1
    logp = torch.cat(parts)
    return logp if c["kind"] == "score" else {"logp": logp, **{k: v.grad for k, v in leaves.items()}}


def _exact_prefill(c, seed):
    m = _Exact(c, _weights(c, seed))
    g = _rng(c, seed)
    P, L = c["prompts"], c["hi"]
    ids = _ids(c, g, P, L)
    lens = torch.tensor(_spread(c["lo"], L, P), device="cuda")
    ids[torch.arange(L, device="cuda")[None, :] >= lens[:, None]] = 0
    with torch.no_grad():
        h, _ = m.sequence(ids)
        logits = m.logits(h[torch.arange(P, device="cuda"), lens - 1])
    return [logits, [None] * c["layers"], [None] * c["layers"]]         # where a cache keeps a token is the decoder's own affair


def _exact_decode(c, seed):
    m = _Exact(c, _weights(c, seed))
    lens, kv_len, tokens, layers = _cache(c, seed)
    pos = kv_len.long()
    h = m.embed(tokens[:, None])
    states = []
    with torch.no_grad():
        for i, kind in enumerate(_types(c)):
            kept = layers[i]
            masks = {}
            if kind != "linear_attention":
                slots = kept[0].shape[1]
                at = torch.arange(slots + 1, device="cuda")[None, :]
                if kind == "sliding_attention" and slots == c["window"]:        # the new token takes the slot of the one that leaves
                    past = (at != (pos % slots)[:, None]) & ((at < pos[:, None]) | (pos >= slots)[:, None])
                else:
                    past = at < pos[:, None]
                masks[kind] = (past | (at == slots))[:, None]
            h, new = m.layer(i, kind, h, pos[:, None], masks, kept)
            if kind == "linear_attention":
                states.append(new)
        return [m.logits(h[:, 0]), *states]


def _exact_sample(c, seed):
    logits, rows, at = _sample_inputs(c, seed)
    p = torch.softmax(logits.double() / c["temperature"], -1)
    keep = torch.ones_like(p, dtype=torch.bool)
    if c["top_p"] < 1:
        sp = p.sort(-1, descending=True).values
        cross = (sp.cumsum(-1) >= c["top_p"]).int().argmax(-1, keepdim=True)
        keep = p >= sp.gather(-1, cross)
    cdf = (p * keep).cumsum(-1)
    M, gold = (1 << 64) - 1, 0x9E3779B97F4A7C15

    def mix(z):
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M
        return z ^ (z >> 31)
    u = [(mix((mix((seed + r * gold) & M) + (at + 1) * gold) & M) >> 40) / (1 << 24) for r in rows.tolist()]
    u = torch.tensor(u, dtype=torch.float64, device="cuda")
    tok = (cdf > (u * cdf[:, -1])[:, None]).int().argmax(-1)
    return [tok, (p.gather(-1, tok[:, None]) / cdf[:, -1:]).log()[:, 0]]


def exact(case, seed):
    kinds = {"train": _exact_rows, "score": _exact_rows, "prefill": _exact_prefill, "decode": _exact_decode, "sample": _exact_sample}
    return kinds[case["kind"]](case, seed)
