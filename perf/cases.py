"""What this framework is used for, as cases that can be timed and compared.

Six kinds of calls, all through the public entry points:

* ``tah_generate``   ``TaHEngine.generate`` on TaH-plus-1.7B: prompts in, tokens out, 6 % of the tokens take a second pass
* ``tah_prefill``    ``TaHEngine.prefill`` of the same model: prompts in, logits of the last tokens and a filled cache out
* ``tah_train``      forward and backward of a fine-tuning step of the same model (every weight and adapter trainable)
* ``gunuvik_prefill`` / ``gunuvik_generate``   the same for a layered decoder (windowed attention, mLSTM): gunuvik-1.7b
* ``ditilix_prefill`` / ``ditilix_generate``   the same with routed experts: the first layers of ditilix-moe

Weights are random and made name by name from the seed, of the architectures' own sizes.  Embeddings are of unit size, output
projections are scaled with the depth and the head reads embeddings, so that a model is as sure of its next token as a trained one is,
and rounding does not change which token that is: a layered decoder counts upwards, TaH repeats a token (its second pass reads the
token that the first one proposed, and has to agree with it).  Everything is bf16.
"""
from __future__ import annotations

import math
import zlib

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

VOCAB, WIDTH, HEADS, KV_HEADS, DIM, FF = 151936, 2048, 16, 8, 128, 6144       # Qwen3-1.7B and the presets of its size
LAYERS = 28
RANK, TOPK, HARD = 64, 100, 0.06
MOE_LAYERS, EXPERTS, TOP, EXPERT_FF, DENSE_FF, GROUPS = 10, 64, 8, 768, 9216, 4
EPS, THETA = 1e-6, 1e6


def listed():
    return [
        # one user at a terminal: a question, a short answer.  Latency and launches count.
        dict(name="answer_one", kind="tah_generate", rows=1, prompt=45, ragged=False, new=24, sample=False),
        # a handful of users, questions of different lengths, sampled as a chat is
        dict(name="chat_few", kind="tah_generate", rows=6, prompt=310, ragged=True, new=32, sample=True),
        # a small batch on long documents: the cache is what is read
        dict(name="documents", kind="tah_generate", rows=20, prompt=1900, ragged=True, new=24, sample=False),
        # the serving batch of the headline benchmark
        dict(name="serving_batch", kind="tah_generate", rows=256, prompt=64, ragged=False, new=32, sample=False),
        # time to the first token of one ordinary prompt
        dict(name="first_token", kind="tah_prefill", rows=1, prompt=700, ragged=False),
        # prompts of an evaluation batch, read in one call
        dict(name="read_batch", kind="tah_prefill", rows=7, prompt=3500, ragged=True),
        # fine-tuning on labelled tokens, a padded micro-batch of short examples
        dict(name="tune_short", kind="tah_train", rows=3, prompt=500, ragged=True, all_iterate=False),
        # fine-tuning on one packed sequence whose tokens all take the second pass
        dict(name="tune_packed", kind="tah_train", rows=1, prompt=3072, ragged=False, all_iterate=True),
        # the layered decoder: long prompts, then a batch that decodes
        dict(name="hybrid_read", kind="gunuvik_prefill", rows=4, prompt=3000, ragged=True),
        dict(name="hybrid_decode", kind="gunuvik_generate", rows=50, prompt=120, ragged=True, new=24, sample=False),
        # routed experts: a medium prompt batch, and a few rows that decode
        dict(name="experts_read", kind="ditilix_prefill", rows=3, prompt=1100, ragged=True),
        dict(name="experts_decode", kind="ditilix_generate", rows=12, prompt=90, ragged=True, new=24, sample=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tah_generate"] * 4 + ["tah_prefill"] * 3 + ["tah_train"] * 3 +
                      ["gunuvik_prefill", "gunuvik_generate", "ditilix_prefill", "ditilix_generate"])
    ragged = rng.random() < 0.6
    if kind.endswith("_generate"):
        rows = _log(rng, 1, 256)
        prompt = _log(rng, 20, max(24, min(1900, 20000 // rows)))
        return dict(kind=kind, rows=rows, prompt=prompt, ragged=ragged, new=rng.randint(12, 32), sample=rng.random() < 0.4)
    if kind.endswith("_prefill"):
        rows = _log(rng, 1, 64)
        return dict(kind=kind, rows=rows, prompt=_log(rng, 16, max(20, min(4000, 14000 // rows))), ragged=ragged)
    rows = rng.randint(1, 4)
    return dict(kind=kind, rows=rows, prompt=_log(rng, 64, 2000 // rows), ragged=ragged and rows > 1, all_iterate=rng.random() < 0.5)


# ------------------------------------------------------------------------------------------------
# inputs and weights, from the seed alone
# ------------------------------------------------------------------------------------------------
def _generator(seed, name, device="cuda"):
    return torch.Generator(device=device).manual_seed((seed * 1000003 + zlib.crc32(name.encode())) % (2 ** 62))


def _normal(seed, name, shape, std, mean=0.0):
    t = torch.randn(shape, generator=_generator(seed, name), device="cuda", dtype=torch.bfloat16)
    return t.mul_(std).add_(mean) if mean else t.mul_(std)


def _lengths(case, seed):
    if not case["ragged"]:
        return [case["prompt"]] * case["rows"]
    g = _generator(seed, "lengths", "cpu")
    lens = (case["prompt"] * (0.25 + 0.75 * torch.rand(case["rows"], generator=g))).long().clamp(min=2).tolist()
    lens[seed % case["rows"]] = case["prompt"]
    return lens


def _prompts(case, seed, pad_left=True):
    """Token ids ``[rows, longest]`` and their mask (None without padding)."""
    lens = _lengths(case, seed)
    T = max(lens)
    ids = torch.randint(0, VOCAB, (case["rows"], T), generator=_generator(seed, "ids"), device="cuda")
    if min(lens) == T:
        return ids, None, lens
    n, at = torch.tensor(lens, device="cuda").view(-1, 1), torch.arange(T, device="cuda")
    mask = (at >= T - n if pad_left else at < n).long()
    return ids * mask, mask, lens


def _hard(case, seed, length):
    """``[rows, length]``: 1 where the token takes a second pass."""
    return (torch.rand(case["rows"], length, generator=_generator(seed, "hard"), device="cuda") < HARD).to(torch.int8)


def _tah_shapes():
    q, kv = HEADS * DIM, KV_HEADS * DIM
    out = {"model.embed_tokens.weight": (VOCAB, WIDTH)}
    for i in range(LAYERS):
        p = f"model.layers.{i}."
        for mod, splits, k in (("self_attn.qkv_proj", (q, kv, kv), WIDTH), ("self_attn.o_proj", (WIDTH,), q),
                               ("mlp.gate_up_proj", (FF, FF), WIDTH), ("mlp.down_proj", (WIDTH,), FF)):
            out[p + mod + ".weight"] = (sum(splits), k)
            out[p + mod + ".lora_A"] = (len(splits) * RANK, k)
            for j, f in enumerate(splits):
                out[p + mod + f".lora_B.{j}"] = (f, RANK)
        out[p + "self_attn.q_norm.weight"] = out[p + "self_attn.k_norm.weight"] = (DIM,)
        out[p + "input_layernorm.weight"] = out[p + "post_attention_layernorm.weight"] = (WIDTH,)
    out["model.norm.weight"], out["lm_head.weight"] = (WIDTH,), (VOCAB, WIDTH)
    return out


def _tah_weight(seed, name, shape):
    back = 1.0 / math.sqrt(2 * LAYERS) if "o_proj" in name or "down_proj" in name else 1.0
    if "lm_head" in name:
        return _tah_weight(seed, "model.embed_tokens.weight", shape).mul_(0.012)
    if "embed" in name:
        return _normal(seed, name, shape, 1.0)
    if "norm" in name:
        return _normal(seed, name, shape, 0.1, 1.0)
    if "lora_A" in name:
        return _normal(seed, name, shape, 0.6 / math.sqrt(shape[1]))
    return _normal(seed, name, shape, (0.01 if "lora_B" in name else 0.02) * back)


def _tah_model(seed):
    from tah_b200 import TaHConfig, TaHForCausalLM
    from tah_b200.models import Qwen3ForCausalLM, preset
    cfg = preset("tah-plus-1.7b", tie_word_embeddings=False)
    with torch.device("cuda"):
        base = Qwen3ForCausalLM(cfg, dtype=torch.bfloat16)
    adapter = dict(r=RANK, lora_alpha=2 * RANK, lora_dropout=0.0, target_modules="all-linear")
    return base, TaHConfig, TaHForCausalLM, adapter


def _load(base, seed):
    shapes = _tah_shapes()
    with torch.no_grad():
        for name, p in base.named_parameters():
            p.copy_(_tah_weight(seed, name, shapes[name]))


def _prepare_tah_engine(case, seed):
    from tah_b200.engine import TaHEngine
    base, TaHConfig, TaHForCausalLM, adapter = _tah_model(seed)
    decider = dict(hidden_states_size=WIDTH, inner_size=WIDTH // 4, hidden_states_layer_nums=[LAYERS], threshold=0.5)
    model = TaHForCausalLM(base, TaHConfig(max_iter=2, iter_decider="SimpleMLPIterDecider", iter_decider_kwargs=decider,
                                           adapter_kwargs=adapter, input_updater_kwargs={"topk": TOPK},
                                           train_loss="NextTokenPredLoss"))
    model.iter_decider.to(device="cuda", dtype=torch.bfloat16)
    _load(base, seed)
    ids, mask, lens = _prompts(case, seed)
    length = max(lens) + case.get("new", 1) + 16
    eng = TaHEngine(model.eval(), max_rows=case["rows"], max_seq_len=length)
    eng.hard_override = _hard(case, seed, length)
    return dict(case=case, engine=eng, ids=ids, mask=mask)


def _prepare_tah_train(case, seed):
    base, TaHConfig, TaHForCausalLM, adapter = _tah_model(seed)
    model = TaHForCausalLM(base, TaHConfig(max_iter=2, iter_decider="IterLabelDecider", iter_decider_kwargs={}, adapter_kwargs=adapter,
                                           input_updater_kwargs={"topk": TOPK}, train_loss="NextTokenPredLoss"))
    _load(base, seed)
    model.train()
    # gradients lie in one buffer per kind of weight, as they do under a sharded optimizer
    params, grads = dict(base.named_parameters()), {}
    for kind, names in _kinds().items():
        grads[kind] = torch.zeros(sum(params[n].numel() for n in names), dtype=torch.bfloat16, device="cuda")
        at = 0
        for n in names:
            params[n].grad = grads[kind][at:at + params[n].numel()].view_as(params[n])
            at += params[n].numel()
    ids, mask, labels, iters = _examples(case, seed)
    return dict(case=case, model=model, grads=grads, ids=ids, mask=mask, labels=labels, iters=iters)


def _kinds():
    """Names of the trainable weights by kind, in the order of the model."""
    out = {}
    for n in _tah_shapes():
        kind = "norms" if "norm" in n else "lora_B" if "lora_B" in n else "lora_A" if "lora_A" in n else \
            n.split(".")[-2]
        out.setdefault(kind, []).append(n)
    return out


def _examples(case, seed):
    """Sequences in which most tokens are what the model expects, labels, and how many passes each token takes."""
    ids, mask, _ = _prompts(case, seed, pad_left=False)
    jump = torch.rand(ids.shape, generator=_generator(seed, "jump"), device="cuda") < 0.3
    jump[:, 0] = True
    at = torch.arange(ids.shape[1], device="cuda").expand_as(ids)
    start = torch.where(jump, at, torch.zeros_like(at)).cummax(1).values
    ids = ids.gather(1, start)
    labels = ids if mask is None else torch.where(mask == 1, ids, torch.full_like(ids, -100))
    more = torch.ones_like(ids) if case["all_iterate"] else _hard(case, seed, ids.shape[1]).long()
    return ids, mask, labels, more + 1


def _layered_weight(seed, family, name, shape):
    last = name.rsplit(".", 1)[-1]
    if name == "embed":
        t = _normal(seed, name, shape, 1.0)
        if family == "ditilix":                # the router has no close calls: it reads flags that only the token sets
            high = torch.rand(VOCAB, EXPERTS, generator=_generator(seed, "flags"), device="cuda").topk(TOP, -1).indices
            t[:, :EXPERTS] = -4.0
            t.scatter_(1, high, 4.0)
        return t
    if name == "head":
        t = _layered_weight(seed, family, "embed", shape).roll(1, 0).mul_({"gunuvik": 0.5, "ditilix": 1.6}[family] / math.sqrt(WIDTH))
        if family == "ditilix":
            t[:, :EXPERTS] = 0.0
        return t
    if last == "router":
        t = _normal(seed, name, shape, 0.2 / math.sqrt(shape[1]))
        flag = torch.randperm(EXPERTS, generator=_generator(seed, name + "/flag", "cpu"))
        t[torch.arange(EXPERTS), flag] = 0.5
        return t
    if last in ("ls1", "ls2"):
        return _normal(seed, name, shape, 0.02, 0.15)
    if last in ("norm", "norm1", "norm1b", "norm2", "norm2b"):
        return _normal(seed, name, shape, 0.1, 1.0)
    if last == "act":
        return torch.tensor([0.6, -0.4, 0.3, 0.1], device="cuda").to(torch.bfloat16)
    if name.endswith("f.b"):
        return _normal(seed, name, shape, 0.5, 4.0)
    if len(shape) == 1:
        return _normal(seed, name, shape, 0.2)
    if last == "rel":
        return _normal(seed, name, shape, 0.5)
    if family == "gunuvik" and name.endswith(".mix.q") and shape[0] < HEADS * DIM:      # mLSTM: q . k of a token is positive
        own = _normal(seed, name, shape, 0.7 / math.sqrt(shape[1]))
        return own.add_(_layered_weight(seed, family, name[:-1] + "k", shape), alpha=0.7)
    if last in ("o", "down") and family == "ditilix":
        t = _normal(seed, name, shape, 0.5 / math.sqrt(shape[1]))
        t[:EXPERTS] = 0.0
        return t
    return _normal(seed, name, shape, 1.0 / math.sqrt(shape[1]))


def _prepare_layered(case, seed):
    from tah_b200.engine import HybridEngine
    from tah_b200.models import DitilixConfig, DitilixForCausalLM, GunuvikForCausalLM, ditilix_preset, gunuvik_preset
    family = case["kind"].split("_")[0]
    if family == "gunuvik":
        cls, cfg = GunuvikForCausalLM, gunuvik_preset("gunuvik-1.7b")
    else:
        d = ditilix_preset("ditilix-moe").to_dict()
        cls, cfg = DitilixForCausalLM, DitilixConfig.from_dict(dict(d, layers=d["layers"][:MOE_LAYERS]))
    model = cls(cfg, dtype=torch.bfloat16, device="cuda")
    with torch.no_grad():
        for name, shape in cfg.tensor_shapes().items():
            model.tensor(name).copy_(_layered_weight(seed, family, name, shape))
    ids, mask, _ = _prompts(case, seed)
    return dict(case=case, engine=HybridEngine(model, max_rows=case["rows"]), ids=ids, mask=mask)


def prepare(case, seed):
    if case["kind"] == "tah_train":
        return _prepare_tah_train(case, seed)
    return _prepare_tah_engine(case, seed) if case["kind"].startswith("tah") else _prepare_layered(case, seed)


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def _watched(case):
    """The decode tick whose logits are kept: the last one before the first row is done."""
    return case["new"] - 1


def run(state):
    case = state["case"]
    if case["kind"] == "tah_train":
        for g in state["grads"].values():
            g.zero_()
        out = state["model"](state["ids"], attention_mask=state["mask"], labels=state["labels"], iter_count_labels=state["iters"])
        out.loss.backward()
        return dict(loss=out.loss.detach(), grads=state["grads"])
    eng = state["engine"]
    if case["kind"].endswith("_prefill"):
        logits, _, _ = eng.prefill(state["ids"], state["mask"], 1)
        return dict(logits=logits, cache=eng.kv.pool, memory=[] if getattr(eng, "state", None) is None else eng.state.layers)
    kept = {}

    def on_tick(t, s):
        if t == _watched(case):
            kept["logits"] = s.cum[:case["rows"]].clone()

    how = dict(do_sample=True, temperature=0.6, top_p=0.95, top_k=20, seed=11) if case["sample"] else {}
    res = eng.generate(state["ids"], state["mask"], max_new_tokens=case["new"], sync_every=8, on_tick=on_tick, **how)
    return dict(tokens=torch.tensor(res.tokens), logits=kept["logits"])


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _model_numbers(family):
    """(weights a token meets in the layers, all weights of the layers, cache numbers a token leaves per layer run, attention
    layers, window)"""
    q, kv = HEADS * DIM, KV_HEADS * DIM
    attn = WIDTH * (2 * q + 2 * kv)
    if family == "tah":
        per = attn + 3 * WIDTH * FF
        return per * LAYERS, per * LAYERS, 2 * kv, LAYERS, None
    if family == "gunuvik":                    # of four layers: two with keys of their own, one that reads another's, one mLSTM
        per = 2 * attn + WIDTH * 2 * q + 9 * WIDTH * FF + WIDTH * (2 * 8 * 128 + 3 * 8 * 256)
        return per * LAYERS // 4, per * LAYERS // 4, 2 * kv, LAYERS * 3 // 4, 1024
    unit = 3 * WIDTH * EXPERT_FF
    own = [attn if i % 4 != 3 else WIDTH * 2 * q for i in range(MOE_LAYERS)]
    met = sum(own) + 2 * WIDTH * DENSE_FF + (MOE_LAYERS - 1) * (TOP + 1) * unit
    return met, sum(own) + 2 * WIDTH * DENSE_FF + (MOE_LAYERS - 1) * (EXPERTS + 1) * unit, 2 * kv, MOE_LAYERS, None


def work(case):
    family = case["kind"].split("_")[0]
    met, held, cache, layers, window = _model_numbers(family)
    mean = case["prompt"] * (0.625 if case["ragged"] else 1.0)
    n, again = case["rows"] * mean, HARD if family == "tah" else 0.0
    see = lambda t: t if window is None else min(t, window)
    attn = lambda tokens, keys: tokens * keys * 4 * HEADS * DIM * layers
    head = VOCAB * WIDTH

    def weights(tokens):                       # numbers of the layers' weights that a pass over that many tokens reads
        if family != "ditilix":
            return held
        unit, used = 3 * WIDTH * EXPERT_FF, EXPERTS * (1 - (1 - TOP / EXPERTS) ** tokens)
        return held - (MOE_LAYERS - 1) * unit * (EXPERTS - used)

    if case["kind"] == "tah_train":
        twice = 2.0 if case["all_iterate"] else 1 + HARD
        flops = 3 * twice * (n * 2 * (met + head) + attn(n, mean / 2))
        return dict(flops=flops, bytes=2.0 * 2 * (held + 2 * head) + 2 * 2 * n * WIDTH)
    flops = (1 + again) * (n * 2 * met + attn(n, see(mean) / 2 if window is None else see(mean / 2))) + 2 * head * (case["rows"] + again * n)
    size = 2.0 * (weights(n) + head) + 2.0 * n * cache * layers + 2.0 * n * WIDTH
    if case["kind"].endswith("_generate"):
        ticks = (case["new"] - 1) * (1 + again)
        flops += ticks * case["rows"] * (2 * (met + head) + 4 * HEADS * DIM * layers * see(mean))
        size += ticks * 2.0 * (weights(case["rows"]) + head + case["rows"] * (see(mean) * cache * layers + VOCAB))
    return dict(flops=float(flops), bytes=float(size))


def tolerance(case):
    # Against exact(): logits of the 28 layers with a bf16 residual stream are 0.012 to 0.014 off, of the layered decoders (32-bit
    # residual) 0.0037 to 0.0046, gradients up to 0.021.  Four times that, where 0.03 allows it.
    return {"rel": 0.03 if case["kind"].startswith("tah") else 0.018, "max": 0.9 if case["kind"] == "tah_train" else 0.5}


# ------------------------------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ------------------------------------------------------------------------------------------------
def _rms(x, w=None, groups=1):
    y = x.unflatten(-1, (groups, -1))
    y = (y * torch.rsqrt(y.square().mean(-1, keepdim=True) + EPS)).flatten(-2)
    return y if w is None else y * w


def _rope(x, pos):
    f = THETA ** (-torch.arange(0, DIM, 2, device="cuda", dtype=torch.float64) / DIM)
    a = (pos.double().unsqueeze(-1) * f).unsqueeze(1)
    lo, hi = x.chunk(2, -1)
    return torch.cat([lo * a.cos() - hi * a.sin(), hi * a.cos() + lo * a.sin()], -1)


def _attend(q, k, v, seen, scale=DIM ** -0.5, edit=None, sink=None):
    """``q [n, H, d]`` over ``k, v [m, G, d]``; ``seen [n, m]``; ``edit`` changes the scores; ``sink [H]`` joins the denominator."""
    H, G = q.shape[1], k.shape[1]
    s = torch.einsum("nghd,mgd->ghnm", q.unflatten(1, (G, H // G)), k).flatten(0, 1) * scale
    s = (s if edit is None else edit(s)).masked_fill(~seen, -math.inf)
    if sink is not None:
        s = torch.cat([s, sink.view(H, 1, 1).expand(H, s.shape[1], 1)], -1)
    p = torch.softmax(s, -1)[..., :k.shape[0]]
    return torch.einsum("ghnm,mgd->nghd", p.unflatten(0, (G, H // G)), v).flatten(1, 2).flatten(1)


def _tah_layer(w, h, pos, rows, before, lora):
    """One layer for packed tokens ``h``; ``rows``: first and last token of every row; ``before``: keys, values, positions and rows
    of the pass before, or None.  Returns the new ``h`` and the keys and values of these tokens."""
    def lin(x, mod, splits):
        y = x @ w[mod + ".weight"].T
        if not lora:
            return y
        t = (x @ w[mod + ".lora_A"].T).split(RANK, -1)
        return y + 2.0 * torch.cat([a @ w[f"{mod}.lora_B.{j}"].T for j, a in enumerate(t)], -1)

    q, kv = HEADS * DIM, KV_HEADS * DIM
    x = _rms(h, w["input_layernorm.weight"])
    q, k, v = (t.unflatten(-1, (-1, DIM)) for t in lin(x, "self_attn.qkv_proj", 3).split([q, kv, kv], -1))
    q = _rope(_rms(q, w["self_attn.q_norm.weight"]), pos)
    k = _rope(_rms(k, w["self_attn.k_norm.weight"]), pos)
    out = []
    for r, (a, b) in enumerate(rows):
        if a == b:
            continue
        ks, vs, ps = k[a:b], v[a:b], pos[a:b]
        if before is not None:
            c, d = before[3][r]
            ks, vs, ps = (torch.cat([old[c:d], new]) for old, new in zip(before, (ks, vs, ps)))
        out.append(_attend(q[a:b], ks, vs, ps.unsqueeze(0) <= pos[a:b].unsqueeze(1)))
    h = h + lin(torch.cat(out), "self_attn.o_proj", 1)
    g, u = lin(_rms(h, w["post_attention_layernorm.weight"]), "mlp.gate_up_proj", 2).chunk(2, -1)
    return h + lin(F.silu(g) * u, "mlp.down_proj", 1), k, v


def _spans(counts):
    ends = torch.tensor([0] + list(counts)).cumsum(0).tolist()
    return list(zip(ends[:-1], ends[1:]))


def _tah_passes(weight, tokens, lens, hard, layer_call):
    """Final hidden states of both passes over packed ``tokens`` (rows of ``lens``), and the logits function.  ``hard``: which of
    them take the second pass; ``weight(name)``: a weight in 64 bits; ``layer_call``: how a layer is called."""
    embed, head = weight("model.embed_tokens.weight"), weight("lm_head.weight")
    rows, pos = _spans(lens), torch.cat([torch.arange(n, device="cuda") for n in lens])
    again = hard.nonzero().flatten()
    rows1 = _spans([int(hard[a:b].sum()) for a, b in rows])
    h, kept = embed[tokens], []
    layers = []
    for i in range(LAYERS):
        p = f"model.layers.{i}."
        names = [n[len(p):] for n in _tah_shapes() if n.startswith(p)]
        get = lambda p=p, names=names: {n: weight(p + n) for n in names}
        layers.append(get)
        h, k, v = layer_call(get, h, pos, rows, None, False)
        kept.append((k, v))
    norm = weight("model.norm.weight")
    logits = lambda x: x @ head.T
    first = _rms(h, norm)
    if again.numel() == 0:
        return first, None, logits, again
    val, idx = [], []
    for part in first[again].split(2048):
        a, b = logits(part).topk(TOPK, -1)
        val.append(a), idx.append(b)
    mix = torch.softmax(torch.cat(val), -1).unsqueeze(1)
    h = torch.cat([torch.bmm(m, embed[j]) for m, j in zip(mix.split(512), torch.cat(idx).split(512))]).squeeze(1)
    for get, (k, v) in zip(layers, kept):
        h, _, _ = layer_call(get, h, pos[again], rows1, (k, v, pos, rows), True)
    return first, _rms(h, norm), logits, again


def _followed(case, ids, mask, lens):
    """The tokens of every row: its prompt, and behind it the tokens that the model generates."""
    rows = [ids[r][mask[r].bool()] if mask is not None else ids[r] for r in range(len(lens))]
    new = case.get("new", 0)
    more = torch.arange(1, new + 1, device="cuda") * (0 if case["kind"].startswith("tah") else 1)
    return [torch.cat([t, (t[-1:] + more) % VOCAB]) if new else t for t in rows]


def _exact_tah(case, seed):
    ids, mask, lens = _prompts(case, seed)
    new = case.get("new", 0)
    seqs = _followed(case, ids, mask, lens)
    hard = _hard(case, seed, max(lens) + case.get("new", 1) + 16).bool()
    full = [t.numel() for t in seqs]
    flat = torch.cat([hard[r, :n] for r, n in enumerate(full)])
    shapes = _tah_shapes()
    weight = lambda name: _tah_weight(seed, name, shapes[name]).double()
    call = lambda get, *a: _tah_layer(get(), *a)
    first, second, logits, again = _tah_passes(weight, torch.cat(seqs), full, flat, call)
    place = torch.full((flat.numel(),), -1, device="cuda")
    place[again] = torch.arange(again.numel(), device="cuda")
    at, deep = [], []                          # the token whose logits are wanted, and whether its second pass counts
    for r, (n, (a, _)) in enumerate(zip(lens, _spans(full))):
        here = hard[r].tolist()
        if not new:
            p, d = n - 1, int(here[n - 1])
        else:
            p, d = n, 0                        # tick 1 runs the first new token
            for _ in range(_watched(case) - 1):
                p, d = (p, 1) if here[p] and d == 0 else (p + 1, 0)
        at.append(a + p)
        deep.append(d)
    at = torch.tensor(at, device="cuda")
    out = logits(first[at])
    for r, d in enumerate(deep):
        if d:
            out[r] += logits(second[place[at[r]]])
    return dict(logits=out, tokens=None) if new else dict(logits=out, cache=None, memory=None)


def _exact_tah_train(case, seed):
    ids, mask, labels, iters = _examples(case, seed)
    lens = [ids.shape[1]] * ids.shape[0] if mask is None else mask.sum(1).tolist()
    keep = torch.ones_like(ids, dtype=torch.bool) if mask is None else mask.bool()
    shapes = _tah_shapes()
    W = {n: _tah_weight(seed, n, s).double().requires_grad_() for n, s in shapes.items()}
    call = lambda get, *a: checkpoint(_tah_layer, get(), *a, use_reentrant=False)
    first, second, logits, again = _tah_passes(W.__getitem__, ids[keep], lens, (iters > 1)[keep], call)
    target = F.pad(labels, (0, 1), value=-100)[:, 1:][keep]
    place = torch.full((target.numel(),), -1, device="cuda")
    place[again] = torch.arange(again.numel(), device="cuda")

    def piece(a, b, head):
        z, more = first[a:b] @ head.T, place[a:b] >= 0
        if second is not None:
            z = z.index_add(0, more.nonzero().flatten(), second[place[a:b][more]] @ head.T)
        return F.cross_entropy(z, target[a:b], ignore_index=-100, reduction="sum")

    total = 0.0
    for a in range(0, target.numel(), 1024):
        total = total + checkpoint(piece, a, min(target.numel(), a + 1024), W["lm_head.weight"], use_reentrant=False)
    loss = total / (target != -100).sum()
    loss.backward()
    grad = lambda n: torch.zeros(shapes[n], dtype=torch.float64, device="cuda") if W[n].grad is None else W[n].grad
    return dict(loss=loss.detach(), grads={k: torch.cat([grad(n).flatten() for n in names]) for k, names in _kinds().items()})


def _bucket_bias(rel, T, far):
    """``[H, T]`` learned bias by distance: rows of the table, exact for half of them, logarithmic behind."""
    n_rows, half = rel.shape[0], rel.shape[0] // 2
    m, out = n_rows - half, []
    for n in range(T):
        k = n
        if n >= half:
            k = 0
            while k < m and far ** (k + 1) * half ** (m - k - 1) <= n ** m:
                k += 1
            k = min(n_rows - 1, half + k)
        out.append(k)
    return rel[torch.tensor(out, device="cuda")].T


def _exact_gunuvik(case, seed):
    ids, mask, lens = _prompts(case, seed)
    seqs = _followed(case, ids, mask, lens)
    if case.get("new"):
        seqs = [t[:n + _watched(case)] for t, n in zip(seqs, lens)]
    spans, H, G, MH, MK, MV = _spans([t.numel() for t in seqs]), HEADS, KV_HEADS, 8, 128, 256
    get = lambda name, *shape: _layered_weight(seed, "gunuvik", name, shape).double()
    W, T = WIDTH, max(t.numel() for t in seqs)
    x, kv = get("embed", VOCAB, W)[torch.cat(seqs)], {}
    for i in range(LAYERS):
        p, m = f"l{i}.", f"l{i}.mix."
        h = _rms(x, get(p + "norm1", W))
        if i % 4 == 1:
            q, k = (h @ get(m + n, MH * MK, W).T for n in "qk")
            v, gate = (h @ get(m + n, MH * MV, W).T for n in "vg")
            cap = lambda n: 15.0 * torch.tanh((h @ get(m + n, MH, W).T + get(m + n + ".b", MH)) / 15.0)
            li, lf = cap("i"), F.logsigmoid(cap("f"))
            out = []
            for a, b in spans:
                fs = lf[a:b].cumsum(0).T                                    # [heads, T]
                gain = li[a:b].T - fs
                top = fs + torch.cummax(gain, 1).values.clamp(min=0)
                tri = torch.ones(b - a, b - a, dtype=torch.bool, device="cuda").tril()
                d = torch.exp((fs - top).unsqueeze(2) + gain.unsqueeze(1)).masked_fill(~tri, 0)
                s = torch.einsum("thd,shd->hts", q[a:b].unflatten(1, (MH, MK)), k[a:b].unflatten(1, (MH, MK))) * MK ** -0.5 * d
                o = torch.einsum("hts,shd->htd", s, v[a:b].unflatten(1, (MH, MV)))
                o = o / (torch.maximum(s.sum(-1).abs(), torch.exp(-top)) + 1e-6).unsqueeze(-1)
                out.append(o.transpose(0, 1))
            y = (_rms(torch.cat(out)).flatten(1) * get(m + "norm", MH * MV) * torch.sigmoid(gate)) @ get(m + "o", W, MH * MV).T
        else:
            q = _rms((h @ get(m + "q", H * DIM, W).T + get(m + "q.b", H * DIM)).unflatten(1, (H, DIM)), get(m + "q.norm", DIM))
            if i % 4 != 3:
                k, v = ((h @ get(m + n, G * DIM, W).T + get(m + n + ".b", G * DIM)).unflatten(1, (G, DIM)) for n in "kv")
                kv[i] = _rms(k, get(m + "k.norm", DIM)), v
            k, v = kv[i if i % 4 != 3 else i - 3]
            bias = _bucket_bias(get(m + "rel", 32, H), T, 512)
            out = []
            for a, b in spans:
                n = torch.arange(b - a, device="cuda")
                dist = n.unsqueeze(1) - n
                seen = (dist >= 0) & ((dist < 1024) | (n < 4))
                by = bias[:, dist.clamp(min=0)]
                out.append(_attend(q[a:b], k[a:b], v[a:b], seen, edit=lambda s: s + by, sink=get(m + "sink", H)))
            o = torch.cat(out).unflatten(1, (H, DIM)) * torch.sigmoid(h @ get(m + "g", H, W).T).unsqueeze(-1)
            y = o.flatten(1) @ get(m + "o", W, H * DIM).T
        x = x + _rms(y, get(p + "norm1b", W)) * get(p + "ls1", W)
        if i % 4 != 1:
            h = _rms(x, get(p + "norm2", W))
            y = (F.silu(h @ get(p + "mlp.gate", FF, W).T) * (h @ get(p + "mlp.up", FF, W).T)) @ get(p + "mlp.down", W, FF).T
            x = x + _rms(y, get(p + "norm2b", W)) * get(p + "ls2", W)
    last = torch.tensor([b - 1 for _, b in spans], device="cuda")
    return _layered_answer(case, _rms(x[last], get("final.norm", W)) @ get("head", VOCAB, W).T)


def _layered_answer(case, logits):
    return dict(logits=logits, tokens=None) if case.get("new") else dict(logits=logits, cache=None, memory=None)


def _exact_ditilix(case, seed):
    ids, mask, lens = _prompts(case, seed)
    seqs = _followed(case, ids, mask, lens)
    if case.get("new"):
        seqs = [t[:n + _watched(case)] for t, n in zip(seqs, lens)]
    spans, W = _spans([t.numel() for t in seqs]), WIDTH
    get = lambda name, *shape: _layered_weight(seed, "ditilix", name, shape).double()
    pos = torch.cat([torch.arange(t.numel(), device="cuda", dtype=torch.float64) for t in seqs]).unsqueeze(1)
    ang = pos * 10000.0 ** (-torch.arange(0, W, 2, device="cuda", dtype=torch.float64) / W)
    x = get("embed", VOCAB, W)[torch.cat(seqs)] + torch.stack([ang.sin(), ang.cos()], -1).flatten(1)
    temp = (1.0 + 0.1 * torch.log(torch.floor((pos + 1) / 2048) + 1.0)).unsqueeze(-1)

    def unit(z, p, limit=7.0):
        g, u = (z @ get(p + "gate", EXPERT_FF, W).T).clamp(max=limit), (z @ get(p + "up", EXPERT_FF, W).T).clamp(-limit, limit)
        return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ get(p + "down", W, EXPERT_FF).T

    for i in range(MOE_LAYERS):
        m, f = f"l{i}.mix.", f"l{i}.mlp."
        h = _rms(x, get(f"l{i}.norm1", W), GROUPS)
        q = (h @ get(m + "q", HEADS * DIM, W).T).unflatten(1, (HEADS, DIM)) * temp
        if i % 4 != 3:
            k, v = ((h @ get(m + n, KV_HEADS * DIM, W).T).unflatten(1, (KV_HEADS, DIM)) for n in "kv")
        out = []
        for a, b in spans:
            tri = torch.ones(b - a, b - a, dtype=torch.bool, device="cuda").tril()
            out.append(_attend(q[a:b], k[a:b], v[a:b], tri, edit=lambda s: 30.0 * torch.tanh(s / 30.0)))
        y = torch.cat(out) @ get(m + "o", W, HEADS * DIM).T
        if i == 0:
            z, act = h @ get(f + "up", DENSE_FF, W).T, get(f + "act", 4)
            y = y + (act[0] * _rms(z) + act[1] * _rms(z ** 2) + act[2] * _rms(z ** 3) + act[3]) @ get(f + "down", W, DENSE_FF).T
        else:
            score, which = torch.sigmoid(h @ get(f + "router", EXPERTS, W).T).topk(TOP, -1)
            for e in range(EXPERTS):
                t, j = (which == e).nonzero(as_tuple=True)
                if t.numel():
                    y = y.index_add(0, t, unit(score[t, j].unsqueeze(1) * h[t], f"{f}e{e}."))
            y = y + torch.sigmoid(h @ get(f + "shared.sg", 1, W).T) * unit(h, f + "shared.")
        x = x + 0.5 * y
    last = torch.tensor([b - 1 for _, b in spans], device="cuda")
    return _layered_answer(case, 0.5 * (_rms(x[last], get("final.norm", W), GROUPS) @ get("head", VOCAB, W).T))


def exact(case, seed):
    if case["kind"] == "tah_train":
        return _exact_tah_train(case, seed)
    with torch.no_grad():
        if case["kind"].startswith("tah"):
            return _exact_tah(case, seed)
        return (_exact_gunuvik if case["kind"].startswith("gunuvik") else _exact_ditilix)(case, seed)
