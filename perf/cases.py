"""What a user of this engine has it do, as cases that can be timed and compared.

A case is a model (layer sizes of `bench.py`, random weights made from the seed), an element type, and one of four calls:

    prompt    Engine.prefill of one prompt, then its logits (the time to the first token)
    score     Engine.prefill_logits of one text: the logits of every position (perplexity, ranking of answers)
    generate  Engine.prefill of some slots, Engine.decode, then history and logits (greedy tokens chosen on the device)
    serve     ModelRunner.step over a batch of requests from their prompts to their last token, portions of prompts beside
              decoded rows under a token budget as the scheduler cuts them, the continuations given (trace replay, scoring of
              given answers; the tokens do not depend on rounding, so that two runs can be compared row by row)

A pass is the whole call and leaves nothing behind: its requests end with it. `exact` restates the models in 64 bits on whole
sequences with plain torch."""
from __future__ import annotations

import hashlib
import math
import random

import torch

from hipinfer_b200 import Engine
from hipinfer_b200.engine import StepEntry

DEV = "cuda:0"
PAGE = 16
STD = 0.02
ROPE = dict(rope_type="llama3", factor=32.0, low_freq_factor=1.0, high_freq_factor=4.0, original_max_position_embeddings=8192)
LLAMA = {
    "llama-1b": dict(hidden_size=2048, intermediate_size=8192, num_hidden_layers=16, num_attention_heads=32, num_key_value_heads=8,
                     head_dim=64, tie_word_embeddings=True, rope_scaling=ROPE),
    "llama-3b": dict(hidden_size=3072, intermediate_size=8192, num_hidden_layers=28, num_attention_heads=24, num_key_value_heads=8,
                     head_dim=128, tie_word_embeddings=True, rope_scaling=ROPE),
    # the layer sizes of the 8B shape with 16 of its 32 layers
    "llama-8b": dict(hidden_size=4096, intermediate_size=14336, num_hidden_layers=16, num_attention_heads=32, num_key_value_heads=8,
                     head_dim=128, tie_word_embeddings=False, rope_scaling=dict(ROPE, factor=8.0)),
}
VOCAB = 128256
WIDTH, LAYERS, HEADS, KV_HEADS, HEAD_DIM, FF, WINDOW, POSITIONS = 2048, 16, 32, 8, 64, 8192, 1024, 4096


def llama_config(model):
    return dict(architectures=["LlamaForCausalLM"], vocab_size=VOCAB, max_position_embeddings=131072, rms_norm_eps=1e-5,
                rope_theta=500000.0, hidden_act="silu", **LLAMA[model])


def torirax_config():
    """Delta-rule layers and differential attention (a window that keeps the first tokens) in turn; every second attention
    layer reads the cache of the one before it."""
    layers, owner = [], None
    for i in range(LAYERS):
        if i % 2 == 0:
            layers.append(dict(type="general_delta", mixer=dict(heads=HEADS, dim=HEAD_DIM, decay_rank=64), mlp=None))
            continue
        m = dict(heads=HEADS, kv_heads=KV_HEADS, dim=HEAD_DIM // 2, vdim=HEAD_DIM, scale=(HEAD_DIM // 2) ** -0.5, diff=0.5,
                 mask=dict(size=WINDOW, keep_first=4))
        if owner is not None and (i // 2) % 2 == 1:
            m["kv_from"] = owner
        else:
            owner = i
        layers.append(dict(type="attention", mixer=m, mlp=dict(kind="dense", ff=FF)))
    return dict(architecture="Torirax", vocab=VOCAB, width=WIDTH, max_positions=POSITIONS, embedding=dict(scale=1.0),
                norm=dict(eps=1e-5), layers=layers)


def vegodra_config():
    """Latent attention, gated linear attention, latent attention, chunked attention with a sink, and again; every second
    chunked layer reads the cache of the one before it."""
    layers, owner, count, ff = [], None, 0, dict(kind="dense", ff=FF)
    D = HEAD_DIM
    for i in range(LAYERS):
        if i % 4 in (0, 2):
            m = dict(heads=HEADS, dim=D, rot_dim=D // 2, vdim=D, q_rank=12 * D, kv_rank=4 * D, scale=(D + D // 2) ** -0.5,
                     rot=dict(base=10000.0, dims=D // 2))
            layers.append(dict(type="latent_attention", mixer=m, mlp=ff))
        elif i % 4 == 1:
            layers.append(dict(type="gla", mixer=dict(heads=HEADS, dim=D, vdim=D, tau=16.0, decay_rank=64), mlp=ff))
        else:
            m = dict(heads=HEADS, kv_heads=KV_HEADS, dim=D, vdim=D, scale=0.125, rot=dict(base=1000000.0, dims=D // 2),
                     mask=dict(size=WINDOW))
            if count % 2 == 1:
                m["kv_from"] = owner
            else:
                owner = i
            count += 1
            layers.append(dict(type="attention", mixer=m, mlp=ff))
    return dict(architecture="Vegodra", vocab=VOCAB, width=WIDTH, max_positions=POSITIONS, norm=dict(eps=1e-5), layers=layers)


def config_of(case):
    model = case["model"]
    return llama_config(model) if model in LLAMA else torirax_config() if model == "torirax" else vegodra_config()


def _case(name, model, call, requests, prompt, new, ragged=False, budget=2048, dtype="bfloat16"):
    c = dict(model=model, dtype=dtype, call=call, requests=requests, prompt=prompt, new=new, ragged=ragged, budget=budget)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a short question on an idle engine: launches and latency count
        _case("short_prompt", "llama-1b", "prompt", 1, 23, 1),
        # one chat: a 128-token prompt and its answer
        _case("chat", "llama-1b", "serve", 1, 128, 64),
        # the engine's headline workload: eight requests behind 2,048-token prompts
        _case("batch_8", "llama-1b", "serve", 8, 2048, 128),
        # many small requests at once
        _case("batch_64", "llama-1b", "serve", 64, 512, 64),
        # the first token behind a long prompt
        _case("prompt_2048", "llama-1b", "prompt", 1, 2048, 1),
        # a text scored token by token, an odd length
        _case("score_1531", "llama-1b", "score", 1, 1531, 1),
        # a document larger than a step's budget, at the layer sizes of the 8B shape
        _case("document", "llama-8b", "prompt", 1, 5003, 1),
        # answers to documents at the 8B layer sizes, more rows than a few
        _case("batch_20", "llama-8b", "serve", 20, 700, 32, ragged=True),
        # the scheduler's mix: requests of many lengths, portions of 512 tokens beside decoding rows
        _case("mixed", "llama-3b", "serve", 14, 2048, 24, ragged=True, budget=512),
        # the 32-bit engine
        _case("float32", "llama-1b", "generate", 3, 301, 12, dtype="float32"),
        # the designs with a recurrence: its long prompts and its single tokens
        _case("delta_rule", "torirax", "serve", 4, 1200, 48),
        _case("linear_attention", "vegodra", "serve", 4, 1200, 48),
    ]


def draw(rng):
    """One more case of the same ranges."""
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["prompt", "score", "chat", "batch", "batch", "mixed", "generate", "torirax", "vegodra"])
    if kind == "prompt":
        model = rng.choice(["llama-1b", "llama-1b", "llama-3b", "llama-8b"])
        return _case(None, model, "prompt", 1, log(5, 4500), 1)
    if kind == "score":
        return _case(None, "llama-1b", "score", 1, log(40, 1900), 1)
    if kind == "chat":
        return _case(None, rng.choice(["llama-1b", "llama-3b"]), "serve", 1, log(20, 1500), log(12, 48))
    if kind == "batch":
        model = rng.choice(["llama-1b", "llama-1b", "llama-8b"])
        requests = log(2, 64)
        most = 14000 if model == "llama-1b" else 7000
        return _case(None, model, "serve", requests, log(40, min(2048, most // requests)), log(12, 64 if model == "llama-1b" else 32),
                     ragged=rng.random() < 0.5)
    if kind == "mixed":
        requests = log(3, 14)
        return _case(None, "llama-3b", "serve", requests, log(100, 14000 // requests if requests > 6 else 2048), log(8, 24), ragged=True,
                     budget=rng.choice([256, 512, 1024]))
    if kind == "generate":
        return _case(None, "llama-1b", "generate", rng.randint(1, 3), log(10, 290), log(4, 12), dtype="float32")
    return _case(None, kind, "serve", log(1, 6), log(50, 760), log(16, 48), ragged=rng.random() < 0.5)


# ------------------------------------------------------------------------------------------ what a case's requests are
def lengths(case):
    """The prompts' lengths: all alike, or uniform from a thirty-second of the longest on."""
    n, p = case["requests"], case["prompt"]
    if not case["ragged"]:
        return [p] * n
    rng = random.Random(1000003 * n + 101 * p + case["new"])
    return [rng.randint(max(1, p // 32), p) for _ in range(n)]


def schedule(case):
    """Steps of (request, first position, tokens, whether its last row's logits are wanted): every request that has its prompt
    behind it has one row, what is left of the budget goes to prompts in their order."""
    lens, new, budget = lengths(case), case["new"], case["budget"]
    done, steps = [0] * len(lens), []
    while any(d < n + new - 1 for d, n in zip(done, lens)):
        step, room = [], budget
        for r, n in enumerate(lens):
            if n <= done[r] < n + new - 1 and room:
                step.append((r, done[r], 1, True))
                room -= 1
        for r, n in enumerate(lens):
            if done[r] < n and room:
                k = min(n - done[r], room)
                step.append((r, done[r], k, done[r] + k == n))
                room -= k
        for r, _, k, _ in step:
            done[r] += k
        steps.append(step)
    return steps


def token_ids(case, seed):
    g = torch.Generator().manual_seed(1_000_003 + int(seed))
    return [torch.randint(0, VOCAB, (n + case["new"] - 1,), generator=g).tolist() for n in lengths(case)]


# ------------------------------------------------------------------------------------------ the calls
def prepare(case, seed):
    longest = max(lengths(case)) + case["new"]
    eng = Engine(config=config_of(case), random_weights=int(seed), std=STD, dtype=case["dtype"], max_batch=case["requests"],
                 max_seq=-(-longest // PAGE) * PAGE, max_prefill=case["budget"], page_size=PAGE)
    state = dict(case=case, engine=eng, tokens=token_ids(case, seed))
    if case["call"] == "serve":
        state["steps"] = [[StepEntry(r, state["tokens"][r][p:p + k], [k - 1] if want else []) for r, p, k, want in step]
                          for step in schedule(case)]
    return state


def run(state):
    eng, call, tokens = state["engine"], state["case"]["call"], state["tokens"]
    if call == "prompt":
        eng.prefill(0, tokens[0])
        return {"logits": eng.logits(1)}
    if call == "score":
        return {"logits": eng.prefill_logits(0, tokens[0])}
    if call == "generate":
        new, lens = state["case"]["new"], lengths(state["case"])
        for r, n in enumerate(lens):
            eng.prefill(r, tokens[r][:n])
        eng.decode(len(lens), new - 1)
        return {"logits": eng.logits(len(lens)), "tokens": torch.tensor([eng.history(r, n, new) for r, n in enumerate(lens)])}
    runner, at = eng.runner, 0
    logits = torch.empty(sum(len(e.want) for s in state["steps"] for e in s), VOCAB, dtype=torch.float32, device=DEV)
    for step in state["steps"]:
        rows = runner.step(step)
        logits[at:at + rows.shape[0]].copy_(rows)       # a decoding step's logits are overwritten by the next one's
        at += rows.shape[0]
    for r in range(len(tokens)):
        runner.end(r)
    return {"logits": logits}


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def _layers(case):
    """Per layer (elements of its weights, attention operations per visible key, cached elements per token, the most keys a row
    sees, elements of its state)."""
    if case["model"] in LLAMA:
        m = LLAMA[case["model"]]
        H, Hq, G, D = m["hidden_size"], m["num_attention_heads"], m["num_key_value_heads"], m["head_dim"]
        w = H * D * (2 * Hq + 2 * G) + 3 * H * m["intermediate_size"]
        return H, [(w, 4 * Hq * D, 2 * G * D, 1 << 30, 0)] * m["num_hidden_layers"]
    out, W, H, G, D = [], WIDTH, HEADS, KV_HEADS, HEAD_DIM
    for L in config_of(case)["layers"]:
        ff = 0 if L["mlp"] is None else (2 if case["model"] == "torirax" else 3) * W * FF
        own = 0 if L["mixer"].get("kv_from") is not None else 1
        if L["type"] in ("general_delta", "gla"):
            out.append(((6 if L["type"] == "general_delta" else 5) * W * H * D + 64 * (W + H * D) + ff, 0, 0, 0, H * D * D))
        elif L["type"] == "latent_attention":
            w = W * 12 * D + 12 * D * H * (D + D // 2) + W * (4 * D + D // 2) + 2 * 4 * D * H * D + 2 * W * H * D
            out.append((w + ff, 2 * H * (2 * D + D // 2), 4 * D + D // 2, 1 << 30, 0))
        elif case["model"] == "torirax":
            out.append((W * D * (3 * H + 2 * G * own) + ff, 6 * H * D, 2 * G * D, WINDOW + 4, 0))
        else:
            out.append((W * (D * (2 * H + 2 * G * own) + H) + ff, 4 * H * D, 2 * G * D, WINDOW, 0))
    return W, out


def work(case):
    """A step reads its weights, the cache and state of its requests, and writes its logits and its tokens' cache; a greedy
    generation and a prompt are such steps too."""
    width, layers = _layers(case)
    size = 4 if case["dtype"] == "float32" else 2
    bytes_ = flops = 0.0
    if case["call"] == "serve":
        steps = schedule(case)
    else:
        lens = lengths(case)
        cut = [[(r, p, min(case["budget"], n - p), p + case["budget"] >= n)] for r, n in enumerate(lens) for p in range(0, n, case["budget"])]
        steps = cut + [[(r, n + i, 1, True) for r, n in enumerate(lens)] for i in range(case["new"] - 1)]
    for step in steps:
        rows = sum(k for _, _, k, _ in step)
        wanted = rows if case["call"] == "score" else sum(1 for s in step if s[3])
        bytes_ += size * (VOCAB * width if wanted else 0) + 4 * wanted * VOCAB
        flops += 2.0 * wanted * VOCAB * width
        for w, per_key, cached, seen, state in layers:
            bytes_ += size * w + 8 * state * len(step)
            flops += 2.0 * rows * w + 6.0 * rows * state
            for _, p, k, _ in step:
                keys = sum(min(p + i + 1, seen) for i in range(k)) if seen < 1 << 30 else k * p + k * (k + 1) / 2
                flops += per_key * keys
                bytes_ += size * cached * min(p + k, seen + k)
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # bfloat16: the same passes through the plain kernels, or with portions cut elsewhere, lie 0.005 to 0.020 (2-norm) and 0.03 to
    # 0.12 (largest) apart: every row and product is rounded, through 16 to 28 layers. float32: 8e-6 from the 64-bit logits.
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 4e-4, "differ": 0.0}
    return {"rel": 0.03, "max": 0.4}


# ------------------------------------------------------------------------------------------ the models in 64 bits
F = torch.float64


class Weights:
    """The tensors of the random-weights mode, in 64 bits: every tensor N(0, 0.02) from a stream of its own keyed by the seed
    and its name, drawn in 32 bits and stored in bfloat16."""

    def __init__(self, seed):
        self.seed = int(seed)

    def __call__(self, name, *shape):
        key = int.from_bytes(hashlib.sha256(f"{self.seed}:{name}".encode()).digest()[:8], "little") & 0x7FFFFFFFFFFFFFFF
        g = torch.Generator(device=DEV)
        g.manual_seed(key)
        return (torch.randn(shape, generator=g, dtype=torch.float32, device=DEV) * STD).to(torch.bfloat16).to(F)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _layer_norm(x, eps):
    d = x - x.mean(-1, keepdim=True)
    return d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps)


def _angles(pos, freq):
    """The angle is position times frequency in 32 bits, as the models define it; cos and sin of it in 64."""
    a = (pos.to(torch.float32)[:, None] * freq.to(torch.float32)[None, :]).to(F)
    return torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]


def _rotate(t, pos, freq, interleaved=False):
    """t [T, heads, D]: the first 2 len(freq) dimensions rotated, in halves or in neighbouring pairs; the rest passes."""
    n = freq.numel()
    c, s = _angles(pos, freq)
    u, v = (t[..., 0:2 * n:2], t[..., 1:2 * n:2]) if interleaved else (t[..., :n], t[..., n:2 * n])
    a, b = u * c - v * s, v * c + u * s
    turned = torch.stack([a, b], -1).flatten(-2) if interleaved else torch.cat([a, b], -1)
    return torch.cat([turned, t[..., 2 * n:]], -1)


def _frequencies(dims, base):
    return float(base) ** (-torch.arange(0, dims, 2, dtype=F, device=DEV) / dims)


def _llama_frequencies(dims, base, sc):
    f = 1.0 / float(base) ** (torch.arange(0, dims, 2, dtype=F, device=DEV) / dims)
    wave, orig = 2.0 * math.pi / f, sc["original_max_position_embeddings"]
    smooth = (orig / wave - sc["low_freq_factor"]) / (sc["high_freq_factor"] - sc["low_freq_factor"])
    mid = (1.0 - smooth) * f / sc["factor"] + smooth * f
    return torch.where(wave < orig / sc["high_freq_factor"], f, torch.where(wave > orig / sc["low_freq_factor"], f / sc["factor"], mid))


def _attend(q, k, v, scale, seen, sink=None):
    """q [T, H, D], k [T, G, D], v [T, G, E], seen [T, T]; one group of heads at a time. sink: a number in every denominator."""
    T, H, _ = q.shape
    per, out = H // k.shape[1], []
    for g in range(k.shape[1]):
        s = torch.einsum("thd,sd->hts", q[:, g * per:(g + 1) * per], k[:, g]) * scale
        s = s.masked_fill(~seen, float("-inf"))
        if sink is not None:
            s = torch.cat([s, torch.full_like(s[..., :1], sink)], -1)
        p = torch.softmax(s, -1)
        out.append(torch.einsum("hts,se->the", p[..., :T], v[:, g]))
    return torch.cat(out, 1)


def _seen(T, rule=None):
    i, j = torch.arange(T, device=DEV)[:, None], torch.arange(T, device=DEV)[None, :]
    return (j <= i) if rule is None else (j <= i) & rule(i, j)


def _llama(case, w, x, spans):
    m = LLAMA[case["model"]]
    H, Hq, G, D, I = m["hidden_size"], m["num_attention_heads"], m["num_key_value_heads"], m["head_dim"], m["intermediate_size"]
    freq = _llama_frequencies(D, 500000.0, m["rope_scaling"])
    for l in range(m["num_hidden_layers"]):
        p = f"model.layers.{l}."
        wq, wk, wv = (w(f"{p}self_attn.{n}_proj.weight", k * D, H) for n, k in (("q", Hq), ("k", G), ("v", G)))
        wo = w(p + "self_attn.o_proj.weight", H, Hq * D)
        h, att = _rms(x, 1e-5), []
        for a, b in spans:
            pos = torch.arange(b - a, device=DEV)
            q, k, v = ((h[a:b] @ m_.T).view(b - a, -1, D) for m_ in (wq, wk, wv))
            att.append(_attend(_rotate(q, pos, freq), _rotate(k, pos, freq), v, D ** -0.5, _seen(b - a)).flatten(1))
        x = x + torch.cat(att) @ wo.T
        h = _rms(x, 1e-5)
        act = torch.nn.functional.silu(h @ w(p + "mlp.gate_proj.weight", I, H).T) * (h @ w(p + "mlp.up_proj.weight", I, H).T)
        x = x + act @ w(p + "mlp.down_proj.weight", H, I).T
    return _rms(x, 1e-5)


def _walk(spans, step, like):
    """A recurrence over the requests side by side: step(the rows of token t of every request that has one, which they are)."""
    out = torch.zeros_like(like)
    longest = max(b - a for a, b in spans)
    order = sorted(range(len(spans)), key=lambda r: spans[r][0] - spans[r][1])        # longest first: a prefix of them goes on
    starts = torch.tensor([spans[r][0] for r in order], device=DEV)
    size = [spans[r][1] - spans[r][0] for r in order]
    for t in range(longest):
        n = sum(1 for s in size if s > t)
        rows = starts[:n] + t
        out[rows] = step(rows, n)
    return out


def _delta(h, w, p, spans, eps):
    H, D, W = HEADS, HEAD_DIM, WIDTH
    r, k, v, a, g = ((h @ w(p + n, H * D, W).T) for n in ("r", "k", "v", "a", "g"))
    decay = torch.tanh(h @ w(p + "w1", 64, W).T) @ w(p + "w2", H * D, 64).T
    decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(decay)).view(-1, H, D)
    r, k, v, a = (t.view(-1, H, D) for t in (r, k, v, torch.sigmoid(a)))
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    S = torch.zeros(len(spans), H, D, D, dtype=F, device=DEV)

    def step(rows, n):
        old = S[:n]
        new = decay[rows][..., None] * old + k[rows][..., None] * v[rows][..., None, :]
        new -= (a[rows] * u[rows])[..., None] * (u[rows][..., None, :] @ old)
        S[:n] = new
        return (r[rows][..., None, :] @ new).squeeze(-2)

    o = _rms(_walk(spans, step, v), eps).flatten(1) * torch.sigmoid(g)
    return o @ w(p + "o", W, H * D).T


def _torirax(case, w, x, spans):
    c, eps, kept = torirax_config(), 1e-5, {}
    place = torch.cat([torch.arange(b - a, device=DEV) for a, b in spans])
    x = x + w("pos", POSITIONS, WIDTH)[place]
    H, G, D, E = HEADS, KV_HEADS, HEAD_DIM // 2, HEAD_DIM
    for i, L in enumerate(c["layers"]):
        h, p, m = _layer_norm(x, eps), f"l{i}.mix.", L["mixer"]
        if L["type"] == "general_delta":
            x = x + _delta(h, w, p, spans, eps)
            continue
        owner = m.get("kv_from", i)
        if owner == i:
            kept[i] = (h @ w(p + "k", G * 2 * D, WIDTH).T, h @ w(p + "v", G * E, WIDTH).T)
        q = h @ w(p + "q", H * 2 * D, WIDTH).T
        dot = lambda a, b: float((w(p + a, D) * w(p + b, D)).sum())
        lam = math.exp(dot("lq1", "lk1")) - math.exp(dot("lq2", "lk2")) + m["diff"]
        att = []
        for a, b in spans:
            T = b - a
            seen = _seen(T, lambda i_, j_: (i_ - j_ < WINDOW) | (j_ < m["mask"]["keep_first"]))
            qs, ks = q[a:b].view(T, H, 2, D), kept[owner][0][a:b].view(T, G, 2, D)
            one, two = (_attend(qs[:, :, j], ks[:, :, j], kept[owner][1][a:b].view(T, G, E), m["scale"], seen) for j in (0, 1))
            att.append((_rms(one - lam * two, eps) * (1.0 - m["diff"])).flatten(1))
        x = x + (torch.cat(att) * torch.sigmoid(h @ w(p + "g", H * E, WIDTH).T)) @ w(p + "o", WIDTH, H * E).T
        z = _layer_norm(x, eps) @ w(f"l{i}.mlp.up", FF, WIDTH).T
        x = x + (_rms(z, eps) + _rms(z * z, eps) + _rms(z * z * z, eps) + 1.0) @ w(f"l{i}.mlp.down", WIDTH, FF).T
    return _layer_norm(x, eps)


def _gla(h, w, p, m, spans, eps):
    H, D, W = HEADS, HEAD_DIM, WIDTH
    q, k, v = ((h @ w(p + n, H * D, W).T).view(-1, H, D) for n in ("q", "k", "v"))
    z = (h @ w(p + "a1", 64, W).T) @ w(p + "a2", H * D, 64).T
    alpha = torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"]).view(-1, H, D)
    S = torch.zeros(len(spans), H, D, D, dtype=F, device=DEV)

    def step(rows, n):
        S[:n] = alpha[rows][..., None] * S[:n] + k[rows][..., None] * v[rows][..., None, :]
        return (q[rows][..., None, :] @ S[:n]).squeeze(-2) * D ** -0.5

    o = _rms(_walk(spans, step, v), eps).flatten(1) * torch.nn.functional.silu(h @ w(p + "g", H * D, W).T)
    return o @ w(p + "o", W, H * D).T


def _latent(h, w, p, m, spans, eps):
    H, D, R, W = HEADS, HEAD_DIM, m["rot_dim"], WIDTH
    freq = _frequencies(m["rot"]["dims"], m["rot"]["base"])
    q = (_rms(h @ w(p + "dq", m["q_rank"], W).T, eps) @ w(p + "uq", H * (D + R), m["q_rank"]).T).view(-1, H, D + R)
    ckr = h @ w(p + "dkv", m["kv_rank"] + R, W).T
    c = _rms(ckr[:, :m["kv_rank"]], eps)
    k, v = ((c @ w(p + n, H * D, m["kv_rank"]).T).view(-1, H, D) for n in ("uk", "uv"))
    att = []
    for a, b in spans:
        pos = torch.arange(b - a, device=DEV)
        qr = _rotate(q[a:b, :, D:], pos, freq, True)
        kr = _rotate(ckr[a:b, None, m["kv_rank"]:], pos, freq, True).expand(-1, H, -1)
        att.append(_attend(torch.cat([q[a:b, :, :D], qr], -1), torch.cat([k[a:b], kr], -1), v[a:b], m["scale"], _seen(b - a)).flatten(1))
    return (torch.cat(att) * torch.sigmoid(h @ w(p + "g", H * D, W).T)) @ w(p + "o", W, H * D).T


def _chunked(h, w, p, m, i, kept, spans, eps):
    H, G, D, W = HEADS, KV_HEADS, HEAD_DIM, WIDTH
    freq, owner = _frequencies(m["rot"]["dims"], m["rot"]["base"]), m.get("kv_from", i)
    place = torch.cat([torch.arange(b - a, device=DEV) for a, b in spans])
    if owner == i:
        k = (h @ w(p + "k", G * D, W).T).view(-1, G, D)
        kept[i] = _rms(_rotate(k, place, freq), eps), (h @ w(p + "v", G * D, W).T).view(-1, G, D)
    q = _rms(_rotate((h @ w(p + "q", H * D, W).T).view(-1, H, D), place, freq), eps)
    att = [_attend(q[a:b], kept[owner][0][a:b], kept[owner][1][a:b], m["scale"],
                   _seen(b - a, lambda i_, j_: i_ // WINDOW == j_ // WINDOW), sink=0.0) for a, b in spans]
    return (torch.cat(att) * torch.sigmoid(h @ w(p + "g", H, W).T)[..., None]).flatten(1) @ w(p + "o", W, H * D).T


def _vegodra(case, w, x, spans):
    eps, kept = 1e-5, {}
    x = _layer_norm(x, eps)
    for i, L in enumerate(vegodra_config()["layers"]):
        h, p, m = _layer_norm(x, eps), f"l{i}.mix.", L["mixer"]
        if L["type"] == "latent_attention":
            y = _latent(h, w, p, m, spans, eps)
        elif L["type"] == "gla":
            y = _gla(h, w, p, m, spans, eps)
        else:
            y = _chunked(h, w, p, m, i, kept, spans, eps)
        gate = torch.nn.functional.gelu(h @ w(f"l{i}.mlp.gate", FF, WIDTH).T, approximate="tanh")
        x = x + y + (gate * (h @ w(f"l{i}.mlp.up", FF, WIDTH).T)) @ w(f"l{i}.mlp.down", WIDTH, FF).T
    return _layer_norm(x, eps)


def _logits(case, seed, sequences, rows):
    """64-bit logits of the given rows of the sequences laid end to end."""
    w, ends, at = Weights(seed), [], 0
    for s in sequences:
        ends.append((at, at + len(s)))
        at += len(s)
    flat = torch.tensor([t for s in sequences for t in s], device=DEV)
    llama = case["model"] in LLAMA
    width = LLAMA[case["model"]]["hidden_size"] if llama else WIDTH
    name = "model.embed_tokens.weight" if llama else "embed"
    body = _llama if llama else _torirax if case["model"] == "torirax" else _vegodra
    x = body(case, w, w(name, VOCAB, width)[flat], ends)[torch.tensor(rows, device=DEV)]
    head = name if llama and LLAMA[case["model"]]["tie_word_embeddings"] else "lm_head.weight" if llama else "head"
    return x @ w(head, VOCAB, width).T


def exact(case, seed):
    tokens, lens = token_ids(case, seed), lengths(case)
    first = [sum(len(t) for t in tokens[:r]) for r in range(len(tokens))]
    if case["call"] == "prompt":
        return {"logits": _logits(case, seed, tokens, [lens[0] - 1])}
    if case["call"] == "score":
        return {"logits": _logits(case, seed, tokens, range(lens[0]))}
    if case["call"] == "serve":
        return {"logits": _logits(case, seed, tokens, [first[r] + p + k - 1 for step in schedule(case) for r, p, k, want in step if want])}
    seqs, out = [t[:n] for t, n in zip(tokens, lens)], []
    for _ in range(case["new"]):
        logits = _logits(case, seed, seqs, [sum(len(s) for s in seqs[:r + 1]) - 1 for r in range(len(seqs))])
        out.append(logits.argmax(-1).tolist())
        seqs = [s + [t] for s, t in zip(seqs, out[-1])]
    return {"logits": logits, "tokens": torch.tensor(out).T.contiguous()}
