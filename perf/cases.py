"""What the framework's speed is measured on: batches of requests from their first token to their last.

A pass opens a batch of requests on an engine, brings their prompts in portions under a token budget (running requests decode
beside the portions, as the scheduler mixes them), decodes the given continuations token by token, and closes the requests. It
goes through `Engine.open / step / close` with token ids of the host, decode steps replayed as graphs, and returns the float32
logits of every position a token would be drawn from, as a trace replay or a scoring run keeps them. Token ids of the
continuations are given, so that outputs of two runs can be compared place by place.

Layer sizes are those of the benchmark's models (MiniCPM4-8B and -0.5B sizes, the 2,048 wide Nirozen and Gopitar), with fewer
layers where the whole depth would only repeat the same work. `exact` computes the same logits from whole sequences in float64.
"""
from __future__ import annotations

import math

import torch

from infinilm_b200.config import config_from_json
from infinilm_b200.engine import Engine, StepEntry

DEVICE = "cuda:0"
PAGE = 16
CHUNK = 2048                                      # the longest portion of one prompt in a step (the scheduler's default)
BUDGET = 8192                                     # tokens of a step (the scheduler's default)


# ---- the cases -----------------------------------------------------------------------------------------------------------
def listed():
    return [
        # one short question to a small model: the smallest call, bound by launches and latency
        {"name": "small_b1", "model": "minicpm4_0.5b", "layers": 24, "dtype": "bfloat16", "batch": 1, "shortest": 19, "longest": 19,
         "new": 24, "budget": BUDGET},
        # the headline benchmark's shape: eight requests of 2,048 tokens, then decoding at batch 8
        {"name": "batch8_2048", "model": "minicpm4_8b", "layers": 8, "dtype": "bfloat16", "batch": 8, "shortest": 2048, "longest": 2048,
         "new": 64, "budget": BUDGET},
        # a full batch of chats of odd lengths, mostly decoding
        {"name": "batch64_ragged", "model": "minicpm4_8b", "layers": 8, "dtype": "bfloat16", "batch": 64, "shortest": 17, "longest": 389,
         "new": 32, "budget": BUDGET},
        # time to the first token of one ordinary prompt
        {"name": "prefill_2048", "model": "minicpm4_8b", "layers": 8, "dtype": "bfloat16", "batch": 1, "shortest": 2048, "longest": 2048,
         "new": 1, "budget": BUDGET},
        # a long document and a short answer: portions over a growing cache, decoding over 16 thousand keys
        {"name": "long_16k", "model": "minicpm4_8b", "layers": 8, "dtype": "bfloat16", "batch": 1, "shortest": 16384, "longest": 16384,
         "new": 32, "budget": CHUNK},
        # a server's mix on a small model: requests of all lengths, portions and decoding in the same steps
        {"name": "serving_mix", "model": "minicpm4_0.5b", "layers": 24, "dtype": "bfloat16", "batch": 40, "shortest": 16, "longest": 1931,
         "new": 40, "budget": 2048},
        # the 32-bit path, a single request: a trace replayed for comparison
        {"name": "f32_b1", "model": "minicpm4_0.5b", "layers": 24, "dtype": "float32", "batch": 1, "shortest": 61, "longest": 61,
         "new": 6, "budget": BUDGET},
        # the 32-bit path, a batch of ragged prompts scored
        {"name": "f32_batch4", "model": "minicpm4_0.5b", "layers": 24, "dtype": "float32", "batch": 4, "shortest": 61, "longest": 443,
         "new": 4, "budget": BUDGET},
        # latent attention and routed experts: a small batch, mostly decoding
        {"name": "experts_decode_b8", "model": "nirozen_2k", "layers": 4, "dtype": "bfloat16", "batch": 8, "shortest": 67, "longest": 613,
         "new": 32, "budget": BUDGET},
        # the same design on prompts
        {"name": "experts_prefill", "model": "nirozen_2k", "layers": 4, "dtype": "bfloat16", "batch": 4, "shortest": 700, "longest": 1500,
         "new": 1, "budget": BUDGET},
        # windowed attention beside linear attention, delta-rule layers: a small batch, mostly decoding
        {"name": "recurrent_decode_b8", "model": "gopitar_2k", "layers": 8, "dtype": "bfloat16", "batch": 8, "shortest": 67, "longest": 613,
         "new": 32, "budget": BUDGET},
        # the same design on prompts longer than its window
        {"name": "recurrent_prefill", "model": "gopitar_2k", "layers": 8, "dtype": "bfloat16", "batch": 2, "shortest": 2100, "longest": 2900,
         "new": 1, "budget": BUDGET},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the same ranges: every model, batches of 1 to 64, prompts of 8 to 16,384 tokens, 1 to 64 new ones; a
    quarter in float32 (on the smaller models, with fewer tokens)."""
    most = {d: max(work(c)["flops"] for c in listed() if c["dtype"] == d) for d in ("bfloat16", "float32")}
    bytes_most = max(work(c)["bytes"] for c in listed())
    while True:
        f32 = rng.random() < 0.25
        model = rng.choice(["minicpm4_0.5b", "minicpm4_0.5b", "nirozen_2k", "gopitar_2k"] if f32 else
                           ["minicpm4_8b", "minicpm4_8b", "minicpm4_0.5b", "minicpm4_0.5b", "nirozen_2k", "gopitar_2k"])
        layers = {"minicpm4_0.5b": 24, "minicpm4_8b": 8, "nirozen_2k": 4, "gopitar_2k": 8}[model]
        longest = _log_int(rng, 8, 600 if f32 else 4000 if model == "gopitar_2k" else 16384)
        shortest = longest if rng.random() < 0.3 else _log_int(rng, 8, longest)
        c = {"model": model, "layers": layers, "dtype": "float32" if f32 else "bfloat16", "batch": _log_int(rng, 1, 8 if f32 else 64),
             "shortest": shortest, "longest": longest, "new": _log_int(rng, 1, 6 if f32 else 64), "budget": rng.choice([2048, 4096, BUDGET])}
        w = work(c)
        if w["flops"] <= 0.9 * most[c["dtype"]] and w["bytes"] <= 0.9 * bytes_most and (model != "gopitar_2k" or sum(prompt_lengths(c)) <= 6000):
            return c


def prompt_lengths(case):
    """`batch` lengths between `shortest` and `longest`, spread evenly over their logarithm in a fixed, mixed order."""
    a, b, n = math.log(case["shortest"]), math.log(case["longest"]), case["batch"]
    return [int(round(math.exp(a + (b - a) * ((0.5 + i * 0.6180339887498949) % 1.0)))) for i in range(n)]


def schedule(case):
    """The pass as steps: lists of (request, first token, one past the last, whether its last place's logits are wanted).
    Running requests decode first, then portions of the waiting prompts fill the budget."""
    lens, new = prompt_lengths(case), case["new"]
    at, steps = [0] * len(lens), []
    while any(p < n + new - 1 for p, n in zip(at, lens)):
        step, left = [], case["budget"]
        for i, n in enumerate(lens):
            if n <= at[i] < n + new - 1 and left > 0:
                step.append((i, at[i], at[i] + 1, True))
                left -= 1
        for i, n in enumerate(lens):
            m = min(CHUNK, left, n - at[i])
            if m > 0:
                step.append((i, at[i], at[i] + m, at[i] + m == n))
                left -= m
        for i, _, b, _ in step:
            at[i] = b
        steps.append(step)
    return steps


# ---- the models ----------------------------------------------------------------------------------------------------------
def model_json(case):
    name, layers = case["model"], case["layers"]
    if name.startswith("minicpm4"):
        big = name.endswith("8b")
        hd = 128 if big else 64
        return {"architectures": ["MiniCPMForCausalLM"], "model_type": "minicpm", "num_hidden_layers": layers,
                "hidden_size": 4096 if big else 1024, "num_attention_heads": 32 if big else 16, "num_key_value_heads": 2, "head_dim": hd,
                "intermediate_size": 16384 if big else 4096, "vocab_size": 73448, "rope_theta": 10000.0, "max_position_embeddings": 32768,
                "rope_scaling": {"rope_type": "longrope", "short_factor": [1.0 + 0.05 * i for i in range(hd // 2)],
                                 "long_factor": [1.0 + 0.25 * i for i in range(hd // 2)], "original_max_position_embeddings": 32768},
                "scale_emb": 12, "dim_model_base": 256, "scale_depth": 1.4, "rms_norm_eps": 1e-6, "tie_word_embeddings": not big,
                "torch_dtype": "bfloat16", "eos_token_id": [2]}
    if name == "nirozen_2k":
        mixer = {"heads": 16, "dim": 128, "vdim": 128, "q_rank": 768, "kv_rank": 256, "scale": 128 ** -0.5}
        mlp = {"kind": "moe", "router": {"experts": 64, "top": 6}, "expert": {"ff": 1408}, "shared": {"ff": 2816}}
        return {"architecture": "Nirozen", "vocab": 32000, "width": 2048, "norm": {"eps": 1e-5},
                "embedding": {"scale": 1.0, "bigram": {"buckets": 65521, "mul_prev": 8191, "mul_cur": 31}},
                "layers": [{"type": "latent_attention", "mixer": mixer, "mlp": mlp} for _ in range(layers)]}
    left = {"heads": 16, "kv_heads": 2, "dim": 128, "vdim": 128, "conv": 4, "mask": {"size": 1024}, "rot": {"base": 10000.0, "dims": 128},
            "scale": 128 ** -0.5}
    right = {"heads": 16, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** (-5 - 3 * i / 15) for i in range(16)]}
    par = {"type": "parallel", "mixer": {"left": left, "right": right, "left_scale": 0.5, "right_scale": 0.5}, "mlp": {"kind": "dense", "ff": 8192}}
    delta = {"type": "delta", "mixer": {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "conv": 4}, "mlp": {"kind": "dense", "ff": 8192}}
    return {"architecture": "Gopitar", "vocab": 32000, "width": 2048, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0}, "logit_softcap": 30.0,
            "layers": [delta if i % 4 == 2 else par for i in range(layers)]}


def make_weights(case, seed):
    """Checkpoint tensors by name, in bfloat16 values: matrices with the variance that keeps a row's size, norms around one."""
    raw, out = model_json(case), {}
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed * 2 + 1)

    def mat(name, n, k, gain=1.0):
        out[name] = torch.randn((n, k), generator=g, dtype=torch.bfloat16, device=DEVICE).mul_(gain * k ** -0.5)

    def vec(name, n, std, mean=0.0):
        out[name] = (torch.randn((n,), generator=g, dtype=torch.float32, device=DEVICE) * std + mean).to(torch.bfloat16)

    if case["model"].startswith("minicpm4"):
        H, I, hd = raw["hidden_size"], raw["intermediate_size"], raw["head_dim"]
        nq, nk = raw["num_attention_heads"] * hd, raw["num_key_value_heads"] * hd
        mat("model.embed_tokens.weight", raw["vocab_size"], H, H ** 0.5 / 12)
        for i in range(case["layers"]):
            p = f"model.layers.{i}."
            vec(p + "input_layernorm.weight", H, 0.05, 1.0)
            for n, rows in (("q", nq), ("k", nk), ("v", nk)):
                mat(p + f"self_attn.{n}_proj.weight", rows, H)
            mat(p + "self_attn.o_proj.weight", H, nq)
            vec(p + "post_attention_layernorm.weight", H, 0.05, 1.0)
            mat(p + "mlp.gate_proj.weight", I, H)
            mat(p + "mlp.up_proj.weight", I, H)
            mat(p + "mlp.down_proj.weight", H, I)
        vec("model.norm.weight", H, 0.05, 1.0)
        if not raw["tie_word_embeddings"]:
            mat("lm_head.weight", raw["vocab_size"], H, 16.0)
        return out
    W, V = raw["width"], raw["vocab"]
    mat("embed", V, W, W ** 0.5)
    nirozen = case["model"].startswith("nirozen")
    if nirozen:
        b = raw["embedding"]["bigram"]["buckets"]
        mat("bigram", b + 1, W, 0.5 * W ** 0.5)
    for i, L in enumerate(raw["layers"]):
        m, p = L["mixer"], f"l{i}.mix."
        mean = 0.0 if nirozen else 1.0            # the first design's block norms hold the deviation from one
        vec(f"l{i}.norm1", W, 0.05, mean)
        vec(f"l{i}.norm2", W, 0.05, mean)
        if nirozen:
            H, d, e, qr, r = m["heads"], m["dim"], m["vdim"], m["q_rank"], m["kv_rank"]
            mat(p + "dq", qr, W)
            vec(p + "dq.norm", qr, 0.05, 1.0)
            mat(p + "uq", H * d, qr)
            mat(p + "dkv", r, W)
            vec(p + "dkv.norm", r, 0.05, 1.0)
            mat(p + "uk", H * d, r)
            mat(p + "uv", H * e, r)
            mat(p + "o", W, H * e)
            vec(p + "sink", H, 1.0)
            mat(p + "g", H * e, W)
            f, q = L["mlp"], f"l{i}.mlp."
            E, ff, sh = f["router"]["experts"], f["expert"]["ff"], f["shared"]["ff"]
            mat(q + "router", E, W, 3.0)          # a trained router is sharp: logits of a few units
            vec(q + "router.b", E, 0.3)
            for n, rows, cols in (("gate", ff, W), ("up", ff, W), ("down", W, ff)):
                t = torch.randn((E, rows, cols), generator=g, dtype=torch.bfloat16, device=DEVICE).mul_(cols ** -0.5)
                out.update({f"{q}e{j}.{n}": t[j] for j in range(E)})
            mat(q + "shared.gate", sh, W)
            mat(q + "shared.up", sh, W)
            mat(q + "shared.down", W, sh)
            continue
        if L["type"] == "parallel":
            c, r = m["left"], m["right"]
            for n, rows in (("q", c["heads"] * c["dim"]), ("k", c["kv_heads"] * c["dim"]), ("v", c["kv_heads"] * c["vdim"])):
                mat(p + "left." + n, rows, W)
                vec(p + f"left.{n}.b", rows, 0.02)
                mat(p + f"left.{n}.conv", rows, c["conv"])
            mat(p + "left.g", c["heads"], W)
            mat(p + "left.o", W, c["heads"] * c["vdim"])
            vec(p + "left.o.b", W, 0.02)
            for n in ("q", "k", "v", "g"):
                mat(p + "right." + n, r["heads"] * r["dim"], W)
            mat(p + "right.o", W, r["heads"] * r["vdim"])
            vec(p + "right.norm", r["heads"] * r["vdim"], 0.05, 1.0)
        else:
            nqk, nv = m["kv_heads"] * m["dim"], m["heads"] * m["vdim"]
            for n, rows in (("q", nqk), ("k", nqk), ("v", nv)):
                mat(p + n, rows, W)
                mat(p + n + ".conv", rows, m["conv"])
            mat(p + "b", m["heads"], W)
            mat(p + "a", m["heads"], W)
            mat(p + "g", nv, W)
            mat(p + "o", W, nv)
            vec(p + "A_log", m["heads"], 0.5)
            vec(p + "dt_bias", m["heads"], 0.5)
            vec(p + "norm", m["vdim"], 0.05, 1.0)
        ff, q = L["mlp"]["ff"], f"l{i}.mlp."
        mat(q + "gate", ff, W)
        mat(q + "up", ff, W)
        mat(q + "down", W, ff)
    vec("final.norm", W, 0.05, 0.0 if nirozen else 1.0)
    mat("head", V, W)
    return out


def _vocab(raw):
    return raw["vocab_size"] if "vocab_size" in raw else raw["vocab"]


def make_tokens(case, seed):
    """One list of token ids for each request: its prompt and the continuation that is fed to it."""
    g = torch.Generator().manual_seed(seed * 2)
    v = _vocab(model_json(case))
    return [torch.randint(0, v, (n + case["new"] - 1,), generator=g).tolist() for n in prompt_lengths(case)]


# ---- the pass ------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    """An engine that has served this kind of batch before (its graphs are captured), the requests' tokens, and room for the logits."""
    raw = model_json(case)
    lens, new = prompt_lengths(case), case["new"]
    pages = sum((n + new) // PAGE + 2 for n in lens) + 8
    engine = Engine.from_tensors(config_from_json(raw), make_weights(case, seed), dtype=case["dtype"], device=DEVICE, page_size=PAGE,
                                 num_pages=pages, max_seqs=case["batch"] + 1, max_batch_tokens=case["budget"])
    engine.enable_graphs()
    state = {"engine": engine, "batch": case["batch"], "steps": None,
             "logits": torch.empty((case["batch"] * new, _vocab(raw)), dtype=torch.float32, device=DEVICE)}
    steps = schedule(case)
    for k in (seed + 7919, seed):                 # other tokens first, to warm up; then the requests' own
        tokens = make_tokens(case, k)
        state["steps"] = [[(i, tokens[i][a:b], [b - a - 1] if want else []) for i, a, b, want in step] for step in steps]
        if k != seed:
            for _ in range(3):
                run(state)
    return state


def run(state):
    engine, logits = state["engine"], state["logits"]
    seqs = [engine.open(i) for i in range(state["batch"])]
    row = 0
    for step in state["steps"]:
        got = engine.step([StepEntry(seqs[i], tokens, want) for i, tokens, want in step])
        n = got.shape[0]
        if n:
            logits[row:row + n].copy_(got)
            row += n
    for seq in seqs:
        engine.close(seq)
    return logits


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------
def work(case):
    """Every step reads the weights it needs once, a request's cached keys or state once, writes its own, and writes its logits."""
    raw = model_json(case)
    es = 4 if case["dtype"] == "float32" else 2
    L = case["layers"]
    V = _vocab(raw)
    nbytes = flops = 0.0
    for step in schedule(case):
        T = sum(b - a for _, a, b, _ in step)
        n_want = sum(1 for s in step if s[3])
        if case["model"].startswith("minicpm4"):
            H, I, nh, nkv, hd = raw["hidden_size"], raw["intermediate_size"], raw["num_attention_heads"], raw["num_key_value_heads"], raw["head_dim"]
            weights = L * ((2 * nh + 2 * nkv) * hd * H + 3 * H * I)
            flops += 2.0 * T * weights
            for _, a, b, _ in step:
                keys = (b * (b + 1) - a * (a + 1)) / 2
                flops += L * 4.0 * nh * hd * keys
                nbytes += L * 2.0 * nkv * hd * b * es
        elif case["model"].startswith("nirozen"):
            H = raw["width"]
            m, f = raw["layers"][0]["mixer"], raw["layers"][0]["mlp"]
            nh, d, e, qr, r = m["heads"], m["dim"], m["vdim"], m["q_rank"], m["kv_rank"]
            dense = H * (qr + r + nh * e) + nh * d * qr + nh * (d + e) * r + nh * e * H + 3 * H * f["shared"]["ff"] + f["router"]["experts"] * H
            one, E, top = 3 * H * f["expert"]["ff"], f["router"]["experts"], f["router"]["top"]
            weights = L * (dense + one * E * (1.0 - (1.0 - top / E) ** T))       # the experts that T tokens' choices name
            flops += 2.0 * T * L * (dense + one * top)
            for _, a, b, _ in step:
                keys = (b * (b + 1) - a * (a + 1)) / 2
                flops += L * 4.0 * nh * r * keys
                nbytes += L * 1.0 * r * b * es
        else:
            H = raw["width"]
            weights = 0.0
            for layer in raw["layers"]:
                m, ff = layer["mixer"], layer["mlp"]["ff"]
                weights += 3 * H * ff
                if layer["type"] == "parallel":
                    c, r, win = m["left"], m["right"], m["left"]["mask"]["size"]
                    weights += H * (2 * c["heads"] + 2 * c["kv_heads"]) * c["dim"] + 5 * H * r["heads"] * r["dim"]
                    for _, a, b, _ in step:
                        full = max(0, b - max(a, win - 1))       # queries that see a whole window
                        lo = b - a - full
                        flops += 4.0 * c["heads"] * c["dim"] * (full * win + lo * (2 * a + lo + 1) / 2)
                        nbytes += 2.0 * c["kv_heads"] * c["dim"] * min(b, win + b - a) * es
                    nh, dk, dv = r["heads"], r["dim"], r["vdim"]
                else:
                    nh, dk, dv = m["heads"], m["dim"], m["vdim"]
                    weights += H * (2 * m["kv_heads"] * dk + 2 * nh * dv + 2 * nh) + H * nh * dv
                nbytes += 2.0 * len(step) * nh * dk * dv * 4
                flops += 4.0 * T * nh * dk * dv
            flops += 2.0 * T * weights
        head = V * (raw["hidden_size"] if "hidden_size" in raw else raw["width"])
        flops += 2.0 * n_want * head
        nbytes += (weights + (head if n_want else 0)) * es + 4.0 * n_want * V
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Measured against `exact`: 1.5e-6 in float32; 0.004 to 0.007 in bfloat16, and 0.009 where a rounding can also turn a choice
    between two nearly equal experts. Two correct implementations differ by about 1.4 times that."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 4e-4}
    if case["model"].startswith("nirozen"):
        return {"rel": 0.03, "max": 0.6}
    return {"rel": 0.02, "max": 0.2}


# ---- the same logits from whole sequences, in float64 ------------------------------------------------------------------------
def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _rotate(x, inv_freq):
    """x [T, heads, d]: entry i is paired with entry i + d/2."""
    a = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None] * inv_freq[None, :]
    c, s = a.cos()[:, None, :], a.sin()[:, None, :]
    u, v = x.chunk(2, dim=-1)
    return torch.cat([u * c - v * s, v * c + u * s], dim=-1)


def _attend(q, k, v, scale, window=None, sink=None):
    """Causal attention of one sequence, q [T, H, d], k and v [T, G, d]; in blocks of queries."""
    T, H, _ = q.shape
    rep = H // k.shape[1]
    out = torch.empty((T, H, v.shape[2]), dtype=q.dtype, device=q.device)
    pos = torch.arange(T, device=q.device)
    block = max(1, (1 << 28) // (H * T))
    for a in range(0, T, block):
        b = min(T, a + block)
        lo = 0 if window is None else max(0, a - window + 1)
        hide = pos[None, lo:b] > pos[a:b, None]
        if window is not None:
            hide = hide | (pos[None, lo:b] <= pos[a:b, None] - window)
        qb = q[a:b].reshape(b - a, -1, rep, q.shape[2]).permute(1, 2, 0, 3).flatten(1, 2)
        s = (qb @ k[lo:b].permute(1, 2, 0)).view(-1, rep, b - a, b - lo) * scale
        s = s.masked_fill(hide, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink.view(-1, rep, 1, 1).expand(-1, -1, b - a, 1)], dim=-1)
        p = torch.softmax(s, dim=-1)[..., :b - lo]
        o = p.flatten(1, 2) @ v[lo:b].permute(1, 0, 2)
        out[a:b] = o.view(-1, rep, b - a, v.shape[2]).permute(2, 0, 1, 3).reshape(b - a, H, -1)
    return out.reshape(T, -1)


def _conv(u, w):
    """Causal convolution over time per channel; the last column of w meets the current token."""
    taps = w.shape[1]
    up = torch.cat([u.new_zeros((taps - 1, u.shape[1])), u])
    return sum(w[:, j] * up[j:j + u.shape[0]] for j in range(taps))


def _silu(z):
    return z * torch.sigmoid(z)


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def _minicpm4_layer(raw, w, i, x, cut):
    H, hd = raw["hidden_size"], raw["head_dim"]
    p, eps, f = f"model.layers.{i}.", raw["rms_norm_eps"], torch.float64
    scale = raw["scale_depth"] / math.sqrt(raw["num_hidden_layers"])
    fac = torch.tensor(raw["rope_scaling"]["short_factor"], dtype=f, device=x.device)
    inv = 1.0 / (fac * raw["rope_theta"] ** (2.0 * torch.arange(hd // 2, dtype=f, device=x.device) / hd))
    h = _rms(x, w(p + "input_layernorm.weight"), eps)
    q, k, v = (h @ w(p + f"self_attn.{n}_proj.weight").t() for n in "qkv")
    o = torch.cat([_attend(_rotate(q[s].view(-1, raw["num_attention_heads"], hd), inv), _rotate(k[s].view(-1, raw["num_key_value_heads"], hd), inv),
                           v[s].view(-1, raw["num_key_value_heads"], hd), hd ** -0.5) for s in cut])
    x = x + scale * (o @ w(p + "self_attn.o_proj.weight").t())
    h = _rms(x, w(p + "post_attention_layernorm.weight"), eps)
    a = _silu(h @ w(p + "mlp.gate_proj.weight").t()) * (h @ w(p + "mlp.up_proj.weight").t())
    return x + scale * (a @ w(p + "mlp.down_proj.weight").t())


def _nirozen_layer(raw, w, i, x, cut):
    L, p, q, eps = raw["layers"][i], f"l{i}.mix.", f"l{i}.mlp.", raw["norm"]["eps"]
    m, f = L["mixer"], L["mlp"]
    h = _rms(x, 1.0 + w(f"l{i}.norm1"), eps)
    qs = _rms(h @ w(p + "dq").t(), w(p + "dq.norm"), eps) @ w(p + "uq").t()
    c = _rms(h @ w(p + "dkv").t(), w(p + "dkv.norm"), eps)
    k, v = c @ w(p + "uk").t(), c @ w(p + "uv").t()
    o = torch.cat([_attend(qs[s].view(-1, m["heads"], m["dim"]), k[s].view(-1, m["heads"], m["dim"]), v[s].view(-1, m["heads"], m["vdim"]),
                           m["scale"], sink=w(p + "sink")) for s in cut])
    x = x + (o * torch.sigmoid(h @ w(p + "g").t())) @ w(p + "o").t()
    h = _rms(x, 1.0 + w(f"l{i}.norm2"), eps)

    def unit(n, r):
        return (_silu(r @ w(n + ".gate").t()) * (r @ w(n + ".up").t())) @ w(n + ".down").t()
    val, idx = torch.topk(h @ w(q + "router").t() + w(q + "router.b"), f["router"]["top"], dim=1)
    wt = torch.softmax(val, dim=1)
    y = unit(q + "shared", h)
    for e in range(f["router"]["experts"]):
        t, j = (idx == e).nonzero(as_tuple=True)
        if t.numel():
            y.index_add_(0, t, wt[t, j][:, None] * unit(f"{q}e{e}", h[t]))
    return x + y


def _decayed(q, k, v, decay):
    """o_t = sum over i <= t of decay^(t-i) (k_i . q_t) v_i, per head."""
    pos = torch.arange(q.shape[0], dtype=q.dtype, device=q.device)
    gap = pos[:, None] - pos[None, :]
    out = torch.empty((q.shape[0], q.shape[1], v.shape[2]), dtype=q.dtype, device=q.device)
    for j in range(q.shape[1]):
        d = torch.where(gap >= 0, torch.pow(decay[j], gap.clamp(min=0)), torch.zeros_like(gap))
        out[:, j] = ((q[:, j] @ k[:, j].t()) * d) @ v[:, j]
    return out


def _delta_rule(q, k, v, beta, g):
    """Per head and token: S = g S; u = beta (v - S^T k); S = S + k u^T; o = S^T q."""
    S = torch.zeros((q.shape[1], q.shape[2], v.shape[2]), dtype=q.dtype, device=q.device)
    out = torch.empty((q.shape[0], q.shape[1], v.shape[2]), dtype=q.dtype, device=q.device)
    for t in range(q.shape[0]):
        S = S * g[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None, :], S)[:, 0])
        S = torch.baddbmm(S, k[t][:, :, None], u[:, None, :])
        out[t] = torch.bmm(q[t][:, None, :], S)[:, 0]
    return out


def _gopitar_layer(raw, w, i, x, cut):
    L, eps, f = raw["layers"][i], raw["norm"]["eps"], torch.float64
    h, m = _rms(x, w(f"l{i}.norm1"), eps), L["mixer"]
    if L["type"] == "parallel":
        c, r, p, n = m["left"], m["right"], f"l{i}.mix.left.", f"l{i}.mix.right."
        qkv = [h @ w(p + a).t() + w(p + a + ".b") for a in "qkv"]
        rot = c["rot"]
        inv = rot["base"] ** (-2.0 * torch.arange(rot["dims"] // 2, dtype=f, device=x.device) / rot["dims"])
        decay = torch.tensor(r["decay"], dtype=f, device=x.device)
        rq, rk, rv = (_silu(h @ w(n + a).t()).view(-1, r["heads"], r["dim"]) for a in "qkv")
        o, s_o = [], []
        for s in cut:
            q, k, v = (_conv(t[s], w(p + a + ".conv")) for t, a in zip(qkv, "qkv"))
            o.append(_attend(_rotate(q.view(-1, c["heads"], c["dim"]), inv), _rotate(k.view(-1, c["kv_heads"], c["dim"]), inv),
                             v.view(-1, c["kv_heads"], c["vdim"]), c["scale"], window=c["mask"]["size"]))
            s_o.append(_decayed(rq[s], rk[s], rv[s], decay).flatten(1))
        gate = torch.sigmoid(h @ w(p + "g").t()).repeat_interleave(c["vdim"], dim=1)
        left = (torch.cat(o) * gate) @ w(p + "o").t() + w(p + "o.b")
        right = (_rms(torch.cat(s_o), w(n + "norm"), eps) * torch.sigmoid(h @ w(n + "g").t())) @ w(n + "o").t()
        x = x + m["left_scale"] * left + m["right_scale"] * right
    else:
        p, H, G, d = f"l{i}.mix.", m["heads"], m["kv_heads"], m["dim"]
        qkv = [h @ w(p + a).t() for a in "qkv"]
        beta = torch.sigmoid(h @ w(p + "b").t())
        g = torch.exp(-torch.exp(w(p + "A_log")) * torch.nn.functional.softplus(h @ w(p + "a").t() + w(p + "dt_bias")))
        o = []
        for s in cut:
            q, k, v = (_silu(_conv(t[s], w(p + a + ".conv"))) for t, a in zip(qkv, "qkv"))
            q, k = (_unit(t.view(-1, G, d)).repeat_interleave(H // G, dim=1) for t in (q, k))
            o.append(_delta_rule(q * d ** -0.5, k, v.view(-1, H, m["vdim"]), beta[s], g[s]))
        o = _rms(torch.cat(o), w(p + "norm"), eps) * _silu(h @ w(p + "g").t()).view(-1, H, m["vdim"])
        x = x + o.flatten(1) @ w(p + "o").t()
    h, q = _rms(x, w(f"l{i}.norm2"), eps), f"l{i}.mlp."
    return x + (_gelu(h @ w(q + "gate").t()) * (h @ w(q + "up").t())) @ w(q + "down").t()


def exact(case, seed):
    """`run`'s logits from whole sequences in float64, rows in the order of the pass."""
    raw, tensors, f = model_json(case), make_weights(case, seed), torch.float64

    def w(name):
        return tensors[name].to(f)
    tokens = make_tokens(case, seed)
    cut, at = [], 0
    for t in tokens:                              # each request's rows in the one long matrix
        cut.append(slice(at, at + len(t)))
        at += len(t)
    ids = [torch.tensor(t, device=DEVICE) for t in tokens]
    if case["model"].startswith("minicpm4"):
        x = w("model.embed_tokens.weight")[torch.cat(ids)] * raw["scale_emb"]
        layer, norm, head = _minicpm4_layer, w("model.norm.weight"), w("lm_head.weight" if "lm_head.weight" in tensors else "model.embed_tokens.weight")
        eps, scale = raw["rms_norm_eps"], raw["dim_model_base"] / raw["hidden_size"]
    else:
        W, eps, scale = raw["width"], raw["norm"]["eps"], 1.0
        x = w("embed")[torch.cat(ids)]
        norm, head = w("final.norm"), w("head")
        layer = _gopitar_layer
        if case["model"].startswith("nirozen"):
            layer, norm, b = _nirozen_layer, 1.0 + norm, raw["embedding"]["bigram"]
            rows, waves = [], []
            for t in ids:
                prev = (t[:-1] * b["mul_prev"] + t[1:] * b["mul_cur"]) % b["buckets"]
                rows.append(torch.cat([prev.new_full((1,), b["buckets"]), prev]))
                a = torch.arange(len(t), dtype=f, device=DEVICE)[:, None] * 10000.0 ** (-2.0 * torch.arange(W // 2, dtype=f, device=DEVICE) / W)
                waves.append(torch.stack([a.sin(), a.cos()], dim=-1).flatten(1))
            x = x + w("bigram")[torch.cat(rows)] + torch.cat(waves)
    for i in range(case["layers"]):
        x = layer(raw, w, i, x, cut)
    wanted = [cut[i].start + b - 1 for step in schedule(case) for i, _, b, want in step if want]
    out = _rms(x[torch.tensor(wanted, device=DEVICE)], norm, eps) @ head.t() * scale
    cap = raw.get("logit_softcap")
    return cap * torch.tanh(out / cap) if cap else out
