"""The work that users of this package have it do, as cases that can be timed and checked.

Three kinds, each through the calls a program makes:

* `linear` and `moe`: one call of the ternary layer (`BitLinear.forward`) or of the expert feed-forward
  (`tbl_moe_forward`) on activations that lie on the GPU, as a runtime that owns the rest of the model calls them;
* `hybrid`: a session of the ternary Mamba-2 / attention hybrid (`DecodeEngine`): empty caches, the prompt token by
  token, then the reply, the step replayed from its CUDA graph;
* `stack`: a request to a layer-stack model (`StackEngine`): open a slot per sequence, feed the prompts, decode the reply
  of all sequences together, close the slots.  The reply's tokens are given (as in trace replay), so that every run sees
  the same tokens whatever the rounding of its logits.

`exact` restates `linear`, `moe` and `stack` in 64 bits with plain torch.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from reimagined_b200 import capi
from reimagined_b200.bitlinear import BitLinear, BitLinearPackedState
from reimagined_b200.decode import D768_L16, DecodeEngine, synthetic_params
from reimagined_b200.stack import StackEngine, synthetic_weights
from reimagined_b200.stack_shapes import CONFIGS


def linear(m, k, n, int8, exact_mode, bias):
    return {"kind": "linear", "m": m, "k": k, "n": n, "int8": int8, "exact_mode": exact_mode, "bias": bias}


def stack(model, dtype, width, layers, sequences, prompt, reply, lockstep=False):
    return {"kind": "stack", "model": model, "dtype": dtype, "width": width, "layers": layers, "sequences": sequences, "prompt": prompt, "reply": reply,
            "lockstep": lockstep}


def listed():
    return [
        # one token through a projection of the D768 hybrid (RMS-normed input, magnitude, bias): the smallest call there is
        {"name": "linear_small", **linear(1, 768, 3072, True, False, True)},
        # one token through the widest layer of the sweep: weight streaming
        {"name": "linear_token", **linear(1, 16384, 16384, True, True, False)},
        # a long prompt through a wide layer: int8 tensor-core GEMM behind the row quantiser
        {"name": "linear_prompt", **linear(8192, 8192, 8192, True, True, False)},
        # a batch of tokens through the experts of a mixture-of-experts block, 2-bit weights alone
        {"name": "moe_batch", "kind": "moe", "m": 256, "dim": 2048, "hidden": 5632, "experts": 8, "top": 2},
        # one user of the hybrid: the prompt goes token by token, then the reply
        {"name": "hybrid_chat", "kind": "hybrid", "batch": 1, "prompt": 224, "reply": 32},
        # many users of the hybrid at once
        {"name": "hybrid_batch", "kind": "hybrid", "batch": 64, "prompt": 72, "reply": 24},
        # one user of a layer-stack model: a medium prompt, decoding at batch one
        {"name": "guselix_chat", **stack("guselix", "bfloat16", 2048, 8, 1, 512, 32)},
        # many users at once: short prompts in lockstep, decoding at batch 64
        {"name": "guselix_batch", **stack("guselix", "bfloat16", 4096, 4, 64, 16, 16, lockstep=True)},
        # a long document of ragged length, and the first tokens of the answer
        {"name": "guselix_document", **stack("guselix", "bfloat16", 2048, 8, 1, 6001, 2)},
        # the same in plain fp32, which those choose who compare implementations: a short prompt and reply
        {"name": "guselix_fp32", **stack("guselix", "float32", 2048, 4, 1, 251, 16)},
        # a long document through the design with grouped differential attention
        {"name": "goguvik_document", **stack("goguvik", "bfloat16", 4096, 4, 1, 7777, 2)},
        # some users, each with some history of their own length, decoded together
        {"name": "goguvik_batch", **stack("goguvik", "bfloat16", 2048, 8, 8, 900, 32)},
    ]


def spread(rng, low, high):
    """A whole number whose logarithm is spread evenly."""
    return min(high, int(math.exp(rng.uniform(math.log(low), math.log(high + 1)))))


def draw(rng):
    kind = rng.choice(("linear", "linear", "moe", "hybrid", "stack", "stack", "stack", "stack"))
    if kind == "linear":
        m, step = spread(rng, 1, 8192), rng.choice((16, 256, 256, 256))
        k, n = (spread(rng, 768, 16384) for _ in range(2))
        k = k // step * step
        n = max(64, min(n, 8192 ** 3 // (m * k)))
        return linear(m, k, n, rng.random() < 0.6, rng.random() < 0.5, rng.random() < 0.5)
    if kind == "moe":
        experts = rng.choice((4, 8, 16))
        return {"kind": "moe", "m": spread(rng, 8, 512), "dim": 256 * rng.randint(3, 8), "hidden": 256 * rng.randint(4, 22), "experts": experts,
                "top": rng.randint(1, 2)}
    if kind == "hybrid":
        return {"kind": "hybrid", "batch": spread(rng, 1, 64), "prompt": spread(rng, 8, 72), "reply": rng.randint(4, 24)}
    model, dtype = rng.choice(("guselix", "goguvik")), rng.choice(("bfloat16", "bfloat16", "bfloat16", "float32"))
    width, layers = rng.choice(((1024, 8), (1536, 8), (2048, 8), (3072, 4), (4096, 4)))
    if dtype == "float32":
        layers = 4
    rows = 6000 if dtype == "bfloat16" else 256
    sequences = spread(rng, 1, 64 if dtype == "bfloat16" else 8)
    prompt = spread(rng, 24, rows // sequences)
    lockstep = sequences > 8 or rng.random() < 0.3
    return stack(model, dtype, width, layers, sequences, prompt, rng.randint(1, 12 if dtype == "float32" else 24), lockstep)


# ---- weights and inputs -------------------------------------------------------------------------------------------------
def generator(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)


def packed_layer(gen, k, n, bias, exact_mode, int8):
    """A ternary layer as an import of a checkpoint leaves it: a third of the weights zero, and its codes as int8 [n, k]."""
    codes = torch.randint(0, 3, (n * k // 16, 16), generator=gen, device="cuda", dtype=torch.int32)
    words = (codes << (2 * torch.arange(16, device="cuda", dtype=torch.int32))).sum(dim=1, dtype=torch.int32)
    layer = BitLinear(k, n, bias)
    layer.set_exact_linear_mode(exact_mode)
    draws = torch.randn(2, n, generator=gen, device="cuda").cpu().numpy()
    layer.import_packed_state(BitLinearPackedState(
        k, n, bias, 0.016, words.cpu().numpy().view(np.uint32), (1.0 + 0.1 * draws[0]).astype(np.float32),
        (0.1 * draws[1]).astype(np.float32) if bias else np.zeros(0, np.float32)))
    return layer.to("cuda", with_int8=int8), codes


def activations(gen, rows, width):
    """Rows of unequal size, as a residual stream has them."""
    x = torch.randn(rows, width, generator=gen, device="cuda")
    return x * (0.5 + torch.rand(rows, 1, generator=gen, device="cuda"))


def routing(gen, case):
    """Routing weights [rows, experts]: the `top` experts of a row, their weights adding up to one."""
    scores = torch.rand(case["m"], case["experts"], generator=gen, device="cuda")
    top = scores.topk(case["top"], dim=1)
    out = torch.zeros_like(scores)
    return out.scatter_(1, top.indices, top.values / top.values.sum(dim=1, keepdim=True))


@functools.lru_cache(maxsize=1)
def hybrid_params():
    return synthetic_params(D768_L16, 1)


def lengths(case):
    """Prompt lengths: all alike in lockstep, else every sequence has its own."""
    return [case["prompt"] if case["lockstep"] else case["prompt"] - (17 * i % 64) * case["prompt"] // 256 for i in range(case["sequences"])]


def token_ids(case, seed, vocab):
    """Per sequence the prompt's and the reply's token ids."""
    rng = np.random.default_rng(seed)
    return [rng.integers(0, vocab, n + case["reply"]).tolist() for n in lengths(case)]


def stack_model(case, seed):
    cfg = CONFIGS[case["model"]](case["width"], case["layers"])
    return cfg, synthetic_weights(cfg, seed, rank=case["width"] // 32, device="cuda")


def prepare(case, seed):
    gen, kind = generator(seed), case["kind"]
    if kind == "linear":
        layer, _ = packed_layer(gen, case["k"], case["n"], case["bias"], case["exact_mode"], case["int8"])
        return {"kind": kind, "layer": layer, "x": activations(gen, case["m"], case["k"])}
    if kind == "moe":
        m, dim, hidden, experts = case["m"], case["dim"], case["hidden"], case["experts"]
        layers = [packed_layer(gen, *shape, True, False, False)[0] for shape in [(dim, hidden)] * experts + [(hidden, dim)] * experts]
        size = capi.lib().tbl_moe_workspace_bytes(m, dim, hidden, experts, case["top"])
        return {"kind": kind, "case": case, "layers": layers, "views": (capi.LinearView * len(layers))(*(a.prepare_gpu_decode_view() for a in layers)),
                "x": activations(gen, m, dim), "routing": routing(gen, case), "out": torch.empty(m, dim, device="cuda"),
                "workspace": torch.empty(size, dtype=torch.uint8, device="cuda")}
    if kind == "hybrid":
        total = case["prompt"] + case["reply"]
        engine = DecodeEngine(hybrid_params(), batch=case["batch"], capacity=total)
        ids = torch.randint(0, engine.vocab, (total, case["batch"]), generator=gen, device="cuda", dtype=torch.int32)
        engine.step(ids[0])
        engine.capture()
        return {"kind": kind, "engine": engine, "ids": list(ids), "prompt": case["prompt"]}
    cfg, weights = stack_model(case, seed)
    engine = StackEngine(cfg, weights, case["dtype"], slots=case["sequences"], capacity=case["prompt"] + case["reply"])
    ids, n = token_ids(case, seed, cfg["vocab"]), lengths(case)
    return {"kind": kind, "engine": engine, "prompts": [row[:k] for row, k in zip(ids, n)], "lockstep": case["lockstep"],
            "reply": [[[row[k + t]] for row, k in zip(ids, n)] for t in range(case["reply"])]}


# ---- one pass -------------------------------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["layer"].forward(state["x"])
    if kind == "moe":
        c, ws = state["case"], state["workspace"]
        capi.check(capi.lib().tbl_moe_forward(
            state["views"], state["routing"].data_ptr(), state["x"].data_ptr(), c["m"], c["dim"], c["hidden"], c["experts"], c["top"], 1, 0,
            state["out"].data_ptr(), ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream), "tbl_moe_forward")
        return state["out"]
    engine = state["engine"]
    if kind == "hybrid":
        engine.reset()
        logits = [engine.step(ids) if i + 1 < state["prompt"] else engine.step(ids).clone() for i, ids in enumerate(state["ids"])]
        return logits[state["prompt"] - 1:]
    slots = [engine.open() for _ in state["prompts"]]
    if state["lockstep"]:
        logits = [engine.step(slots, state["prompts"])]
    else:
        logits = [engine.feed(s, p) for s, p in zip(slots, state["prompts"])]
    logits += [engine.step(slots, tokens) for tokens in state["reply"]]
    for s in slots:
        engine.close(s)
    return logits if state["lockstep"] else [torch.cat(logits[:len(slots)])] + logits[len(slots):]


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------
def matrices(case):
    """Numbers in the weight matrices that every token goes through, and in the table that is embedding and head."""
    w, ff, v = case["width"], 3 * case["width"], 32000
    mlp = 3 * w * ff
    if case["model"] == "guselix":
        delta = 5 * w * w + 2 * w * (w // 32) + w * w
        heads, q = w // 128, 3 * w // 8
        latent = w * (q + 576) + q * heads * 192 + 512 * heads * 256 + 2 * w * w
        return sum((latent if i % 4 == 3 else delta) + mlp for i in range(case["layers"])), w * v
    kv = max(1, w // 512) * 256
    return sum(3 * w * w + (w * kv if i % 2 == 0 else 0) + mlp for i in range(case["layers"])), w * v


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": n * k / 4 + 4 * m * (k + n), "flops": 2 * m * n * k}
    if kind == "moe":
        m, d, h = case["m"], case["dim"], case["hidden"]
        return {"bytes": case["experts"] * 2 * d * h / 4 + 8 * m * d, "flops": 4 * m * case["top"] * d * h}
    if kind == "hybrid":
        steps, batch = case["prompt"] + case["reply"], case["batch"]
        state = 8 * 16 * 1536 * 16 + 8 * 16 * 3 * 1568
        cache = 2 * 2 * 4 * 768 * (steps + 1) / 2
        return {"bytes": steps * (24.0e6 + batch * (state + cache + 4 * 32000)), "flops": 2.0 * 96.04e6 * steps * batch}
    body, head = matrices(case)
    n, reply, heads = lengths(case), case["reply"], case["width"] // 128
    tokens, steps = sum(n) + reply * len(n), reply + (1 if case["lockstep"] else len(n))
    nbytes = steps * 2 * (body + head) + 4 * 32000 * len(n) * (reply + 1)
    flops = 2 * body * tokens + 2 * head * len(n) * (reply + 1)
    pairs = sum((k + reply) * (k + reply + 1) / 2 for k in n)
    cached = sum(reply * (k + reply / 2) for k in n)
    size = 2 if case["dtype"] == "bfloat16" else 4
    if case["model"] == "guselix":
        attending = sum(i % 4 == 3 for i in range(case["layers"]))
        recurrent = case["layers"] - attending
        nbytes += recurrent * 8 * heads * 128 * 128 * len(n) * (reply + 1) + attending * size * 576 * (cached + tokens)
        flops += recurrent * 10 * heads * 128 * 128 * tokens + attending * 2 * heads * pairs * 320
    else:
        nbytes += case["layers"] * size * max(1, heads // 4) * 256 * (cached + tokens)
        flops += case["layers"] * 2 * heads * 2 * pairs * 192
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "linear":
        # the sums are whole numbers: without the input norm only the last products round; with it a sum of squares in
        # another order can move a value by a step of the 8-bit quantiser, 1 / (30 sqrt(k)) of its row
        return {"rel": 4e-7, "max": 4e-6} if case["exact_mode"] else {"rel": 3e-3, "max": 2e-2}
    if case["kind"] == "moe":
        return {"rel": 3e-3, "max": 4e-2}
    if case["kind"] == "hybrid":
        return {"rel": 2e-2, "max": 4e-1}
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    # measured against 64 bits: 0.004 to 0.009 (the delta rule's head norm widens rounding), and 0.002 to 0.003
    return {"rel": 2e-2, "max": 2e-1} if case["model"] == "guselix" else {"rel": 1e-2, "max": 1e-1}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------------
def ternary_rows(layer, codes, x, k, n, exact_mode):
    """A ternary layer on rows x (64 bits): the 8-bit codes as the quantiser defines them, in 32 bits; all sums in 64."""
    if not exact_mode:
        x = x / torch.sqrt((x * x).mean(dim=1, keepdim=True) + 1e-6)
    x = x.float()
    top = x.abs().amax(dim=1, keepdim=True) + 1e-8
    levels = torch.full_like(top, 127.0)         # a tensor: division by a number is a product with its reciprocal
    q = torch.round(x * (levels / top))
    scale = top / levels * torch.tensor(layer.weight_scale, dtype=torch.float32, device="cuda")
    w = codes.reshape(n, k).double() - 1.0
    y = q.double() @ w.t() * scale.double()
    if not exact_mode:
        y = y * torch.from_numpy(layer.magnitude).cuda().double()
    return y + torch.from_numpy(layer.bias).cuda().double() if layer.use_bias else y


def exact(case, seed):
    kind = case["kind"]
    if kind == "linear":
        gen = generator(seed)
        layer, codes = packed_layer(gen, case["k"], case["n"], case["bias"], case["exact_mode"], case["int8"])
        return ternary_rows(layer, codes, activations(gen, case["m"], case["k"]).double(), case["k"], case["n"], case["exact_mode"])
    if kind == "moe":
        gen, d, h, experts = generator(seed), case["dim"], case["hidden"], case["experts"]
        both = [packed_layer(gen, *shape, True, False, False) for shape in [(d, h)] * experts + [(h, d)] * experts]
        x = activations(gen, case["m"], d).double()
        weight, out = routing(gen, case).double(), torch.zeros_like(x)
        for e in range(experts):
            at = weight[:, e].nonzero().squeeze(1)
            if at.numel():
                hidden = ternary_rows(*both[e], x[at], d, h, False).clamp(min=0.0) ** 2
                out[at] += weight[at, e:e + 1] * ternary_rows(*both[experts + e], hidden, h, d, False)
        return out
    if kind == "hybrid":
        # every one of its 107 layers rounds its input to 8 bits, a hundred steps feed the states: in 64 bits other values
        # fall on the other side of a rounding step than in 32, so that there is no one right result to compare with
        return None
    return exact_stack(case, seed)


def rms(x, w, eps):
    y = x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)
    return y if w is None else y * w


def causal(q, k, v, scale):
    """Softmax attention of every token over those up to it; q, k [heads, tokens, .], v [heads, tokens, .]."""
    out = torch.empty(q.shape[0], q.shape[1], v.shape[2], dtype=torch.float64, device="cuda")
    for lo in range(0, q.shape[1], 512):
        hi = min(lo + 512, q.shape[1])
        s = q[:, lo:hi] @ k[:, :hi].transpose(1, 2) * scale
        late = torch.arange(hi, device="cuda")[None, :] > torch.arange(lo, hi, device="cuda")[:, None]
        out[:, lo:hi] = s.masked_fill_(late, -math.inf).softmax(dim=-1) @ v[:, :hi]
    return out


def exact_delta(h, P, m, eps):
    """Generalized delta rule; h [sequences, tokens, width]."""
    S, T, H, d = h.shape[0], h.shape[1], m["heads"], m["dim"]
    split = lambda x: x.reshape(S, T, H, d).permute(1, 0, 2, 3).reshape(T, S * H, d).contiguous()
    r, k, v = (split(h @ P(n).t()) for n in ("r", "k", "v"))
    w = split(torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ P("w1").t()) @ P("w2").t() + P("w0"))))
    a = split(torch.sigmoid(h @ P("a").t() + P("a.b")))
    u = k / torch.sqrt((k * k).sum(dim=-1, keepdim=True) + 1e-6)
    left, state, o = torch.stack((-a * u, k), dim=3), torch.zeros(S * H, d, d, dtype=torch.float64, device="cuda"), torch.empty_like(r)
    right = torch.stack((v, v), dim=2)
    for t in range(T):
        right[t, :, :1] = u[t, :, None] @ state
        state.mul_(w[t, :, :, None]).baddbmm_(left[t], right[t])
        o[t] = (r[t, :, None] @ state)[:, 0]
    o = rms(o, None, eps).reshape(T, S, H * d).transpose(0, 1) * P("norm")
    return (o * torch.sigmoid(h @ P("g").t())) @ P("o").t()


def exact_latent(h, P, m, eps):
    S, T, H, d, rd, vd, R = h.shape[0], h.shape[1], m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
    freq = m["rot"]["base"] ** (-2.0 * torch.arange(rd // 2, dtype=torch.float64, device="cuda") / rd)
    angle = torch.arange(T, dtype=torch.float64, device="cuda")[:, None] * freq

    def rotate(x):           # [tokens, heads, rd]
        u, v, c, s = x[..., :rd // 2], x[..., rd // 2:], angle.cos()[:, None], angle.sin()[:, None]
        return torch.cat((u * c - v * s, v * c + u * s), dim=-1)

    out = torch.empty(S, T, H * vd, dtype=torch.float64, device="cuda")
    for s in range(S):
        q = (rms(h[s] @ P("dq").t(), P("dq.norm"), eps) @ P("uq").t()).reshape(T, H, d + rd)
        kv = h[s] @ P("dkv").t()
        c = rms(kv[:, :R], P("dkv.norm"), eps)
        keys = torch.cat(((c @ P("uk").t()).reshape(T, H, d), rotate(kv[:, None, R:]).expand(T, H, rd)), dim=2).transpose(0, 1)
        q = torch.cat((q[..., :d], rotate(q[..., d:])), dim=2).transpose(0, 1)
        o = causal(q, keys, (c @ P("uv").t()).reshape(T, H, vd).transpose(0, 1), m["scale"])
        out[s] = o.transpose(0, 1).reshape(T, H * vd)
    return (out * torch.sigmoid(h @ P("g").t())) @ P("o").t()


def exact_attention(h, P, m, eps, cache):
    S, T, H, G, d, vd = h.shape[0], h.shape[1], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    if m.get("kv_from") is None:
        cache = ((h @ P("k").t() + P("k.b")).reshape(S, T, G, 2, d), (h @ P("v").t() + P("v.b")).reshape(S, T, G, vd))
    steps = torch.floor((torch.arange(T, dtype=torch.float64, device="cuda") + 1) / m["q_temp"]["every"])
    warm = 1.0 + m["q_temp"]["coef"] * torch.log(steps + 1.0)
    lam = torch.exp((P("lq1") * P("lk1")).sum()) - torch.exp((P("lq2") * P("lk2")).sum()) + m["diff"]
    q = (h @ P("q").t() + P("q.b")).reshape(S, T, H, 2, d) * warm[:, None, None, None]
    out = torch.empty(S, T, H, vd, dtype=torch.float64, device="cuda")
    for s in range(S):
        for g in range(G):
            at = slice(g * (H // G), (g + 1) * (H // G))
            a = [causal(q[s, :, at, i].transpose(0, 1), cache[0][s, :, g, i].expand(H // G, T, d), cache[1][s, :, g].expand(H // G, T, vd), m["scale"])
                 for i in range(2)]
            out[s, :, at] = (rms(a[0] - lam * a[1], None, eps) * (1.0 - m["diff"])).transpose(0, 1)
    o = out.reshape(S, T, H * vd) * torch.sigmoid(h @ P("g").t())
    return o @ P("o").t() + P("o.b"), cache


def exact_stack(case, seed):
    """All sequences at once, the shorter ones filled up behind their end (which nothing before it sees)."""
    cfg, weights = stack_model(case, seed)
    ids, n = token_ids(case, seed, cfg["vocab"]), lengths(case)
    tokens = torch.zeros(len(ids), max(map(len, ids)), dtype=torch.int64)
    for row, t in zip(tokens, ids):
        row[:len(t)] = torch.tensor(t)
    W, eps = (lambda name: weights[name].double()), cfg["norm"]["eps"]
    x = W("embed")[tokens.cuda()]
    if case["model"] == "guselix":
        xs = [x]
        for i, layer in enumerate(cfg["layers"]):
            p, mixer = f"l{i}.", exact_delta if layer["type"] == "general_delta" else exact_latent
            x = x + mixer(rms(x, W(p + "norm1"), eps), lambda name: W(p + "mix." + name), layer["mixer"], eps)
            h, part = rms(x, W(p + "norm2"), eps), lambda name: h @ W(p + "mlp." + name).t() + W(p + "mlp." + name + ".b")
            x = x + (torch.nn.functional.silu(part("gate")) * part("up")) @ W(p + "mlp.down").t() + W(p + "mlp.down.b")
            xs.append(x)
            x = sum(c * y for c, y in zip(W(p + "dwa"), xs))
        norm = lambda y: rms(y, W("final.norm"), eps)
    else:
        tanh = lambda y, name: torch.tanh(W(name + ".alpha") * y) * W(name) + W(name + ".b")
        xs, caches = [x] * cfg["streams"], []

        def update(xs, hc, sublayer):
            y = sublayer(sum(c * z for c, z in zip(W(hc + "in"), xs)))
            mix = W(hc + "mix")
            return [sum(mix[s, t] * xs[s] for s in range(len(xs))) + W(hc + "out")[t] * y for t in range(len(xs))]

        for i, layer in enumerate(cfg["layers"]):
            p, m = f"l{i}.", layer["mixer"]

            def attend(z):
                o, kv = exact_attention(tanh(z, p + "norm1"), lambda name: W(p + "mix." + name), m, eps, caches[m["kv_from"]] if "kv_from" in m else None)
                caches.append(kv)
                return o

            def feed_forward(z):
                h = tanh(z, p + "norm2")
                act = torch.nn.functional.gelu(h @ W(p + "mlp.gate").t(), approximate="tanh")
                return (act * (h @ W(p + "mlp.up").t())) @ W(p + "mlp.down").t()

            xs = update(xs, p + "hc1.", attend)
            xs = update(xs, p + "hc2.", feed_forward)
        x, norm = sum(xs), lambda y: tanh(y, "final.norm")
    at = torch.tensor([[k - 1 + t for k in n] for t in range(case["reply"] + 1)], device="cuda")
    rows = x[torch.arange(len(n), device="cuda")[None, :], at]
    logits = norm(rows) @ W("embed").t()
    return list(logits)
