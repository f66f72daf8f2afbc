"""What a program built on this library has it do, as cases that can be timed and compared.

A case is a model (layers of a configuration that the benchmark names, fewer of them), what is done with it, how many
sequences there are and how long they are:

  decode    one token for each of ``batch`` sequences that hold up to ``length`` tokens: a step of generation
  prompt    ``batch`` prompts of up to ``length`` tokens in one step, then their sequences are released
  turn      ``batch`` sequences that hold up to ``length`` tokens go on by ``new`` tokens each in one step: the next turn of
            a conversation, or the last piece of a long prompt
  request   ``batch`` prompts of up to ``length`` tokens in one step, then ``new`` single-token steps, then release: a whole
            request (designs whose sequences carry a state cannot be rewound, so their decoding is measured so)

Models: ``moe-2048`` (bfloat16), ``moe-2048-fp32`` (true 32-bit, a window on the last layer), ``moe-3584`` (grouped heads, 64
experts of which a token takes 8) and ``kulanex-2048`` (windowed attention beside an mLSTM memory, the delta rule with a
decay a channel, sigmoid-scored experts).  Results are the float32 logits at the last place of every sequence.

The tokens are given, as when a recorded text is replayed, so that the work does not hang on a sampled token.  Weights
are random.  A trained layer changes the residual stream by a small part of it; with all tensors drawn alike the stream
would be whatever the last layer wrote, so the embedding is drawn wider than the rest.
"""
from __future__ import annotations

import math

import torch

import moe_b200
from moe_b200.models import DecoderModel
from moe_b200.weights import TensorDictStore

DEV = "cuda"
F8 = torch.float64

MOE_2048 = dict(
    architectures=["Qwen2MoeForCausalLM"], model_type="qwen2_moe", num_hidden_layers=6, hidden_size=2048,
    num_attention_heads=16, num_key_value_heads=16, head_dim=128, num_experts=60, num_experts_per_tok=4,
    moe_intermediate_size=1408, shared_expert_intermediate_size=5632, intermediate_size=5632, norm_topk_prob=False,
    decoder_sparse_step=1, mlp_only_layers=[], vocab_size=151936, rope_theta=1e6, rms_norm_eps=1e-6,
    use_sliding_window=False, tie_word_embeddings=False, max_position_embeddings=32768,
)
MODELS = {
    "moe-2048": (MOE_2048, "bfloat16"),
    # (the layers before ``max_window_layers`` see every position, the others a window)
    "moe-2048-fp32": (dict(MOE_2048, num_hidden_layers=3, use_sliding_window=True, sliding_window=4096, max_window_layers=2),
                      "float32"),
    "moe-3584": (dict(MOE_2048, num_hidden_layers=3, hidden_size=3584, num_attention_heads=28, num_key_value_heads=4,
                      num_experts=64, num_experts_per_tok=8, moe_intermediate_size=2560,
                      shared_expert_intermediate_size=20480, intermediate_size=18944), "bfloat16"),
}
_PARALLEL = {
    "type": "parallel",
    "mixer": {
        "left": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "conv": 4, "scale": 128 ** -0.5,
                 "mask": {"size": 1024, "keep_first": 16},
                 "rot": {"dims": 64, "base": 1e6, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 4096}}},
        "right": {"heads": 16, "dim": 64, "vdim": 128, "gate_cap": 15.0}, "left_scale": 0.5, "right_scale": 0.5},
}
_DELTA = {"type": "channel_delta", "mixer": {"heads": 16, "kv_heads": 16, "dim": 128, "vdim": 128, "conv": 4}}
RANK, E_KUL = 128, 16          # the width of the delta layers' narrow projections; experts a layer
_EXPERTS = {"kind": "moe", "router": {"experts": E_KUL, "top": 2}, "expert": {"ff": 1408}}
MODELS["kulanex-2048"] = ({
    "architecture": "Kulanex", "vocab": 32768, "width": 2048, "norm": {"eps": 1e-5}, "residual_mult": 0.5,
    "layers": [dict(m, mlp=_EXPERTS) for m in (_DELTA, _PARALLEL, _DELTA, _PARALLEL)]}, "bfloat16")


def _case(model, do, batch, length, new=0, unequal=False, **more):
    return dict(more, model=model, do=do, batch=batch, length=length, new=new, unequal=unequal)


def listed():
    return [
        # one user waits for the next token: every launch and every wait between two kernels counts
        _case("moe-2048", "decode", 1, 512, name="decode-1"),
        # the benchmark's headline: a small batch, sequences of their own lengths
        _case("moe-2048", "decode", 8, 900, unequal=True, name="decode-8"),
        # a busy server: every expert is read, and each sequence's keys and values
        _case("moe-2048", "decode", 64, 512, name="decode-64"),
        # the larger shape: seven query heads on a key head, long sequences of unequal length
        _case("moe-3584", "decode", 16, 2048, unequal=True, name="decode-16-wide"),
        # a few short questions that arrive together
        _case("moe-2048", "prompt", 3, 61, unequal=True, name="prompts-short"),
        # one prompt of ordinary length, as the benchmark's prefill
        _case("moe-2048", "prompt", 1, 2048, name="prompt-2048"),
        # a document: attention over itself is a good part of the work
        _case("moe-2048", "prompt", 1, 8192, name="prompt-8192"),
        # conversations that go on: some new tokens behind a cache that is already long
        _case("moe-2048", "turn", 4, 1500, new=100, unequal=True, name="turn-100"),
        # the 32-bit path, which scores and checks the other one: prompts, then a step of decoding
        _case("moe-2048-fp32", "prompt", 2, 4000, unequal=True, name="fp32-prompts"),
        _case("moe-2048-fp32", "decode", 8, 3000, unequal=True, name="fp32-decode-8"),
        # a design with recurrent mixers: a prompt, whose scans are chains over its tokens, and whole short requests
        _case("kulanex-2048", "prompt", 1, 2048, name="recurrent-prompt"),
        _case("kulanex-2048", "request", 8, 200, new=16, unequal=True, name="recurrent-requests"),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """A case of the listed ones' ranges.  The tokens that a batch holds are bounded, so that none costs more than the
    largest listed case."""
    kind = rng.choice(["decode", "decode", "wide", "prompt", "prompt", "turn", "fp32-prompt", "fp32-decode", "recurrent-prompt",
                       "recurrent-request"])
    unequal = rng.random() < 0.6
    if kind == "decode":
        batch = _log(rng, 1, 96)
        return _case("moe-2048", "decode", batch, _log(rng, 40, min(8000, 40000 // batch)), unequal=unequal)
    if kind == "wide":
        batch = _log(rng, 1, 32)
        return _case("moe-3584", "decode", batch, _log(rng, 100, min(4000, 20000 // batch)), unequal=unequal)
    if kind == "prompt":
        batch = _log(rng, 1, 8)
        return _case("moe-2048", "prompt", batch, _log(rng, 8, 8000 // batch), unequal=unequal)
    if kind == "turn":
        batch = _log(rng, 1, 8)
        return _case("moe-2048", "turn", batch, _log(rng, 60, 8000 // batch), new=_log(rng, 2, 2000 // batch), unequal=unequal)
    if kind == "fp32-prompt":
        batch = _log(rng, 1, 6)
        return _case("moe-2048-fp32", "prompt", batch, _log(rng, 8, 4000 // batch), unequal=unequal)
    if kind == "fp32-decode":
        batch = _log(rng, 1, 12)
        return _case("moe-2048-fp32", "decode", batch, _log(rng, 40, min(4000, 24000 // batch)), unequal=unequal)
    batch = _log(rng, 1, 8)
    if kind == "recurrent-prompt":
        return _case("kulanex-2048", "prompt", batch, _log(rng, 16, 6000 // batch), unequal=unequal)
    return _case("kulanex-2048", "request", batch, _log(rng, 8, 2000 // batch), new=_log(rng, 2, 24), unequal=unequal)


# ---- inputs ---------------------------------------------------------------------------------------------------------
def _lengths(case):
    """Tokens of every sequence before the timed step (or of its prompt): all alike, or from ``length`` down to about a
    quarter of it."""
    B, n = case["batch"], case["length"]
    return [max(1, round(n * (1 - 0.77 * i / max(B - 1, 1)))) if case["unequal"] else n for i in range(B)]


def _tokens(case, seed):
    """Per sequence: its tokens, those of the timed step included."""
    cfg, _ = MODELS[case["model"]]
    vocab = cfg.get("vocab_size") or cfg["vocab"]
    more = {"decode": 1, "prompt": 0, "turn": case["new"], "request": case["new"]}[case["do"]]
    g = torch.Generator().manual_seed(seed)
    return [torch.randint(0, vocab, (n + more,), generator=g).tolist() for n in _lengths(case)]


def _weights(case, seed):
    cfg, dtype = MODELS[case["model"]]
    g = torch.Generator(device=DEV).manual_seed(seed)
    dt = {"bfloat16": torch.bfloat16, "float32": torch.float32}[dtype]
    w = {}

    def mat(name, *shape, std=0.02):
        w[name] = torch.randn(shape, generator=g, device=DEV, dtype=dt).mul_(std)

    def vec(name, n, mean=0.0, std=0.0):
        w[name] = torch.randn(n, generator=g, device=DEV, dtype=dt).mul_(std).add_(mean)

    if case["model"] != "kulanex-2048":
        H, E, V, d = cfg["hidden_size"], cfg["num_experts"], cfg["vocab_size"], cfg["head_dim"]
        nq, nk, m, s = (cfg[k] for k in ("num_attention_heads", "num_key_value_heads", "moe_intermediate_size",
                                         "shared_expert_intermediate_size"))
        mat("model.embed_tokens.weight", V, H, std=2.0)
        mat("lm_head.weight", V, H)
        vec("model.norm.weight", H, 1.0, 0.1)
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            vec(p + "input_layernorm.weight", H, 1.0, 0.1)
            vec(p + "post_attention_layernorm.weight", H, 1.0, 0.1)
            for x, n in (("q", nq * d), ("k", nk * d), ("v", nk * d)):
                mat(p + f"self_attn.{x}_proj.weight", n, H)
                vec(p + f"self_attn.{x}_proj.bias", n, 0.0, 0.1)
            mat(p + "self_attn.o_proj.weight", H, nq * d)
            mat(p + "mlp.gate.weight", E, H)
            mat(p + "mlp.experts.gate_up_proj", E, 2 * m, H)
            mat(p + "mlp.experts.down_proj", E, H, m)
            mat(p + "mlp.shared_expert.gate_proj.weight", s, H)
            mat(p + "mlp.shared_expert.up_proj.weight", s, H)
            mat(p + "mlp.shared_expert.down_proj.weight", H, s)
            mat(p + "mlp.shared_expert_gate.weight", 1, H)
        return w
    V, W = cfg["vocab"], cfg["width"]
    # Sigmoid scores multiply what an expert reads, so a pick that hangs on a rounding would change a token's whole
    # output: some channels of the embedding rank the experts, the routers read mostly those, and the sublayers write little
    # into them.
    E = E_KUL
    mat("embed", V, W, std=1.0)
    rank = (torch.arange(V, device=DEV)[:, None] * 5 + torch.arange(E, device=DEV)[None, :]) % E
    w["embed"][:, :E] = (3.0 * (rank - E / 2)).to(dt)
    mat("head", V, W)
    vec("final.norm", W, 0.0, 0.1)
    for i, L in enumerate(cfg["layers"]):
        p, m = f"l{i}.mix.", L["mixer"]
        for x in ("norm1", "norm2"):
            vec(f"l{i}.{x}", W, 0.0, 0.1)
            w[f"l{i}.{x}"][:E] -= 0.9
        if L["type"] == "channel_delta":
            H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            for x, n in (("q", G * d), ("k", G * d), ("v", H * dv)):
                mat(p + x, n, W)
                w[p + x + ".conv"] = (0.4 * torch.randn(n, m["conv"], generator=g, device=DEV) + 0.4).to(dt)
            mat(p + "b", H, W)
            mat(p + "a1", RANK, W), mat(p + "a2", H * d, RANK, std=0.08)
            mat(p + "g1", RANK, W), mat(p + "g2", H * dv, RANK, std=0.08)
            vec(p + "A_log", H, -1.0, 0.8), vec(p + "dt_bias", H * d, -1.0, 0.8)
            vec(p + "norm", dv, 1.0, 0.1)
            mat(p + "o", W, H * dv)
        else:
            a, r = m["left"], m["right"]
            for x, n in (("left.q", a["heads"] * a["dim"]), ("left.k", a["kv_heads"] * a["dim"])):
                mat(p + x, n, W)
                w[p + x + ".conv"] = (0.4 * torch.randn(n, a["conv"], generator=g, device=DEV) + 0.4).to(dt)
                vec(p + x + ".norm", n, 1.0, 0.1)
            mat(p + "left.o", W, a["heads"] * a["dim"])
            H, d, dv = r["heads"], r["dim"], r["vdim"]
            for x, n in (("q", H * d), ("k", H * d), ("v", H * dv), ("g", H * dv), ("i", H), ("f", H)):
                mat(p + "right." + x, n, W, std=0.014)
            vec(p + "right.i.b", H, -0.5, 1.0), vec(p + "right.f.b", H, 2.5, 1.0)
            vec(p + "right.norm", H * dv, 1.0, 0.1)
            mat(p + "right.o", W, H * dv)
        mat(f"l{i}.mlp.router", E, W, std=0.001)
        w[f"l{i}.mlp.router"][range(E), range(E)] += 0.15
        ff = _EXPERTS["expert"]["ff"]
        for e in range(E):
            mat(f"l{i}.mlp.e{e}.gate", ff, W), mat(f"l{i}.mlp.e{e}.up", ff, W), mat(f"l{i}.mlp.e{e}.down", W, ff)
    return w


def prepare(case, seed):
    """A model, its engine, and the sequences as they stand before the step."""
    cfg, dtype = MODELS[case["model"]]
    arch, typed = moe_b200.parse_config(cfg)
    spec = arch.model_spec(typed)
    dt = {"bfloat16": torch.bfloat16, "float32": torch.float32}[dtype]
    model = DecoderModel(spec, TensorDictStore(_weights(case, seed)), moe_b200.Runtime(DEV, dt))
    model.config = typed
    tokens, n0 = _tokens(case, seed), _lengths(case)
    room = sum(-(-len(t) // 64) * 64 for t in tokens) + 64 * len(tokens)
    engine = moe_b200.Engine(model, max_tokens=room, max_slots=len(tokens))
    state = dict(case=case, engine=engine, n0=n0, slots=None)
    if case["do"] in ("decode", "turn"):
        state["slots"] = [engine.new_sequence() for _ in tokens]
        engine.step(state["slots"], [t[:n] for t, n in zip(tokens, n0)], [[] for _ in tokens])
        state["steps"] = [[t[n:] for t, n in zip(tokens, n0)]]
    else:
        state["steps"] = [[t[:n] for t, n in zip(tokens, n0)]]
        if case["do"] == "request":
            state["steps"] += [[[t[n + j]] for t, n in zip(tokens, n0)] for j in range(case["new"])]
    # a program that serves has run its kind of step before
    run(state)
    return state


def run(state):
    engine, case = state["engine"], state["case"]
    if case["do"] in ("decode", "turn"):
        logits = engine.step(state["slots"], state["steps"][0], check=False)
        for slot, n in zip(state["slots"], state["n0"]):
            engine.truncate(slot, n)
        return logits
    slots = [engine.new_sequence() for _ in state["n0"]]
    out = []
    for tokens in state["steps"]:
        logits = engine.step(slots, tokens, check=False)
        # (the logits of a step may lie in a buffer that the next step writes over)
        out.append(logits.clone() if len(state["steps"]) > 1 else logits)
    for slot in slots:
        engine.release(slot)
    return out


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _model_work(case, steps):
    """``steps``: (tokens before, new tokens) of every sequence, step by step."""
    cfg, dtype = MODELS[case["model"]]
    size = 2 if dtype == "bfloat16" else 4
    nbytes = flops = 0.0

    def product(rows, weights, reads=None):
        nonlocal nbytes, flops
        flops += 2.0 * rows * weights
        nbytes += size * (weights if reads is None else reads)

    def experts(T, E, k, weights):
        product(T * k, weights, weights * E * (1 - (1 - k / E) ** T))

    for seqs in steps:
        T, B = sum(n for _, n in seqs), len(seqs)

        def attention(heads, kv, d, planes, window=None, keep=0):
            nonlocal nbytes, flops
            for old, n in seqs:
                held = old if window is None else min(old, window + keep)
                nbytes += size * planes * kv * d * (held + n)
                if window is None:
                    seen = n * old + n * (n + 1) / 2
                else:
                    seen = sum(min(old + i + 1, window + keep) for i in range(n))
                flops += 4.0 * heads * d * seen

        if case["model"] != "kulanex-2048":
            H, V, d = cfg["hidden_size"], cfg["vocab_size"], cfg["head_dim"]
            nq, nk = cfg["num_attention_heads"], cfg["num_key_value_heads"]
            for i in range(cfg["num_hidden_layers"]):
                product(T, (nq + 2 * nk) * d * H)
                product(T, H * nq * d)
                win = cfg["sliding_window"] if cfg["use_sliding_window"] and i >= cfg["max_window_layers"] else None
                attention(nq, nk, d, 2, win)
                product(T, (cfg["num_experts"] + 1) * H)
                experts(T, cfg["num_experts"], cfg["num_experts_per_tok"], 3 * cfg["moe_intermediate_size"] * H)
                product(T, 3 * cfg["shared_expert_intermediate_size"] * H)
        else:
            H, V = cfg["width"], cfg["vocab"]
            for L in cfg["layers"]:
                m = L["mixer"]
                if L["type"] == "channel_delta":
                    h, d, dv = m["heads"], m["dim"], m["vdim"]
                    product(T, H * (2 * m["kv_heads"] * d + 2 * h * dv + h + 2 * RANK) + RANK * h * (d + dv))
                    flops += 8.0 * T * h * d * dv
                    nbytes += 2 * 4.0 * B * h * d * dv
                else:
                    a, r = m["left"], m["right"]
                    product(T, H * (2 * a["heads"] + a["kv_heads"]) * a["dim"])
                    attention(a["heads"], a["kv_heads"], a["dim"], 1, a["mask"]["size"], a["mask"]["keep_first"])
                    h, d, dv = r["heads"], r["dim"], r["vdim"]
                    product(T, H * (2 * h * d + 3 * h * dv + 2 * h))
                    flops += 6.0 * T * h * d * dv
                    nbytes += 2 * 4.0 * B * h * d * dv
                product(T, E_KUL * H)
                experts(T, E_KUL, _EXPERTS["router"]["top"], 3 * _EXPERTS["expert"]["ff"] * H)
        product(B, V * H)
        nbytes += size * T * H + 4 * B * V
    return nbytes, flops



def work(case):
    n0 = _lengths(case)
    if case["do"] == "decode":
        steps = [[(n, 1) for n in n0]]
    elif case["do"] == "turn":
        steps = [[(n, case["new"]) for n in n0]]
    else:
        steps = [[(0, n) for n in n0]]
        if case["do"] == "request":
            steps += [[(n + j, 1) for n in n0] for j in range(case["new"])]
    nbytes, flops = _model_work(case, steps)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # measured against 64 bits and between two orders of the sums; about four times that
    if MODELS[case["model"]][1] == "float32":
        return {"rel": 2e-5, "max": 1e-3}
    return {"rel": 0.02, "max": 0.5}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------
def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _attend(q, k, v, scale, window=None, keep=0, rows=512):
    """q: [T, heads, d], k, v: [T, kv, d]; causal, with a window beside which the first ``keep`` positions stay in sight."""
    T, H, d = q.shape
    G = k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=F8, device=q.device)
    kk, vv = k.permute(1, 2, 0), v.permute(1, 0, 2)
    for a in range(0, T, rows):
        b = min(T, a + rows)
        s = torch.matmul(q[a:b].permute(1, 0, 2).reshape(G, H // G * (b - a), d), kk[:, :, :b]) * scale
        i, j = torch.arange(a, b, device=q.device)[:, None], torch.arange(b, device=q.device)[None, :]
        seen = j <= i
        if window is not None:
            seen &= (i - j < window) | (j < keep)
        s = s.view(G, H // G, b - a, b).masked_fill_(~seen, float("-inf"))
        o = torch.matmul(torch.softmax(s, -1).view(G, H // G * (b - a), b), vv[:, :b])
        out[a:b] = o.view(G * (H // G), b - a, -1).permute(1, 0, 2)
    return out


def _exact_moe(cfg, w, seqs, want):
    d, eps, H = cfg["head_dim"], cfg["rms_norm_eps"], cfg["hidden_size"]
    nq, nk, E, k = (cfg[x] for x in ("num_attention_heads", "num_key_value_heads", "num_experts", "num_experts_per_tok"))
    lens = [len(t) for t in seqs]
    pos = torch.cat([torch.arange(n, device=DEV) for n in lens]).to(F8)
    f = cfg["rope_theta"] ** (-torch.arange(0, d, 2, device=DEV, dtype=F8) / d)
    cos, sin = torch.cos(pos[:, None] * f)[:, None], torch.sin(pos[:, None] * f)[:, None]

    def turn(x):
        u, v = x[..., :d // 2], x[..., d // 2:]
        return torch.cat([u * cos - v * sin, v * cos + u * sin], -1)

    def lin(x, name, bias=None):
        y = torch.empty(x.shape[0], w[name].shape[0], dtype=F8, device=DEV)
        m = w[name].to(F8).T
        for a in range(0, x.shape[0], 8192):
            torch.matmul(x[a:a + 8192], m, out=y[a:a + 8192])
        return y if bias is None else y.add_(w[bias].to(F8))

    def swiglu(x, gate, up, down):
        out = torch.empty(x.shape[0], down.shape[0], dtype=F8, device=DEV)
        for a in range(0, x.shape[0], 4096):
            y = x[a:a + 4096]
            out[a:a + 4096] = (torch.nn.functional.silu(y @ gate.T) * (y @ up.T)) @ down.T
        return out

    x = w["model.embed_tokens.weight"][torch.tensor([t for s in seqs for t in s], device=DEV)].to(F8)
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        n = _rms(x, eps) * w[p + "input_layernorm.weight"].to(F8)
        q, kk, v = (lin(n, p + f"self_attn.{s}_proj.weight", p + f"self_attn.{s}_proj.bias").view(-1, h, d)
                    for s, h in (("q", nq), ("k", nk), ("v", nk)))
        q, kk = turn(q), turn(kk)
        win = cfg["sliding_window"] if cfg["use_sliding_window"] and i >= cfg["max_window_layers"] else None
        o = torch.cat([_attend(a, b, c, d ** -0.5, win) for a, b, c in zip(q.split(lens), kk.split(lens), v.split(lens))])
        x = x + lin(o.reshape(-1, nq * d), p + "self_attn.o_proj.weight")
        del q, kk, v, o
        n = _rms(x, eps) * w[p + "post_attention_layernorm.weight"].to(F8)
        prob, pick = torch.softmax(lin(n, p + "mlp.gate.weight"), -1).topk(k, -1)
        if cfg["norm_topk_prob"]:
            prob = prob / prob.sum(-1, keepdim=True)
        ws = [w[p + f"mlp.shared_expert.{s}_proj.weight"].to(F8) for s in ("gate", "up", "down")]
        out = torch.sigmoid(lin(n, p + "mlp.shared_expert_gate.weight")) * swiglu(n, *ws)
        for e in range(E):
            t, j = (pick == e).nonzero(as_tuple=True)
            if t.numel():
                gu = w[p + "mlp.experts.gate_up_proj"][e].to(F8)
                half = gu.shape[0] // 2
                out.index_add_(0, t, prob[t, j][:, None] * swiglu(n[t], gu[:half], gu[half:],
                                                                  w[p + "mlp.experts.down_proj"][e].to(F8)))
        x = x + out
        del out, n
    return _rms(x[want], eps) * w["model.norm.weight"].to(F8) @ w["lm_head.weight"].to(F8).T


def _exact_kulanex(cfg, w, seqs, want):
    eps, mult = cfg["norm"]["eps"], cfg["residual_mult"]
    lens = [len(t) for t in seqs]
    get = lambda name: w[name].to(F8)  # noqa: E731

    def lin(x, name):
        return x @ get(name).T

    def taps(u, name):
        t = get(name)
        n = t.shape[1]
        out = []
        for s in u.split(lens):
            s = torch.cat([torch.zeros(n - 1, s.shape[1], dtype=F8, device=DEV), s])
            out.append(sum(s[j:len(s) - n + 1 + j] * t[:, j] for j in range(n)))
        return torch.cat(out)

    def padded(u):
        """[T, ...] as [longest, sequences, ...], for the recurrences, which all sequences take together."""
        return torch.nn.utils.rnn.pad_sequence(list(u.split(lens)))

    def packed(u):
        return torch.cat([u[:n, b] for b, n in enumerate(lens)])

    def attention(x, p, m):
        H, G, d, rot = m["heads"], m["kv_heads"], m["dim"], m["rot"]
        q, k = taps(lin(x, p + "q"), p + "q.conv"), taps(lin(x, p + "k"), p + "k.conv")
        v = k.view(-1, G, d)
        q = (_rms(q, eps) * get(p + "q.norm")).view(-1, H, d)
        k = (_rms(k, eps) * get(p + "k.norm")).view(-1, G, d)
        r, sc = rot["dims"], rot["scaling"]
        f = rot["base"] ** (-torch.arange(0, r, 2, device=DEV, dtype=F8) / r)
        length = 2 * math.pi / f
        mix = ((sc["original"] / length - sc["low"]) / (sc["high"] - sc["low"])).clamp(0.0, 1.0)
        f = (1 - mix) * f / sc["factor"] + mix * f
        ang = torch.cat([torch.arange(n, device=DEV) for n in lens]).to(F8)[:, None] * f
        cos, sin = torch.cos(ang)[:, None], torch.sin(ang)[:, None]

        def turn(z):
            a, b = z[..., 0:r:2], z[..., 1:r:2]
            return torch.cat([torch.stack([a * cos - b * sin, b * cos + a * sin], -1).flatten(-2), z[..., r:]], -1)

        q, k = turn(q), turn(k)
        o = [_attend(a, b, c, m["scale"], m["mask"]["size"], m["mask"]["keep_first"])
             for a, b, c in zip(q.split(lens), k.split(lens), v.split(lens))]
        return lin(torch.cat(o).reshape(-1, H * d), p + "o")

    def memory(x, p, m):
        H, d, dv, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
        q, k = padded(lin(x, p + "q") / math.sqrt(d)).unflatten(-1, (H, d)), padded(lin(x, p + "k")).unflatten(-1, (H, d))
        v = padded(lin(x, p + "v")).unflatten(-1, (H, dv))
        gi, gf = (padded(cap * torch.tanh((lin(x, p + s) + get(p + s + ".b")) / cap)) for s in ("i", "f"))
        gf = torch.nn.functional.logsigmoid(gf)
        B = len(lens)
        S, z = torch.zeros(B, H, d, dv, dtype=F8, device=DEV), torch.zeros(B, H, d, dtype=F8, device=DEV)
        mu = torch.zeros(B, H, dtype=F8, device=DEV)
        out = torch.empty_like(v)
        for t in range(v.shape[0]):
            new = torch.maximum(gf[t] + mu, gi[t])
            keep, add = torch.exp(gf[t] + mu - new), torch.exp(gi[t] - new)
            mu = new
            ak = add[..., None] * k[t]
            S = torch.addcmul(keep[..., None, None] * S, ak[..., None], v[t][..., None, :])
            z = keep[..., None] * z + ak
            size = torch.maximum((z * q[t]).sum(-1).abs(), torch.exp(-mu)) + 1e-6
            out[t] = torch.matmul(q[t][..., None, :], S)[..., 0, :] / size[..., None]
        o = packed(_rms(out, eps).flatten(-2)) * get(p + "norm") * torch.sigmoid(lin(x, p + "g"))
        return lin(o, p + "o")

    def delta(x, p, m):
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        q, k, v = (torch.nn.functional.silu(taps(lin(x, p + s), p + s + ".conv")) for s in "qkv")

        def unit(u):
            u = u.view(-1, m["kv_heads"], d)
            return (u / torch.sqrt((u * u).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // m["kv_heads"], 1)

        q, k, v = padded(unit(q) / math.sqrt(d)), padded(unit(k)), padded(v.view(-1, H, dv))
        beta = padded(torch.sigmoid(lin(x, p + "b")))
        pace = torch.nn.functional.softplus(lin(lin(x, p + "a1"), p + "a2") + get(p + "dt_bias")).view(-1, H, d)
        decay = padded(torch.exp(-torch.exp(get(p + "A_log"))[:, None] * pace))
        S = torch.zeros(len(lens), H, d, dv, dtype=F8, device=DEV)
        out = torch.empty_like(v)
        for t in range(v.shape[0]):
            S = S * decay[t][..., None]
            held = torch.matmul(k[t][..., None, :], S)[..., 0, :]
            S = torch.addcmul(S, k[t][..., None], (beta[t][..., None] * (v[t] - held))[..., None, :])
            out[t] = torch.matmul(q[t][..., None, :], S)[..., 0, :]
        o = packed((_rms(out, eps) * get(p + "norm")).flatten(-2))
        return lin(o * torch.sigmoid(lin(lin(x, p + "g1"), p + "g2")), p + "o")

    x = get("embed")[torch.tensor([t for s in seqs for t in s], device=DEV)]
    for i, L in enumerate(cfg["layers"]):
        p, m = f"l{i}.mix.", L["mixer"]
        if L["type"] == "channel_delta":
            y = delta(x, p, m)
        else:
            y = m["left_scale"] * attention(x, p + "left.", m["left"]) + m["right_scale"] * memory(x, p + "right.", m["right"])
        x = x + mult * _rms(y, eps) * (1 + get(f"l{i}.norm1"))
        score = torch.sigmoid(lin(x, f"l{i}.mlp.router"))
        pick = score.topk(L["mlp"]["router"]["top"], -1).indices
        y = torch.zeros_like(x)
        for e in range(E_KUL):
            t = (pick == e).any(-1).nonzero()[:, 0]
            if t.numel():
                h = score[t, e][:, None] * x[t]
                g, u, dn = (f"l{i}.mlp.e{e}.{s}" for s in ("gate", "up", "down"))
                y.index_add_(0, t, lin(torch.nn.functional.silu(lin(h, g)) * lin(h, u), dn))
        x = x + mult * _rms(y, eps) * (1 + get(f"l{i}.norm2"))
    return _rms(x[want], eps) * (1 + get("final.norm")) @ get("head").T


def exact(case, seed):
    cfg, _ = MODELS[case["model"]]
    w, seqs, n0 = _weights(case, seed), _tokens(case, seed), _lengths(case)
    at, rows = 0, []
    for t, n in zip(seqs, n0):
        rows.append([at + n - 1 + j for j in range(case["new"] + 1)] if case["do"] == "request" else [at + len(t) - 1])
        at += len(t)
    want = torch.tensor([r[j] for j in range(len(rows[0])) for r in rows], device=DEV)
    logits = (_exact_kulanex if case["model"] == "kulanex-2048" else _exact_moe)(cfg, w, seqs, want)
    if case["do"] in ("decode", "turn"):
        return logits
    return list(logits.split(len(seqs)))
