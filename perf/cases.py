"""The calls whose speed and accuracy are watched, over the range that a program of this framework uses.

Families (``case["kind"]``), each through an entry point that a program calls:

* ``linear``    ``FusedSession.matmul_bias_w16``: ``x @ w + bias`` over a resident weight, optionally with the GELU
                and the residual of the epilogue; inference, from a handful of rows to a large batch.
* ``mha``       ``FusedSession.mha``: bidirectional attention over per-token projections (encoder inference).
* ``mlp``       ``ops.fused.mlp_up_down`` on a tape, forward and backward: a transformer block's MLP in training.
* ``attention`` ``ops.fused.attention_packed`` on a tape, forward and backward, head size 64 or 128.
* ``norm``      ``ops.fused.layernorm`` / ``rmsnorm`` on a tape, forward and backward.
* ``head``      ``ops.fused.lm_head_cross_entropy`` on a tape, forward and backward.
* ``train``     ``TrainEngine.step``: one whole optimizer step of a GPT from a host batch (loss, gradients, weights).
* ``encoder``   ``EncoderGpu.forward_stack``: the layer stack of an encoder on resident activations.

Parameter gradients go to bound buffers, as the models bind them.  All compute is bf16 with fp32 accumulation,
statistics, parameter gradients and optimizer state.
"""
import math

import torch
import torch.nn.functional as TF

DEV = "cuda"
BF = torch.bfloat16


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # a classifier or serving head on a small batch: one launch, nothing but latency
        {"name": "linear_small", "kind": "linear", "rows": 32, "k": 512, "n": 2048, "gelu": False, "resid": False},
        # the MLP up projection of an audio encoder: ragged rows, GELU in the epilogue
        {"name": "linear_encoder_up", "kind": "linear", "rows": 1500, "k": 1280, "n": 5120, "gelu": True,
         "resid": False},
        # the MLP down projection of a 1.3B decoder over a full batch, with the residual
        {"name": "linear_large_down", "kind": "linear", "rows": 8192, "k": 8192, "n": 2048, "gelu": False,
         "resid": True},
        # self-attention of the same audio encoder: ragged, bidirectional
        {"name": "mha_encoder", "kind": "mha", "seq": 1500, "heads": 20, "hd": 64},
        # the MLP of a GPT-2 small block in training, micro-batch 8 x 1024
        {"name": "mlp_gpt2_small", "kind": "mlp", "rows": 8192, "d": 768, "ff": 3072, "act": "gelu_tanh"},
        # attention of GPT-2 small in training, micro-batch 8 x 1024
        {"name": "attention_gpt2_small", "kind": "attention", "batch": 8, "seq": 1024, "heads": 12, "hd": 64,
         "causal": True},
        # attention of the 1.3B decoder in training, micro-batch 4 x 2048
        {"name": "attention_gpt_1b", "kind": "attention", "batch": 4, "seq": 2048, "heads": 16, "hd": 128,
         "causal": True},
        # a LayerNorm of GPT-2 medium in training, micro-batch 4 x 2048
        {"name": "norm_gpt2_medium", "kind": "norm", "rows": 8192, "cols": 1024, "rms": False},
        # tied LM head and loss of GPT-2 small in training, micro-batch 8 x 1024
        {"name": "head_gpt2_small", "kind": "head", "rows": 8192, "d": 768, "vocab": 50257},
        # a tiny model's whole step: about fifty launches of a few microseconds each
        {"name": "train_tiny", "kind": "train", "layers": 2, "d": 128, "heads": 2, "vocab": 1000, "batch": 4,
         "seq": 128},
        # GPT-2 small, the benchmark's step
        {"name": "train_gpt2_small", "kind": "train", "layers": 12, "d": 768, "heads": 12, "vocab": 50257, "batch": 8,
         "seq": 1024},
        # the large audio encoder, whole stack
        {"name": "encoder_turbo", "kind": "encoder", "seq": 1500, "d": 1280, "heads": 20, "layers": 32},
    ]


def _log_int(rng, lo, hi, mult=1):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(mult, v // mult * mult)


MAX_FLOPS = 2.5e12      # a drawn case stays below the largest listed one


def draw(rng):
    """One more case of the same families; extents are odd where the entry point takes odd extents."""
    while True:
        kind = rng.choice(["linear", "linear", "mha", "mlp", "attention", "attention", "norm", "head", "train",
                           "encoder"])
        c = {"kind": kind}
        if kind == "linear":
            c.update(rows=_log_int(rng, 1, 16384), k=_log_int(rng, 64, 8192, 8), n=_log_int(rng, 64, 8192, 8),
                     gelu=rng.random() < 0.4, resid=rng.random() < 0.4)
        elif kind == "mha":
            c.update(seq=_log_int(rng, 16, 4096), heads=rng.randint(1, 20), hd=rng.choice([64, 128]))
        elif kind == "mlp":
            d = _log_int(rng, 128, 2048, 8)
            c.update(rows=_log_int(rng, 64, 16384), d=d, ff=4 * d,
                     act=rng.choice(["gelu_tanh", "gelu_erf", "relu"]))
        elif kind == "attention":
            c.update(batch=rng.randint(1, 8), seq=_log_int(rng, 64, 4096), heads=rng.randint(1, 16),
                     hd=rng.choice([64, 128]), causal=rng.random() < 0.75)
        elif kind == "norm":
            c.update(rows=_log_int(rng, 16, 65536), cols=_log_int(rng, 64, 8192, 8), rms=rng.random() < 0.3)
            if c["rows"] * c["cols"] > 1.5e8:
                continue
        elif kind == "head":
            c.update(rows=_log_int(rng, 16, 8192), d=_log_int(rng, 128, 1024, 8), vocab=_log_int(rng, 1000, 50257))
        elif kind == "train":
            hd = 64
            heads = rng.randint(2, 12)
            c.update(layers=rng.randint(1, 4), d=hd * heads, heads=heads, vocab=_log_int(rng, 500, 20000),
                     batch=rng.randint(1, 8), seq=_log_int(rng, 64, 1024))
        else:
            hd = rng.choice([64, 128])
            heads = rng.randint(4, 12)
            c.update(seq=_log_int(rng, 64, 3000), d=hd * heads, heads=heads, layers=rng.randint(1, 8))
        if work(c)["flops"] <= MAX_FLOPS:
            return c


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _n(g, *shape, std=1.0, mean=0.0, dtype=BF):
    return (torch.randn(*shape, generator=g, device=DEV) * std + mean).to(dtype)


def _linear_inputs(c, g):
    m, k, n = c["rows"], c["k"], c["n"]
    return {"x": _n(g, m, k), "w": _n(g, k, n, std=k ** -0.5), "b": _n(g, n, std=0.02),
            "r": _n(g, m, n) if c["resid"] else None}


def _mha_inputs(c, g):
    d = c["heads"] * c["hd"]
    return {t: _n(g, c["seq"], d) for t in "qkv"}


def _mlp_inputs(c, g):
    m, d, ff = c["rows"], c["d"], c["ff"]
    return {"x": _n(g, m, d), "w1": _n(g, ff, d, std=d ** -0.5), "b1": _n(g, ff, std=0.02),
            "w2": _n(g, d, ff, std=ff ** -0.5), "b2": _n(g, d, std=0.02), "resid": _n(g, m, d),
            "gy": _n(g, m, d, std=1e-2)}


def _attention_inputs(c, g):
    d = c["heads"] * c["hd"]
    return {"qkv": _n(g, c["batch"], c["seq"], 3 * d), "gy": _n(g, c["batch"], c["seq"], d, std=1e-2)}


def _norm_inputs(c, g):
    r, n = c["rows"], c["cols"]
    i = {"x": _n(g, r, n, std=2.0, mean=0.25), "gamma": _n(g, n, std=0.05, mean=1.0), "gy": _n(g, r, n, std=1e-2)}
    if not c["rms"]:
        i["beta"] = _n(g, n, std=0.05)
    return i


def _pad128(v):
    return (v + 127) // 128 * 128


def _head_inputs(c, g):
    w = _n(g, _pad128(c["vocab"]), c["d"], std=0.02)
    w[c["vocab"]:] = 0
    return {"x": _n(g, c["rows"], c["d"]), "w": w,
            "ids": torch.randint(0, c["vocab"], (c["rows"],), generator=g, device=DEV)}


def _train_names(c):
    """(name, shape, std, mean) of every parameter, the vocabulary without its padding rows."""
    d, ff, L = c["d"], 4 * c["d"], c["layers"]
    out = [("wte.weight", (c["vocab"], d), 0.02, 0.0), ("wpe.weight", (max(c["seq"], 64), d), 0.02, 0.0)]
    proj = 0.02 / math.sqrt(2 * L)
    for l in range(L):
        p = "blocks.%d." % l
        out += [(p + "ln1.weight", (d,), 0.02, 1.0), (p + "ln1.bias", (d,), 0.02, 0.0),
                (p + "attn.qkv_proj.weight", (3 * d, d), 0.02, 0.0), (p + "attn.qkv_proj.bias", (3 * d,), 0.02, 0.0),
                (p + "attn.out_proj.weight", (d, d), proj, 0.0), (p + "attn.out_proj.bias", (d,), 0.02, 0.0),
                (p + "ln2.weight", (d,), 0.02, 1.0), (p + "ln2.bias", (d,), 0.02, 0.0),
                (p + "mlp.fc1.weight", (ff, d), 0.02, 0.0), (p + "mlp.fc1.bias", (ff,), 0.02, 0.0),
                (p + "mlp.fc2.weight", (d, ff), proj, 0.0), (p + "mlp.fc2.bias", (d,), 0.02, 0.0)]
    return out + [("ln_f.weight", (d,), 0.02, 1.0), ("ln_f.bias", (d,), 0.02, 0.0)]


def _train_inputs(c, g):
    sd = {name: _n(g, *shape, std=std, mean=mean, dtype=torch.float32) for name, shape, std, mean in _train_names(c)}
    ids, targets = (torch.randint(0, c["vocab"], (c["batch"], c["seq"]), generator=g, device=DEV) for _ in range(2))
    return sd, ids, targets


ENC_FIELDS = ("ln1_g", "ln1_b", "wq", "bq", "wk", "wv", "bv", "wo", "bo", "ln2_g", "ln2_b", "w1", "b1", "w2", "b2")


def _encoder_layer(c, g):
    d, ff = c["d"], 4 * c["d"]
    mat = lambda o, i: _n(g, o, i, std=i ** -0.5)                        # noqa: E731
    vec = lambda n, s=0.02, m=0.0: _n(g, n, std=s, mean=m)               # noqa: E731
    return dict(zip(ENC_FIELDS, (vec(d, 0.05, 1.0), vec(d), mat(d, d), vec(d), mat(d, d), mat(d, d), vec(d), mat(d, d),
                                 vec(d), vec(d, 0.05, 1.0), vec(d), mat(ff, d), vec(ff), mat(d, ff), vec(d))))


class _OnTape:
    """Leaves on a tape: parameters with a bound fp32 gradient buffer, activations without one."""

    def __init__(self, params, acts):
        from frankentorch_b200.autograd.tape import TensorTape
        self.tape = TensorTape(grad_dtype=None)
        self.ids, self.bufs = {}, {}
        for name, t in params.items():
            self.ids[name] = self.tape.leaf(t, requires_grad=True, name=name)
            self.bufs[name] = torch.empty(t.shape, dtype=torch.float32, device=DEV)
            self.tape.bind_grad_buffer(self.ids[name], self.bufs[name])
        for name, t in acts.items():
            self.ids[name] = self.tape.leaf(t, requires_grad=True, name=name)
        self.acts = list(acts)
        self.boundary = len(self.tape)

    def step(self, root, seed=None):
        """Backward from ``root``; the value and every gradient, the graph dropped."""
        y = self.tape.value(root)
        rep = self.tape.backward(root, seed=seed)
        out = {"y": y}
        for name in self.acts:
            out["d_" + name] = rep.gradient(self.ids[name])
        for name, buf in self.bufs.items():
            out["d_" + name] = buf
        self.tape.truncate_graph_to(self.boundary)
        return out

    def begin(self):
        for nid in self.ids.values():
            self.tape.zero_accumulated_gradient(nid)


def prepare(case, seed):
    c, g, kind = case, _gen(seed), case["kind"]
    if kind == "linear":
        from frankentorch_b200.ops.fused_session import FusedSession
        s, i = FusedSession(DEV + ":0"), _linear_inputs(c, g)
        return {"case": c, "s": s, "x": i["x"], "w": s.weight(i["w"]), "b": i["b"], "r": i["r"]}
    if kind == "mha":
        from frankentorch_b200.ops.fused_session import FusedSession
        return {"case": c, "s": FusedSession(DEV + ":0"), **_mha_inputs(c, g)}
    if kind == "mlp":
        i = _mlp_inputs(c, g)
        gy = i.pop("gy")
        return {"case": c, "t": _OnTape({k: i[k] for k in ("w1", "b1", "w2", "b2")},
                                        {k: i[k] for k in ("x", "resid")}), "gy": gy}
    if kind == "attention":
        i = _attention_inputs(c, g)
        return {"case": c, "t": _OnTape({}, {"qkv": i["qkv"]}), "gy": i["gy"]}
    if kind == "norm":
        i = _norm_inputs(c, g)
        return {"case": c, "t": _OnTape({k: i[k] for k in ("gamma", "beta") if k in i}, {"x": i["x"]}), "gy": i["gy"]}
    if kind == "head":
        i = _head_inputs(c, g)
        return {"case": c, "t": _OnTape({"w": i["w"]}, {"x": i["x"]}), "ids": i["ids"]}
    if kind == "train":
        from frankentorch_b200.autograd.tape import TensorTape
        from frankentorch_b200.models.gpt import GPT, GPTConfig
        from frankentorch_b200.training.engine import TrainEngine
        sd, ids, targets = _train_inputs(c, g)
        cfg = GPTConfig(n_layer=c["layers"], d_model=c["d"], n_head=c["heads"], d_ff=4 * c["d"],
                        vocab_size=c["vocab"], max_seq=max(c["seq"], 64), name="case")
        model = GPT(cfg, TensorTape(grad_dtype=None), device=DEV)
        model.load_state_dict(sd)
        return {"case": c, "model": model, "engine": TrainEngine(model, c["batch"], c["seq"]),
                "ids": ids.cpu().pin_memory(), "targets": targets.cpu().pin_memory()}
    from frankentorch_b200.models.encoder import EncoderGpu, EncoderLayerWeights
    x = _n(g, c["seq"], c["d"])
    layers = [EncoderLayerWeights(**_encoder_layer(c, g)) for _ in range(c["layers"])]
    return {"case": c, "x": x, "enc": EncoderGpu(layers, c["heads"], device=DEV + ":0")}


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    from frankentorch_b200.ops import fused as F
    c = state["case"]
    kind = c["kind"]
    if kind == "linear":
        return state["s"].matmul_bias_w16(state["x"], state["w"], state["b"], gelu=c["gelu"], resid=state["r"])
    if kind == "mha":
        return state["s"].mha(state["q"], state["k"], state["v"], c["heads"])
    if kind == "train":
        e, a = state["engine"], state["model"].arena
        e.step(state["ids"], state["targets"], read_loss=False)
        return {"loss": e.loss_dev, "grads": a.grads, "weights": a.master}     # the model's flat arenas
    if kind == "encoder":
        return state["enc"].forward_stack(state["x"])
    t = state["t"]
    i = t.ids
    t.begin()
    if kind == "mlp":
        root = F.mlp_up_down(t.tape, i["x"], i["w1"], i["b1"], i["w2"], i["b2"], i["resid"], act=c["act"])
    elif kind == "attention":
        root = F.attention_packed(t.tape, i["qkv"], c["heads"], causal=c["causal"])
    elif kind == "norm":
        root = F.rmsnorm(t.tape, i["x"], i["gamma"]) if c["rms"] else \
            F.layernorm(t.tape, i["x"], i["gamma"], i["beta"])
    else:
        root = F.lm_head_cross_entropy(t.tape, i["x"], i["w"], state["ids"], c["vocab"])
    return t.step(root, state.get("gy"))


# ------------------------------------------------------------------------------------------------ work
def work(case):
    c, kind = case, case["kind"]
    if kind == "linear":
        m, k, n = c["rows"], c["k"], c["n"]
        return {"bytes": 2 * (m * k + k * n + n + m * n * (2 if c["resid"] else 1)), "flops": 2 * m * k * n}
    if kind == "mha":
        d = c["heads"] * c["hd"]
        return {"bytes": 2 * 4 * c["seq"] * d, "flops": 4 * c["seq"] ** 2 * d}
    if kind == "mlp":
        m, d, ff = c["rows"], c["d"], c["ff"]
        # in: x, resid, gy, weights; out: y, dx, d_resid (the incoming gradient itself) and fp32 weight gradients
        return {"bytes": 2 * 5 * m * d + (2 + 4) * (2 * d * ff + d + ff), "flops": 3 * 4 * m * d * ff}
    if kind == "attention":
        d, s, b = c["heads"] * c["hd"], c["seq"], c["batch"]
        pairs = s * (s + 1) // 2 if c["causal"] else s * s
        # forward: two products; backward: five (the scores again, dP, dV, dK, dQ)
        return {"bytes": 2 * b * s * (3 * d + d + d + 3 * d), "flops": 7 * 2 * b * pairs * d}
    if kind == "norm":
        r, n = c["rows"], c["cols"]
        return {"bytes": 2 * 4 * r * n + (2 + 4) * n * (1 if c["rms"] else 2), "flops": 20 * r * n}
    if kind == "head":
        m, d, v = c["rows"], c["d"], c["vocab"]
        return {"bytes": 2 * 2 * m * d + (2 + 4) * v * d + 8 * m, "flops": 3 * 2 * m * d * v}
    if kind == "train":
        d, L, m, s = c["d"], c["layers"], c["batch"] * c["seq"], c["seq"]
        params = sum(math.prod(shape) for _, shape, _, _ in _train_names(c))
        # master and both moments are read and written, gradients and the bf16 copy written
        return {"bytes": params * (3 * 8 + 4 + 2) + 16 * m,
                "flops": 6 * m * (12 * L * d * d + c["vocab"] * d) + 7 * L * m * (s + 1) * d}
    m, d, L = c["seq"], c["d"], c["layers"]
    return {"bytes": 2 * (2 * m * d + 12 * L * d * d), "flops": L * (24 * m * d * d + 4 * m * m * d)}


# ------------------------------------------------------------------------------------------------ accuracy
# A bf16 result carries a rounding error of 2^-9 relative at most, 1.1e-3 of the 2-norm; intermediates rounded to bf16
# (probabilities, activations, the logit gradient) add their own.  The figures are about four times the distance that
# the path shows from 64-bit arithmetic.
REL = {"linear": 7e-3, "mha": 1e-2, "mlp": 1e-2, "attention": 1e-2, "norm": 7e-3, "head": 1.2e-2, "train": 4e-2,
       "encoder": 4e-2}


def tolerance(case):
    return {"rel": REL[case["kind"]]}


def _gelu(x, act="gelu_tanh"):
    if act == "relu":
        return torch.relu(x)
    return TF.gelu(x, approximate="tanh" if act == "gelu_tanh" else "none")


def _attend(q, k, v, causal):
    """``[..., S, hd]`` in 64 bits, one leading index at a time to bound the score matrix."""
    s = q.shape[-2]
    mask = torch.ones(s, s, dtype=torch.bool, device=q.device).triu(1) if causal else None
    outs = []
    for qq, kk, vv in zip(q, k, v):
        p = qq @ kk.transpose(-1, -2) / math.sqrt(q.shape[-1])
        if causal:
            p = p.masked_fill(mask, -math.inf)
        outs.append(torch.softmax(p, -1) @ vv)
    return torch.stack(outs)


def _packed_attention(qkv, heads, causal):
    b, s, d3 = qkv.shape
    hd = d3 // 3 // heads
    q, k, v = (t.reshape(b, s, heads, hd).transpose(1, 2) for t in qkv.split(d3 // 3, -1))
    return _attend(q, k, v, causal).transpose(1, 2).reshape(b, s, d3 // 3)


def _head_loss(x, w, ids, vocab):
    return TF.cross_entropy(x @ w[:vocab].T, ids)


def _exact_train(c, g):
    sd, ids, targets = _train_inputs(c, g)
    P = {n: t.to(BF).double().requires_grad_(True) for n, t in sd.items()}
    d = c["d"]
    x = P["wte.weight"][ids] + P["wpe.weight"][: c["seq"]]
    norm = lambda t, p: TF.layer_norm(t, (d,), P[p + ".weight"], P[p + ".bias"], 1e-5)     # noqa: E731
    lin = lambda t, p: TF.linear(t, P[p + ".weight"], P[p + ".bias"])                      # noqa: E731
    for l in range(c["layers"]):
        p = "blocks.%d." % l
        a = _packed_attention(lin(norm(x, p + "ln1"), p + "attn.qkv_proj"), c["heads"], True)
        x = x + lin(a, p + "attn.out_proj")
        x = x + lin(_gelu(lin(norm(x, p + "ln2"), p + "mlp.fc1")), p + "mlp.fc2")
    loss = _head_loss(norm(x, "ln_f").reshape(-1, d), P["wte.weight"], targets.reshape(-1), c["vocab"])
    loss.backward()
    gn = math.sqrt(sum(float((p.grad ** 2).sum()) for p in P.values()))
    clip = 1.0 / gn if gn > 1.0 else 1.0
    lr, eps, wd = 3e-4, 1e-8, 0.01
    grads, weights = [], []
    for n, p in P.items():
        gr, w0 = p.grad, sd[n].double()
        # the first AdamW step: both bias-corrected moments are those of this gradient
        w = w0 * (1 - lr * wd) - lr * (gr * clip) / ((gr * clip).abs() + eps)
        rows = _pad128(c["vocab"]) - c["vocab"] if n == "wte.weight" else 0     # the stored table has whole tiles
        for out, t in ((grads, gr), (weights, w)):
            t = TF.pad(t, (0, 0, 0, rows)) if rows else t
            out.append(TF.pad(t.reshape(-1), (0, -t.numel() % 128)))            # a slot is a multiple of 128 elements
    flat = lambda ts: TF.pad(torch.cat(ts), (0, -sum(t.numel() for t in ts) % 1024))     # noqa: E731
    return {"loss": loss.detach(), "grads": flat(grads), "weights": flat(weights)}


def exact(case, seed):
    c, g, kind = case, _gen(seed), case["kind"]
    D = lambda t: None if t is None else t.double()      # noqa: E731
    if kind == "linear":
        i = _linear_inputs(c, g)
        y = D(i["x"]) @ D(i["w"]) + D(i["b"])
        y = _gelu(y) if c["gelu"] else y
        return y if i["r"] is None else y + D(i["r"])
    if kind == "mha":
        i = _mha_inputs(c, g)
        q, k, v = (D(i[t]).view(c["seq"], c["heads"], c["hd"]).transpose(0, 1) for t in "qkv")
        return _attend(q, k, v, False).transpose(0, 1).reshape(c["seq"], -1)
    if kind == "train":
        return _exact_train(c, g)
    if kind == "encoder":
        x = D(_n(g, c["seq"], c["d"]))
        d, h = c["d"], c["heads"]
        for _ in range(c["layers"]):
            w = {k: D(t) for k, t in _encoder_layer(c, g).items()}
            n1 = TF.layer_norm(x, (d,), w["ln1_g"], w["ln1_b"], 1e-5)
            q, k, v = ((n1 @ m.T + (0 if b is None else b)).view(-1, h, d // h).transpose(0, 1)
                       for m, b in ((w["wq"], w["bq"]), (w["wk"], None), (w["wv"], w["bv"])))
            x = x + _attend(q, k, v, False).transpose(0, 1).reshape(-1, d) @ w["wo"].T + w["bo"]
            n2 = TF.layer_norm(x, (d,), w["ln2_g"], w["ln2_b"], 1e-5)
            x = x + _gelu(n2 @ w["w1"].T + w["b1"]) @ w["w2"].T + w["b2"]
        return x
    if kind == "mlp":
        i = {k: D(t).requires_grad_(True) for k, t in _mlp_inputs(c, g).items()}
        y = i["resid"] + TF.linear(_gelu(TF.linear(i["x"], i["w1"], i["b1"]), c["act"]), i["w2"], i["b2"])
        order = ("x", "resid", "w1", "b1", "w2", "b2")
    elif kind == "attention":
        i = {k: D(t).requires_grad_(True) for k, t in _attention_inputs(c, g).items()}
        y = _packed_attention(i["qkv"], c["heads"], c["causal"])
        order = ("qkv",)
    elif kind == "norm":
        i = {k: D(t).requires_grad_(True) for k, t in _norm_inputs(c, g).items()}
        if c["rms"]:
            y = i["x"] * torch.rsqrt((i["x"] ** 2).mean(-1, keepdim=True) + 1e-6) * i["gamma"]
            order = ("x", "gamma")
        else:
            y = TF.layer_norm(i["x"], (c["cols"],), i["gamma"], i["beta"], 1e-5)
            order = ("x", "gamma", "beta")
    else:
        i = _head_inputs(c, g)
        ids = i.pop("ids")
        i = {k: D(t).requires_grad_(True) for k, t in i.items()}
        y = _head_loss(i["x"], i["w"], ids, c["vocab"])
        order = ("x", "w")
    grads = torch.autograd.grad(y, [i[k] for k in order], D(i["gy"].detach()) if "gy" in i else None)
    out = {"y": y.detach()}
    out.update({"d_" + k: gr for k, gr in zip(order, grads)})
    return out
