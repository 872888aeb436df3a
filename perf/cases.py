"""What the performance of this framework is measured on.

Each case is work that the training runtime has the kernels do for a user's model, through the operators a stage
graph calls (``rannc_b200.ops.functional``) or, for one case, through ``RaNNCModule`` itself.  Parameters are laid
out the way the runtime deploys them: 16-bit views of one flat buffer, each with an fp32 ``main_grad`` view of a
flat gradient buffer that a pass clears first (``flat`` true), or plain leaves whose gradients come back through
autograd (``flat`` false: the operators called on their own).  ``train`` false is evaluation under ``no_grad``.
"""
import math

import torch
import torch.nn as nn
import torch.nn.functional as F

DT = {"bf16": torch.bfloat16, "fp16": torch.float16}
LN_WIDTHS = (256, 512, 768, 1024, 1536, 2048, 4096)


def listed():
    return [
        # the pooler of a BERT-Large micro-batch (one row per sequence): the smallest call, bound by latency
        dict(name="linear_pooler", kind="linear", rows=32, inp=1024, out=1024, gelu=False, dtype="bf16", flat=True,
             train=True),
        # a ragged evaluation batch through a BERT-Base FFN input layer (odd number of tokens, GELU fused)
        dict(name="linear_gelu_eval", kind="linear", rows=3 * 117, inp=768, out=3072, gelu=True, dtype="fp16",
             flat=False, train=False),
        # the FFN block of BERT-Large at 32 sequences of 512: the bulk of a pre-training step
        dict(name="mlp_large", kind="mlp", rows=16384, hidden=1024, inner=4096, dtype="bf16", flat=True, train=True),
        # QKV projection + attention of BERT-Large with dropout and a padding mask, same batch
        dict(name="attention_large", kind="attention", batch=32, seq=512, heads=16, mask=True, p=0.1, dtype="bf16",
             flat=True, train=True),
        # fine-tuning a BERT-Base layer on sequences of an odd length, operators called on their own
        dict(name="attention_ragged", kind="attention", batch=6, seq=197, heads=12, mask=False, p=0.0, dtype="fp16",
             flat=False, train=True),
        # dropout + residual + LayerNorm after a BERT-Large sub-layer
        dict(name="norm_large", kind="norm", rows=16384, hidden=1024, p=0.1, residual=True, dtype="bf16", flat=True,
             train=True),
        # the widest encoder's LayerNorm on a small ragged batch
        dict(name="norm_wide_ragged", kind="norm", rows=387, hidden=4096, p=0.0, residual=True, dtype="bf16",
             flat=False, train=True),
        # word + position + segment embeddings, summed, normalised; token frequencies as in text
        dict(name="embedding_large", kind="embedding", batch=32, seq=512, vocab=30528, hidden=1024, dtype="bf16",
             flat=True, train=True),
        # masked-LM head: vocabulary projection and loss, 15 % of the positions labelled
        dict(name="mlm_head", kind="head", rows=8192, hidden=1024, vocab=30522, labelled=0.15, dtype="bf16",
             flat=True, train=True),
        # 3x3 convolution + batch norm + ReLU of a wide ResNet at 28 x 28
        dict(name="conv3_28", kind="conv", images=32, size=28, inp=1024, out=1024, k=3, residual=False, dtype="fp16",
             flat=True, train=True),
        # 1x1 expansion + batch norm + shortcut + ReLU that ends a bottleneck block at 14 x 14
        dict(name="conv1_14", kind="conv", images=32, size=14, inp=512, out=2048, k=1, residual=True, dtype="fp16",
             flat=True, train=True),
        # a whole optimizer step of a two-layer BERT-Large-wide encoder under RaNNCModule with mixed precision
        dict(name="train_step", kind="step", batch=16, seq=384, layers=2, hidden=1024, heads=16, vocab=30522,
             dtype="bf16"),
    ]


def _log(rng, lo, hi, unit=1):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / unit)) * unit))


def draw(rng):
    kind = rng.choice(["linear", "mlp", "attention", "norm", "embedding", "head", "conv", "linear", "mlp",
                       "attention", "norm", "conv"])
    c = dict(kind=kind, dtype=rng.choice(["bf16", "bf16", "fp16"]), flat=rng.random() < 0.6, train=rng.random() < 0.8)
    width = lambda lo, hi: _log(rng, lo, hi, 8)  # noqa: E731
    if kind == "linear":
        c.update(rows=_log(rng, 8, 16384), inp=width(256, 2048), out=width(256, 4096), gelu=rng.random() < 0.4)
    elif kind == "mlp":
        h = rng.choice([256, 512, 768, 1000, 1024, 1536])
        c.update(rows=_log(rng, 64, 12000), hidden=h, inner=min(4096, 4 * h))
    elif kind == "attention":
        heads, seq = rng.choice([4, 8, 12, 16]), _log(rng, 32, 1024)
        c.update(seq=seq, heads=heads, batch=max(1, min(32, int(8192 // seq) or 1, _log(rng, 1, 32))),
                 mask=rng.random() < 0.5, p=rng.choice([0.0, 0.1]))
    elif kind == "norm":
        h = rng.choice(LN_WIDTHS)
        c.update(hidden=h, rows=_log(rng, 32, (16 << 20) // h), p=rng.choice([0.0, 0.0, 0.1]),
                 residual=rng.random() < 0.7)
    elif kind == "embedding":
        seq = _log(rng, 32, 512)
        c.update(seq=seq, batch=max(1, min(32, _log(rng, 1, 32))), vocab=width(1000, 50304),
                 hidden=rng.choice([256, 512, 768, 1024]))
    elif kind == "head":
        c.update(rows=_log(rng, 64, 8192), hidden=rng.choice([256, 512, 768, 1024]), vocab=_log(rng, 1000, 30522),
                 labelled=rng.choice([0.15, 0.15, 1.0]))
    else:
        c["train"] = True            # evaluation uses the running statistics, which is not the kernels' path
        size = rng.choice([7, 14, 28, 28, 56])
        top = {7: 1024, 14: 1024, 28: 512, 56: 256}[size]
        k = rng.choice([1, 3])
        c.update(size=size, images=_log(rng, 2, 32), k=k, inp=_log(rng, 64, top, 64), out=_log(rng, 64, top, 64),
                 residual=rng.random() < 0.4)
    return c


# ----------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * (seed + 1))


def _randn(g, *shape, std=1.0, dtype=torch.float32):
    return (torch.randn(*shape, generator=g, device="cuda") * std).to(dtype)


def _params(values, flat):
    """Leaves for the given tensors; ``flat``: views of one buffer per element type with fp32 gradient views."""
    if not flat:
        return [v.clone().requires_grad_(True) for v in values], []
    out, grads = [None] * len(values), []
    for dt in sorted({v.dtype for v in values}, key=str):
        own = [i for i, v in enumerate(values) if v.dtype == dt]
        starts, end = [], 0
        for i in own:
            starts.append(end)
            end += (values[i].numel() + 63) // 64 * 64
        buf = torch.empty(end, dtype=dt, device="cuda")
        grad = torch.zeros(end, dtype=torch.float32, device="cuda")
        for i, a in zip(own, starts):
            n = values[i].numel()
            buf[a:a + n] = values[i].reshape(-1)
            p = nn.Parameter(buf[a:a + n].view(values[i].shape))
            p.main_grad = grad[a:a + n].view(values[i].shape)
            out[i] = p
        grads.append(grad)
    return out, grads


def _inputs(case, seed):
    """Everything one case works on, as plain tensors made from the seed alone: (params, activations, constants)."""
    g, dt, kind = _gen(seed), DT[case["dtype"]], case["kind"]
    if kind == "linear":
        K, N, R = case["inp"], case["out"], case["rows"]
        return ([_randn(g, N, K, std=K ** -0.5, dtype=dt), _randn(g, N, std=0.1, dtype=dt)],
                [_randn(g, R, K, dtype=dt)], {"dy": _randn(g, R, N, dtype=dt)})
    if kind == "mlp":
        H, I, R = case["hidden"], case["inner"], case["rows"]
        return ([_randn(g, I, H, std=H ** -0.5, dtype=dt), _randn(g, I, std=0.1, dtype=dt),
                 _randn(g, H, I, std=I ** -0.5, dtype=dt), _randn(g, H, std=0.1, dtype=dt)],
                [_randn(g, R, H, dtype=dt)], {"dy": _randn(g, R, H, dtype=dt)})
    if kind == "attention":
        B, S, H = case["batch"], case["seq"], 64 * case["heads"]
        ws = [_randn(g, H, H, std=H ** -0.5, dtype=dt) for _ in range(3)]
        bs = [_randn(g, H, std=0.1, dtype=dt) for _ in range(3)]
        const = {"dy": _randn(g, B, S, H, dtype=dt), "bias": None}
        if case["mask"]:
            # sequences of different lengths, padded: masked keys get a large negative bias
            n = torch.randint(max(1, S // 2), S + 1, (B, 1), generator=g, device="cuda")
            const["bias"] = (torch.arange(S, device="cuda")[None] >= n).to(dt).mul(-10000.0).view(B, 1, 1, S)
        return ws + bs, [_randn(g, B, S, H, dtype=dt)], const
    if kind == "norm":
        R, H = case["rows"], case["hidden"]
        xs = [_randn(g, R, H, dtype=dt)] + ([_randn(g, R, H, dtype=dt)] if case["residual"] else [])
        return ([_randn(g, H, std=0.1, dtype=dt) + 1, _randn(g, H, std=0.1, dtype=dt)], xs,
                {"dy": _randn(g, R, H, dtype=dt)})
    if kind == "embedding":
        B, S, V, H = case["batch"], case["seq"], case["vocab"], case["hidden"]
        # log-uniform ranks: token frequencies fall like 1 / rank, as in text
        ids = torch.exp(torch.rand(B, S, generator=g, device="cuda") * math.log(V)).long().clamp_(1, V) - 1
        seg = (torch.arange(S, device="cuda") >= S // 2).long().expand(B, S).contiguous()
        pos = torch.arange(S, device="cuda")[None]
        return ([_randn(g, V, H, std=0.02, dtype=dt), _randn(g, 512, H, std=0.02, dtype=dt),
                 _randn(g, 2, H, std=0.02, dtype=dt), _randn(g, H, std=0.1, dtype=dt) + 1,
                 _randn(g, H, std=0.1, dtype=dt)], [], {"ids": ids, "seg": seg, "pos": pos,
                                                        "dy": _randn(g, B, S, H, std=0.1, dtype=dt)})
    if kind == "head":
        R, H, V = case["rows"], case["hidden"], case["vocab"]
        labels = torch.randint(0, V, (R,), generator=g, device="cuda")
        labels[torch.rand(R, generator=g, device="cuda") >= case["labelled"]] = -100
        labels[0] = V - 1
        Vp = (V + 63) // 64 * 64
        # loss scaling as mixed-precision training has it, so that 16-bit gradients are normal numbers
        return ([_randn(g, Vp, H, std=0.05, dtype=dt), _randn(g, Vp, std=0.02, dtype=dt)],
                [_randn(g, R, H, dtype=dt)], {"labels": labels, "scale": torch.tensor(4096.0, device="cuda")})
    if kind == "conv":
        N, S, Ci, Co, k = case["images"], case["size"], case["inp"], case["out"], case["k"]
        cl = lambda c, std=1.0: _randn(g, N, S, S, c, std=std, dtype=dt).permute(0, 3, 1, 2)  # noqa: E731
        ps = [_randn(g, Co, Ci, k, k, std=(Ci * k * k) ** -0.5, dtype=dt), _randn(g, Co, std=0.1) + 1,
              _randn(g, Co, std=0.1)]
        xs = [cl(Ci).relu()] + ([cl(Co).relu()] if case["residual"] else [])
        return ps, xs, {"dy": cl(Co)}
    raise ValueError(kind)


# ----------------------------------------------------------------------------------------------- the user's model
class _Layer(nn.Module):
    def __init__(self, hid, heads):
        super().__init__()
        self.heads = heads
        self.q, self.k, self.v, self.o = (nn.Linear(hid, hid) for _ in range(4))
        self.up, self.down = nn.Linear(hid, 4 * hid), nn.Linear(4 * hid, hid)
        self.n1, self.n2 = nn.LayerNorm(hid), nn.LayerNorm(hid)

    def forward(self, x):
        B, S, H = x.shape
        q, k, v = (f(x).view(B, S, self.heads, 64).transpose(1, 2) for f in (self.q, self.k, self.v))
        a = F.scaled_dot_product_attention(q, k, v).transpose(1, 2).reshape(B, S, H)
        x = self.n1(self.o(a) + x)
        return self.n2(self.down(F.gelu(self.up(x))) + x)


class _Encoder(nn.Module):
    """A masked-LM encoder as a user would write it; returns the loss."""

    def __init__(self, case):
        super().__init__()
        hid, self.vocab = case["hidden"], case["vocab"]
        self.words = nn.Embedding((self.vocab + 63) // 64 * 64, hid)
        self.places = nn.Embedding(512, hid)
        self.norm = nn.LayerNorm(hid)
        self.layers = nn.ModuleList(_Layer(hid, case["heads"]) for _ in range(case["layers"]))
        self.bias = nn.Parameter(torch.zeros(self.words.num_embeddings))
        nn.init.normal_(self.words.weight, std=0.02)
        nn.init.normal_(self.places.weight, std=0.02)

    def forward(self, ids, pos, labels):
        x = self.norm(self.words(ids) + self.places(pos))
        for layer in self.layers:
            x = layer(x)
        logits = F.linear(x, self.words.weight, self.bias)
        V = self.vocab
        return F.cross_entropy(logits[..., :V].reshape(-1, V).float(), labels.reshape(-1), ignore_index=-100)


def _step_model(case, seed):
    with torch.random.fork_rng(devices=[]):
        torch.manual_seed(seed)
        net = _Encoder(case)
        B, S, V = case["batch"], case["seq"], case["vocab"]
        ids = torch.exp(torch.rand(B, S) * math.log(V)).long().clamp_(1, V) - 1
        labels = torch.where(torch.rand(B, S) < 0.15, ids, torch.full_like(ids, -100))
    pos = torch.arange(S).expand(B, S).contiguous()
    return net, tuple(t.cuda() for t in (ids, pos, labels))


def _reported(named):
    """Gradients that are compared: all but those of the key biases, which are zero but for rounding."""
    return {n: p for n, p in named if not n.endswith("k.bias")}


# ----------------------------------------------------------------------------------------------- one pass
def prepare(case, seed):
    if case["kind"] == "step":
        import logging

        import rannc_b200

        logging.getLogger("rannc").setLevel(logging.WARNING)
        net, batch = _step_model(case, seed)
        opt = torch.optim.Adam(net.parameters(), lr=1e-5)
        model = rannc_b200.RaNNCModule(net, opt, enable_apex_amp=True)
        with torch.no_grad():
            model(*batch)          # partitions and deploys the model
        return {"case": case, "model": model, "opt": opt, "batch": batch}
    values, xs, const = _inputs(case, seed)
    params, grads = _params(values, case["flat"])
    st = dict(case=case, params=params, grads=grads, xs=[x.requires_grad_(case["train"]) for x in xs], **const)
    if case["kind"] == "conv":
        st["run_mean"] = torch.zeros(case["out"], device="cuda")
        st["run_var"] = torch.ones(case["out"], device="cuda")
    return st


def _forward(st):
    from rannc_b200.ops import functional as RF

    case, ps, xs = st["case"], st["params"], st["xs"]
    kind = case["kind"]
    if case.get("p", 0.0) > 0.0:
        RF.manual_seed(11)
    if kind == "linear":
        return RF.linear(xs[0], ps[0], ps[1], act="gelu" if case["gelu"] else None)
    if kind == "mlp":
        return RF.mlp(xs[0], *ps)
    if kind == "attention":
        wq, wk, wv, bq, bk, bv = ps
        return RF.qkv_attention(xs[0], wq, bq, wk, bk, wv, bv, attn_mask=st["bias"], dropout_p=case["p"],
                                num_heads=case["heads"])
    if kind == "norm":
        return RF.dropout_add_layer_norm(xs[0], xs[1] if case["residual"] else None, ps[0], ps[1], case["p"], 1e-12)
    if kind == "embedding":
        e = RF.embedding(ps[0], st["ids"]) + RF.embedding(ps[1], st["pos"]) + RF.embedding(ps[2], st["seg"])
        return RF.dropout_add_layer_norm(e, None, ps[3], ps[4], 0.0, 1e-12)
    if kind == "head":
        return RF.cross_entropy(RF.linear(xs[0], ps[0], ps[1]), st["labels"], num_classes=case["vocab"])
    y = RF.conv2d(xs[0], ps[0], None, 1, case["k"] // 2)
    return RF.batch_norm_act(y, ps[1], ps[2], st["run_mean"], st["run_var"], True, 0.1, 1e-5, True,
                             xs[1] if case["residual"] else None)


def run(st):
    case = st["case"]
    if case["kind"] == "step":
        model, opt = st["model"], st["opt"]
        opt.zero_grad()
        loss = model(*st["batch"])
        loss.backward()
        opt.step()
        named = _reported(model.named_parameters())
        return {"loss": loss.detach(), "grads": {n: p.main_grad for n, p in named.items()},
                "weights": {n: model.get_local_param_segment(n) for n, p in named.items() if p.dim() > 1}}
    if not case["train"]:
        with torch.no_grad():
            y = _forward(st)
        return [y, st["run_mean"], st["run_var"]] if case["kind"] == "conv" else [y]
    for g in st["grads"]:
        g.zero_()
    for t in st["xs"] + ([] if case["flat"] else st["params"]):
        t.grad = None
    y = _forward(st)
    y.backward(st["scale"] if case["kind"] == "head" else st["dy"])
    out = [y.detach()] + [x.grad for x in st["xs"]] + [p.main_grad if case["flat"] else p.grad for p in st["params"]]
    if case["kind"] == "attention":
        del out[-2]                  # the key biases' gradient is zero but for rounding
    if case["kind"] == "conv":
        out += [st["run_mean"], st["run_var"]]
    return out


# ----------------------------------------------------------------------------------------------- what a pass costs
def work(case):
    kind = case["kind"]
    if kind == "step":
        H, L, R = case["hidden"], case["layers"], case["batch"] * case["seq"]
        V = (case["vocab"] + 63) // 64 * 64
        mat = L * 12 * H * H + V * H
        n = mat + L * 13 * H + 514 * H + V
        att = L * 2 * 2 * R * case["seq"] * H
        # fp32 master weights and two moments read and written, gradients cleared, written and read, 16-bit weights
        return {"bytes": n * (24 + 12 + 4), "flops": 6.0 * R * mat + 3.5 * att}
    tr, gb = case["train"], 4 if case["flat"] else 2
    if kind in ("linear", "mlp"):
        R = case["rows"]
        i, o = (case["inp"], case["out"]) if kind == "linear" else (case["hidden"], case["hidden"])
        w = i * o if kind == "linear" else 2 * i * case["inner"]
        return {"bytes": (2 * w + 2 * R * (i + o)) + (tr and w * (2 + gb) + 2 * R * (i + o)),
                "flops": (6.0 if tr else 2.0) * R * w}
    if kind == "attention":
        H, S = 64 * case["heads"], case["seq"]
        R = case["batch"] * S
        return {"bytes": (6 * H * H + 4 * R * H) + (tr and 3 * H * H * (2 + gb) + 4 * R * H),
                "flops": (3.0 if tr else 1.0) * 6 * R * H * H + (3.5 if tr else 1.0) * 4 * R * S * H}
    if kind == "norm":
        e = case["rows"] * case["hidden"] * 2
        fwd = e * (3 if case["residual"] else 2)
        # backward: dy and the normalised rows in, one or two input gradients out
        return {"bytes": fwd + (tr and e * (4 if case["residual"] and case["p"] > 0 else 3)),
                "flops": 8.0 * e}
    if kind == "embedding":
        R, H, V = case["batch"] * case["seq"], case["hidden"], case["vocab"]
        return {"bytes": 2 * R * H * 2 + (tr and 2 * R * H + (V + 514) * H * gb), "flops": 12.0 * R * H}
    if kind == "head":
        R, H, V = case["rows"], case["hidden"], (case["vocab"] + 63) // 64 * 64
        return {"bytes": 2 * (R * H + V * H) + (tr and 2 * R * H + V * H * (2 + gb)),
                "flops": (6.0 if tr else 2.0) * R * V * H}
    R, k2 = case["images"] * case["size"] ** 2, case["k"] ** 2
    w = case["inp"] * case["out"] * k2
    res = case["out"] if case["residual"] else 0
    one = 2 * R * (case["inp"] + case["out"] + res)
    return {"bytes": (2 * w + one) + (tr and w * (2 + gb) + one + 2 * R * case["inp"]),
            "flops": (6.0 if tr else 2.0) * R * w}


def tolerance(case):
    # about four times what the operators show against 64-bit results: each value is rounded to 16 bits three to
    # five times on its way (1.7e-3 a rounding in bf16, 2.1e-4 in fp16); 0.0028 and 0.00056 were measured
    bf = case["dtype"] == "bf16"
    if case["kind"] == "step":
        return {"rel": 0.05}         # 0.013 measured
    if case["kind"] == "conv":
        # a rounding next to zero flips the ReLU mask of its gradient: 0.0084 measured in fp16
        return {"rel": 0.1 if bf else 0.033}
    return {"rel": 1.2e-2 if bf else 2.5e-3}


# ----------------------------------------------------------------------------------------------- 64-bit results
def exact(case, seed):
    if case.get("p", 0.0) > 0.0:
        return None                  # the dropout mask is the framework's own
    if case["kind"] == "step":
        net, batch = _step_model(case, seed)
        net = net.cuda()
        with torch.no_grad():
            for p in net.parameters():
                p.copy_(p.to(DT[case["dtype"]]))
        loss = _double_step(net.double(), batch)
        named = _reported(net.named_parameters())
        return {"loss": loss, "grads": {n: p.grad for n, p in named.items()},
                "weights": {n: None for n, p in named.items() if p.dim() > 1}}
    values, xs, const = _inputs(case, seed)
    ps = [v.double().requires_grad_(case["train"]) for v in values]
    xs = [x.double().requires_grad_(case["train"]) for x in xs]
    kind, extra = case["kind"], []
    with torch.set_grad_enabled(case["train"]):
        if kind == "linear":
            y = F.linear(xs[0], *ps)
            y = F.gelu(y) if case["gelu"] else y
        elif kind == "mlp":
            y = F.linear(F.gelu(F.linear(xs[0], ps[0], ps[1])), ps[2], ps[3])
        elif kind == "attention":
            B, S, H = xs[0].shape
            q, k, v = (F.linear(xs[0], ps[i], ps[3 + i]).view(B, S, -1, 64).transpose(1, 2) for i in range(3))
            s = q @ k.transpose(2, 3) / 8.0
            if const["bias"] is not None:
                s = s + const["bias"].double()
            y = (torch.softmax(s, -1) @ v).transpose(1, 2).reshape(B, S, H)
        elif kind == "norm":
            y = F.layer_norm(sum(xs), xs[0].shape[-1:], ps[0], ps[1], 1e-12)
        elif kind == "embedding":
            e = ps[0][const["ids"]] + ps[1][const["pos"]] + ps[2][const["seg"]]
            y = F.layer_norm(e, e.shape[-1:], ps[3], ps[4], 1e-12)
        elif kind == "head":
            y = F.cross_entropy(F.linear(xs[0], *ps)[:, :case["vocab"]], const["labels"], ignore_index=-100)
        else:
            y = F.conv2d(xs[0], ps[0], None, 1, case["k"] // 2)
            with torch.no_grad():
                n = y.numel() // y.shape[1]
                extra = [0.1 * y.mean((0, 2, 3)), 0.9 + 0.1 * y.var((0, 2, 3), correction=0) * n / (n - 1)]
            y = F.batch_norm(y, None, None, ps[1], ps[2], True, 0.1, 1e-5)
            y = F.relu(y + xs[1] if case["residual"] else y)
    if not case["train"]:
        return [y] + extra
    y.backward(const["scale"].double() if kind == "head" else const["dy"].double())
    out = [y.detach()] + [x.grad for x in xs] + [p.grad for p in ps] + extra
    if kind == "attention":
        del out[-2]
    return out


def _double_step(net, batch):
    ids, pos, labels = batch
    x = net.norm(net.words(ids) + net.places(pos))
    for layer in net.layers:
        x = layer(x)
    logits = F.linear(x, net.words.weight, net.bias)[..., :net.vocab].reshape(-1, net.vocab)
    loss = F.cross_entropy(logits, labels.reshape(-1), ignore_index=-100)
    loss.backward()
    return loss.detach()
