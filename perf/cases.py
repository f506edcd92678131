"""The workloads whose speed this repository is measured by.

Every case is work that a training program has this framework do, called through the same public functions and
classes: the projections, attention, normalisation, activation and loss of a transformer (forward and backward),
the AdamW update, the DiLoCo synchronisation and one whole training step.  Sizes follow the 8B, 1B and tiny
configurations of ``torchft_b200.models.llama``; ``draw`` spreads them over the ranges that those stand for.
"""

import math

import torch

from torchft_b200.local_sgd import DiLoCo
from torchft_b200.models.llama import Llama, LlamaConfig
from torchft_b200.ops import functional as F
from torchft_b200.ops.attention import attention
from torchft_b200.optim import FusedAdamW
from torchft_b200.parallel.hsdp import HSDPEngine

DEV = "cuda"


def listed():
    return [
        # the fused q/k/v projection of the tiny configuration: launches and latency are all there is
        dict(name="linear_tiny", kind="linear", tokens=512, k=256, n=512),
        # a projection whose token count and widths are no multiple of any tile (packed sequences, odd FFN width)
        dict(name="linear_ragged", kind="linear", tokens=1013, k=2048, n=5464),
        # gate and up projection of the 8B configuration at its 4096 tokens: the largest product of a layer
        dict(name="linear_8b_w13", kind="linear", tokens=4096, k=4096, n=28672),
        # a batch of short sequences that end inside a tile
        dict(name="attention_short", kind="attention", batch=4, seq=544, hq=16, hkv=4, hd=128),
        # attention of the 1B configuration (head dimension 64)
        dict(name="attention_1b", kind="attention", batch=2, seq=2048, hq=32, hkv=8, hd=64),
        # attention of the 8B configuration
        dict(name="attention_8b", kind="attention", batch=1, seq=4096, hq=32, hkv=8, hd=128),
        # residual add + RMSNorm of the 8B configuration
        dict(name="add_rmsnorm_8b", kind="add_rmsnorm", rows=4096, dim=4096),
        # the activation between the MLP projections of the 8B configuration
        dict(name="swiglu_8b", kind="swiglu", rows=4096, f=14336),
        # output projection and loss of the 1B configuration
        dict(name="head_loss_1b", kind="head_loss", tokens=2048, k=2048, vocab=128256),
        # optimizer step of a model trained through DistributedDataParallel: norms of a few KB beside large matrices
        dict(name="adamw_1b", kind="adamw", dim=2048, kv=512, ffn=8192, layers=3, vocab=32000),
        # DiLoCo synchronisation of a replica (pack, pseudo-gradient, outer Nesterov step, unpack)
        dict(name="diloco_1b", kind="diloco", dim=2048, kv=512, ffn=8192, layers=3, vocab=32000, dtype="bf16"),
        # one whole training step, 1B widths with two blocks: forward, backward, fused AdamW
        dict(name="train_step_1b", kind="train_step", dim=2048, layers=2, heads=32, kv_heads=8, ffn=8192, vocab=128256,
             batch=1, seq=2048),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _log_mult(rng, lo, hi, step):
    """A multiple of ``step`` (what the entry points ask of a width), spread over the logarithm."""
    return max(lo, min(hi, _log_int(rng, lo, hi) // step * step))


def draw(rng):
    kind = rng.choice(["linear", "linear", "attention", "attention", "add_rmsnorm", "swiglu", "head_loss", "adamw", "diloco",
                       "train_step"])
    if kind == "linear":
        return dict(kind=kind, tokens=_log_int(rng, 16, 4096), k=_log_mult(rng, 128, 4096, 8), n=_log_mult(rng, 128, 28672, 8))
    if kind == "attention":
        hq, hkv = rng.choice([(32, 8), (16, 4), (8, 8), (16, 2)])
        seq = _log_mult(rng, 64, 4096, 32)  # padded to whole warps of rows, not to whole tiles
        batch = rng.randint(1, 4) if seq <= 2048 else 1
        return dict(kind=kind, batch=batch, seq=seq, hq=hq, hkv=hkv, hd=rng.choice([64, 128]))
    if kind == "add_rmsnorm":
        return dict(kind=kind, rows=_log_int(rng, 16, 16384), dim=_log_mult(rng, 256, 4096, 256))
    if kind == "swiglu":
        return dict(kind=kind, rows=_log_int(rng, 16, 8192), f=_log_mult(rng, 256, 14336, 8))
    if kind == "head_loss":
        return dict(kind=kind, tokens=_log_int(rng, 64, 2048), k=_log_mult(rng, 256, 2048, 8), vocab=_log_mult(rng, 1000, 128256, 8))
    if kind in ("adamw", "diloco"):
        case = dict(kind=kind, dim=_log_mult(rng, 256, 2048, 8), layers=rng.randint(1, 3), vocab=_log_int(rng, 1000, 32000))
        case.update(kv=max(64, case["dim"] // 4 // 8 * 8), ffn=_log_mult(rng, 2 * case["dim"], 4 * case["dim"], 8))
        if kind == "diloco":
            case["dtype"] = rng.choice(["bf16", "fp32"])
        return case
    heads, kv_heads, hd = rng.choice([(2, 1, 128), (4, 2, 128), (8, 2, 64), (16, 4, 64), (8, 4, 128)])
    dim = heads * hd
    return dict(kind=kind, dim=dim, layers=rng.randint(1, 3), heads=heads, kv_heads=kv_heads, ffn=_log_mult(rng, 2 * dim, 4 * dim, 64),
                vocab=_log_mult(rng, 1000, 32000, 8), batch=rng.randint(1, 2), seq=_log_mult(rng, 128, 1024, 32))


# ---------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(gen, shape, std=1.0, dtype=torch.bfloat16):
    return torch.empty(shape, dtype=dtype, device=DEV).normal_(0.0, std, generator=gen)


def _shapes(case):
    """Parameter shapes of a decoder in the order in which a program lists them."""
    d, kv, ffn = case["dim"], case["kv"], case["ffn"]
    shapes = [(case["vocab"], d)]
    for _ in range(case["layers"]):
        shapes += [(d,), (d + 2 * kv, d), (d, d), (d,), (2 * ffn, d), (d, ffn)]
    return shapes + [(d,), (case["vocab"], d)]


def _numel(case):
    return sum(math.prod(s) for s in _shapes(case))


def _config(case):
    return LlamaConfig(dim=case["dim"], n_layers=case["layers"], n_heads=case["heads"], n_kv_heads=case["kv_heads"],
                       ffn_dim=case["ffn"], vocab_size=case["vocab"], max_seq_len=case["seq"])


def _llama_shapes(case):
    d, hd, ffn = case["dim"], case["dim"] // case["heads"], case["ffn"]
    shapes = {"tok_embeddings": (case["vocab"], d), "norm": (d,), "output": (case["vocab"], d)}
    for i in range(case["layers"]):
        shapes.update({f"layers.{i}.attn_norm": (d,), f"layers.{i}.wqkv": ((case["heads"] + 2 * case["kv_heads"]) * hd, d),
                       f"layers.{i}.wo": (d, case["heads"] * hd), f"layers.{i}.ffn_norm": (d,), f"layers.{i}.w13": (2 * ffn, d),
                       f"layers.{i}.w2": (d, ffn)})
    return shapes


def _inputs(case, seed):
    g, kind = _gen(seed), case["kind"]
    if kind == "linear":
        t, k, n = case["tokens"], case["k"], case["n"]
        return dict(x=_randn(g, (t, k)), w=_randn(g, (n, k), 0.02), dy=_randn(g, (t, n), 0.1))
    if kind == "attention":
        b, s, hq, hkv, hd = (case[c] for c in ("batch", "seq", "hq", "hkv", "hd"))
        return dict(q=_randn(g, (b, s, hq, hd)), k=_randn(g, (b, s, hkv, hd)), v=_randn(g, (b, s, hkv, hd)),
                    do=_randn(g, (b, s, hq, hd)))
    if kind == "add_rmsnorm":
        shape = (case["rows"], case["dim"])
        return dict(x=_randn(g, shape), res=_randn(g, shape), w=1 + _randn(g, shape[1:], 0.1), dy=_randn(g, shape, 0.1),
                    dh=_randn(g, shape, 0.1))
    if kind == "swiglu":
        return dict(gu=_randn(g, (case["rows"], 2 * case["f"])), dout=_randn(g, (case["rows"], case["f"]), 0.1))
    if kind == "head_loss":
        t, k, v = case["tokens"], case["k"], case["vocab"]
        return dict(x=_randn(g, (t, k)), w=_randn(g, (v, k), 0.02), targets=torch.randint(v, (t,), generator=g, device=DEV))
    if kind == "adamw":
        return dict(p=[_randn(g, s, 0.02) if len(s) > 1 else 1 + _randn(g, s, 0.02) for s in _shapes(case)],
                    g=[_randn(g, s, 1e-3) for s in _shapes(case)])
    if kind == "diloco":
        dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
        start = [_randn(g, s, 0.02, dtype) for s in _shapes(case)]
        # what a few inner steps leave behind: every weight a few percent away from the last global one
        return dict(start=start, local=[p + _randn(g, p.shape, 2e-3, dtype) for p in start])
    assert kind == "train_step"
    shape, v = (case["batch"], case["seq"]), case["vocab"]
    weights = {name: torch.ones(s, dtype=torch.bfloat16, device=DEV) if len(s) == 1 else _randn(g, s, 0.02)
               for name, s in _llama_shapes(case).items()}
    return dict(weights=weights, tokens=torch.randint(v, shape, generator=g, device=DEV),
                targets=torch.randint(v, shape, generator=g, device=DEV))


class _SoloManager:
    """The manager of a replica that is alone in its group: its votes pass and its averages are its own values.  The real
    one adds the waits of the control plane (quorum, vote), which no device code can shorten."""

    _use_async_quorum = False

    def start_quorum(self):
        pass

    def allreduce(self, tensor):
        done = torch.futures.Future()
        done.set_result(tensor)
        return done

    def should_commit(self):
        return True


OUTER_LR, OUTER_MOMENTUM = 0.7, 0.9


def prepare(case, seed):
    st, kind = _inputs(case, seed), case["kind"]
    st["kind"] = kind
    for name in ("x", "w", "q", "k", "v", "res", "gu"):
        if name in st:
            st[name].requires_grad_()
    if kind == "adamw":
        st["params"] = [torch.nn.Parameter(p) for p in st.pop("p")]
        for p, grad in zip(st["params"], st.pop("g")):
            p.grad = grad
        st["opt"] = FusedAdamW(st["params"], lr=1e-3)
    elif kind == "diloco":
        model = torch.nn.ParameterList(torch.nn.Parameter(p) for p in st.pop("start"))
        st["params"] = list(model)
        inner = torch.optim.SGD(model.parameters(), lr=0.0)
        st["outer"] = torch.optim.SGD(model.parameters(), lr=OUTER_LR, momentum=OUTER_MOMENTUM, nesterov=True)
        st["diloco"] = DiLoCo(_SoloManager(), model, inner, st["outer"], sync_every=100)
        with torch.no_grad():
            for p, value in zip(st["params"], st.pop("local")):
                p.copy_(value)
    elif kind == "train_step":
        model = Llama(_config(case), device=DEV)
        with torch.no_grad():
            for (name, p), (ours, value) in zip(model.named_parameters(), st.pop("weights").items()):
                assert name == ours
                p.copy_(value)
        st["model"] = model
        st["engine"] = HSDPEngine(model, model.units())
    return st


def run(st):
    kind = st["kind"]
    if kind == "linear":
        y = F.linear(st["x"], st["w"])
        return (y.detach(), *torch.autograd.grad(y, (st["x"], st["w"]), st["dy"]))
    if kind == "attention":
        o = attention(st["q"], st["k"], st["v"])
        return (o.detach(), *torch.autograd.grad(o, (st["q"], st["k"], st["v"]), st["do"]))
    if kind == "add_rmsnorm":
        y, h = F.add_rmsnorm(st["x"], st["res"], st["w"])
        dx, dres, dw = torch.autograd.grad((y, h), (st["x"], st["res"], st["w"]), (st["dy"], st["dh"]))
        return y.detach(), h.detach(), dx, dres, dw
    if kind == "swiglu":
        out = F.swiglu(st["gu"])
        return (out.detach(), *torch.autograd.grad(out, (st["gu"],), st["dout"]))
    if kind == "head_loss":
        loss = F.cross_entropy(F.linear(st["x"], st["w"]), st["targets"])
        return (loss.detach(), *torch.autograd.grad(loss, (st["x"], st["w"])))
    if kind == "adamw":
        st["opt"].step()
        state = [st["opt"].state[p] for p in st["params"]]
        return [p.detach() for p in st["params"]], [s["exp_avg"] for s in state], [s["exp_avg_sq"] for s in state]
    if kind == "diloco":
        st["diloco"].sync()
        state = [st["outer"].state[p]["momentum_buffer"] for p in st["params"]]
        return [p.detach() for p in st["params"]], list(st["diloco"]._backup_parameters.values()), state
    engine = st["engine"]
    loss = engine.train_step(st["tokens"], st["targets"])
    engine.gather_parameters()  # the caller's stream sees the updated weights, as before an evaluation
    params = list(st["model"].parameters())
    return loss, [p.main_grad for p in params], [p.detach() for p in params]


def work(case):
    kind = case["kind"]
    if kind == "linear":
        t, k, n = case["tokens"], case["k"], case["n"]
        return dict(bytes=2 * (2 * t * k + 2 * n * k + 2 * t * n), flops=6 * t * k * n)
    if kind == "attention":
        b, s, hq, hkv, hd = (case[c] for c in ("batch", "seq", "hq", "hkv", "hd"))
        # q, o, do, dq and k, v, dk, dv; two products forward and five backward over the causal half
        return dict(bytes=2 * b * s * hd * 4 * (hq + hkv), flops=7 * b * hq * s * (s + 1) * hd)
    if kind == "add_rmsnorm":
        n = case["rows"] * case["dim"]
        return dict(bytes=2 * (4 * n + 2 * n) + 4 * case["dim"], flops=12 * n)
    if kind == "swiglu":
        n = case["rows"] * case["f"]
        return dict(bytes=2 * n * (2 + 1 + 1 + 2), flops=15 * n)
    if kind == "head_loss":
        t, k, v = case["tokens"], case["k"], case["vocab"]
        return dict(bytes=2 * (2 * t * k + 2 * v * k) + 8 * t, flops=6 * t * k * v)
    if kind == "adamw":
        return dict(bytes=22 * _numel(case), flops=15 * _numel(case))
    if kind == "diloco":
        size = 2 if case["dtype"] == "bf16" else 4  # weights and backup in and out, fp32 momentum in and out
        return dict(bytes=(4 * size + 8) * _numel(case), flops=6 * _numel(case))
    cfg, tokens = _config(case), case["batch"] * case["seq"]
    return dict(bytes=22 * cfg.num_params() + 16 * tokens, flops=int(cfg.flops_per_token(case["seq"]) * tokens))


def tolerance(case):
    kind = case["kind"]
    if kind == "diloco" and case["dtype"] == "fp32":
        return {"rel": 1e-5}
    # four times the distance from the exact results: 1.7e-3 for one rounding to bf16 of an fp32 sum, 2.5e-3 where
    # attention rounds P and dS on the way, 1.3e-2 for gradients that pass through the roundings of a whole model
    return {"rel": {"attention": 1e-2, "train_step": 5e-2}.get(kind, 8e-3)}


# ---------------------------------------------------------------------------------------- 64-bit results
def _rms(x, w, eps=1e-5):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _attend(q, k, v):
    """Causal attention, one head at a time: [B, S, H, D] with grouped key/value heads."""
    s, group = q.shape[1], q.shape[2] // k.shape[2]
    mask = torch.ones(s, s, dtype=torch.bool, device=q.device).triu(1)
    heads = []
    for h in range(q.shape[2]):
        scores = q[:, :, h] @ k[:, :, h // group].transpose(1, 2) / math.sqrt(q.shape[3])
        heads.append(scores.masked_fill(mask, -math.inf).softmax(-1) @ v[:, :, h // group])
    return torch.stack(heads, 2)


def _rope(x, theta=500000.0):
    s, half = x.shape[1], x.shape[3] // 2
    freq = theta ** (-torch.arange(half, dtype=torch.float64, device=x.device) / half)
    angle = torch.arange(s, dtype=torch.float64, device=x.device)[:, None] * freq
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat((a * cos - b * sin, b * cos + a * sin), -1)


def _llama_loss(case, w, tokens, targets):
    heads, kv_heads, hd, ffn = case["heads"], case["kv_heads"], case["dim"] // case["heads"], case["ffn"]
    b, s = tokens.shape
    h = w["tok_embeddings"][tokens]
    for i in range(case["layers"]):
        p = {name: w[f"layers.{i}.{name}"] for name in ("attn_norm", "wqkv", "wo", "ffn_norm", "w13", "w2")}
        qkv = (_rms(h, p["attn_norm"]) @ p["wqkv"].T).view(b, s, heads + 2 * kv_heads, hd)
        q, k, v = qkv.split((heads, kv_heads, kv_heads), 2)
        h = h + _attend(_rope(q), _rope(k), v).reshape(b, s, heads * hd) @ p["wo"].T
        gate, up = (_rms(h, p["ffn_norm"]) @ p["w13"].T).split(ffn, -1)
        h = h + (torch.nn.functional.silu(gate) * up) @ p["w2"].T
    logits = _rms(h, w["norm"]) @ w["output"].T
    return torch.nn.functional.cross_entropy(logits.view(b * s, -1), targets.view(-1))


def exact(case, seed):
    st, kind = _inputs(case, seed), case["kind"]
    leaf = lambda t: t.double().requires_grad_()  # noqa: E731
    if kind == "linear":
        x, w, dy = (st[n].double() for n in ("x", "w", "dy"))
        return x @ w.T, dy @ w, dy.T @ x
    if kind == "attention":
        q, k, v = leaf(st["q"]), leaf(st["k"]), leaf(st["v"])
        group = case["hq"] // case["hkv"]
        outs, grads = [], [torch.zeros_like(t) for t in (q, k, v)]
        for h in range(case["hq"]):  # a head at a time: the scores of all of them do not fit at 64 bits
            o = _attend(q[:, :, h : h + 1], k[:, :, h // group : h // group + 1], v[:, :, h // group : h // group + 1])
            for total, grad in zip(grads, torch.autograd.grad(o, (q, k, v), st["do"][:, :, h : h + 1].double())):
                total += grad
            outs.append(o.detach())
        return (torch.cat(outs, 2), *grads)
    if kind == "add_rmsnorm":
        x, res, w = leaf(st["x"]), leaf(st["res"]), leaf(st["w"])
        h = x + res
        y = _rms(h, w)
        grads = torch.autograd.grad((y, h), (x, res, w), (st["dy"].double(), st["dh"].double()))
        return (y.detach(), h.detach(), *grads)
    if kind == "swiglu":
        gu = leaf(st["gu"])
        gate, up = gu.split(case["f"], -1)
        out = torch.nn.functional.silu(gate) * up
        return (out.detach(), *torch.autograd.grad(out, (gu,), st["dout"].double()))
    if kind == "head_loss":
        x, w = leaf(st["x"]), leaf(st["w"])
        loss = torch.nn.functional.cross_entropy(x @ w.T, st["targets"])
        return (loss.detach(), *torch.autograd.grad(loss, (x, w)))
    if kind == "adamw":
        new, ms, vs = [], [], []
        for p, g in zip(st["p"], st["g"]):
            p, g = p.double(), g.double()
            ms.append(0.1 * g)
            vs.append(0.001 * g * g)
            new.append(p * (1 - 1e-3 * 1e-2) - 1e-3 * g / (g.abs() + 1e-8))  # first step: both bias corrections cancel
        return new, ms, vs
    if kind == "diloco":
        momentum = [local.double() - start.double() for start, local in zip(st["start"], st["local"])]
        new = [s.double() - OUTER_LR * (1 + OUTER_MOMENTUM) * m for s, m in zip(st["start"], momentum)]
        return new, new, momentum
    weights = {name: leaf(w) for name, w in st["weights"].items()}
    loss = _llama_loss(case, weights, st["tokens"], st["targets"])
    grads = torch.autograd.grad(loss, list(weights.values()))
    return loss.detach(), list(grads), [None] * len(grads)
