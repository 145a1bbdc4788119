"""What the performance of this package is judged by: twelve calls that its users make, and a way to draw more like them.

Every case has a ``kind``; a kind is one public entry point with the sizes that the race driver, the tests and the benchmarks give it:

  v2       ``SuperGrok2.step`` on all tensors of a race decoder (the optimizer that the headline benchmark times)
  element  ``step`` of an element-wise optimizer (AdamW, GrokAdamW, SuperGrok v1.5) on the same models
  muon     ``Muon.step`` on the matrices of decoder blocks
  bilevel  ``SuperGrok2.bilevel_step``: one meta-learning update through model, scan, routing and experts
  norm     LayerNorm / RMSNorm with the residual add, forward and backward
  attn     causal attention over the race's 4- and 8-token sequences, forward and backward
  ce       cross-entropy over a vocabulary, forward and backward
  flash    causal / full flash attention, forward and backward
  model    forward, loss and backward of the whole race decoder

``exact`` restates each of them in 64 bits with plain torch operations."""
import math
import random

import torch
import torch.nn.functional as F

DEV = "cuda"
DT = {"f32": torch.float32, "bf16": torch.bfloat16}


def listed():
    return [
        # the race's default model (422,755 parameters): the smallest step a user takes, bound by launches and short kernels
        {"name": "v2_race", "kind": "v2", "layers": 2, "d": 128, "ntok": 99, "dtype": "f32"},
        # the headline model (19.0 M parameters): the step that the flagship benchmark times
        {"name": "v2_flagship", "kind": "v2", "layers": 6, "d": 512, "ntok": 115, "dtype": "f32"},
        # an element-wise optimizer of the race on the headline model, with its global clip
        {"name": "grokadamw_flagship", "kind": "element", "opt": "grokadamw", "layers": 6, "d": 512, "ntok": 115, "dtype": "f32"},
        # Muon on the race's medium model: sixteen small matrices
        {"name": "muon_medium", "kind": "muon", "layers": 4, "d": 256, "ff": 1024, "fused_qkv": True},
        # Muon on two blocks of the 1.3 B decoder: fourteen large matrices
        {"name": "muon_llama", "kind": "muon", "layers": 2, "d": 2048, "ff": 5504, "fused_qkv": False},
        # meta-learning update on the race's default model (512 training examples a batch)
        {"name": "bilevel_race", "kind": "bilevel", "layers": 2, "d": 128, "ntok": 99, "batch": 512, "interval": 32},
        # LayerNorm of the headline model: 8,192 sequences of four tokens
        {"name": "layernorm_flagship", "kind": "norm", "rms": False, "rows": 32768, "d": 512, "dtype": "bf16"},
        # RMSNorm of the 1.3 B decoder, which hands the residual stream on
        {"name": "rmsnorm_llama", "kind": "norm", "rms": True, "rows": 16384, "d": 2048, "dtype": "bf16"},
        # attention of the headline model
        {"name": "attention_flagship", "kind": "attn", "batch": 8192, "seq": 4, "heads": 8, "hd": 64, "dtype": "bf16"},
        # loss of the 1.3 B decoder over 8,192 tokens
        {"name": "cross_entropy_llama", "kind": "ce", "rows": 8192, "vocab": 32000, "dtype": "bf16"},
        # attention of the 1.3 B decoder on the hand-written kernels
        {"name": "flash_llama", "kind": "flash", "batch": 4, "seq": 2048, "heads": 16, "hd": 128, "causal": True},
        # the whole headline model, forward, loss and backward
        {"name": "model_flagship", "kind": "model", "layers": 6, "d": 512, "heads": 8, "ntok": 115, "batch": 8192, "dtype": "bf16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["v2", "v2", "element", "muon", "muon", "bilevel", "norm", "norm", "attn", "ce", "flash", "model"])
    if kind == "v2":
        return {"kind": kind, "layers": rng.randint(1, 6), "d": 4 * _log(rng, 12, 128), "ntok": rng.randint(20, 200), "dtype": rng.choice(["f32", "f32", "bf16"])}
    if kind == "element":
        return {"kind": kind, "opt": rng.choice(["adamw", "grokadamw", "supergrok15"]), "layers": rng.randint(1, 6), "d": 4 * _log(rng, 12, 128),
                "ntok": rng.randint(20, 200), "dtype": rng.choice(["f32", "bf16"])}
    if kind == "muon":
        d = 8 * _log(rng, 8, 256)
        return {"kind": kind, "layers": rng.randint(1, 6 if d <= 768 else 2), "d": d, "ff": 8 * int(d * rng.uniform(2.0, 4.0) / 8), "fused_qkv": rng.random() < 0.5}
    if kind == "bilevel":
        return {"kind": kind, "layers": rng.randint(1, 3), "d": 4 * _log(rng, 12, 40), "ntok": rng.randint(20, 200), "batch": _log(rng, 64, 1024),
                "interval": rng.choice([1, 16, 32, 64])}
    if kind == "norm":
        d = 4 * _log(rng, 16, 768)
        return {"kind": kind, "rms": rng.random() < 0.5, "rows": _log(rng, 16, max(32, min(65536, 33000000 // d))), "d": d, "dtype": rng.choice(["bf16", "bf16", "f32"])}
    if kind == "attn":
        return {"kind": kind, "batch": _log(rng, 16, 8192), "seq": rng.choice([4, 4, 8]), "heads": rng.randint(1, 8), "hd": rng.choice([32, 64]),
                "dtype": rng.choice(["bf16", "bf16", "f32"])}
    if kind == "ce":
        vocab = 8 * _log(rng, 12, 4000)
        return {"kind": kind, "rows": _log(rng, 16, min(32768, 262000000 // vocab)), "vocab": vocab, "dtype": rng.choice(["bf16", "bf16", "f32"])}
    if kind == "flash":
        seq = 128 * rng.randint(1, 16)
        return {"kind": kind, "batch": rng.randint(1, 4), "seq": seq, "heads": rng.randint(1, 16), "hd": rng.choice([64, 128]), "causal": rng.random() < 0.8}
    heads = rng.choice([4, 8])
    return {"kind": "model", "layers": rng.randint(1, 6), "d": heads * rng.choice([32, 64]), "heads": heads, "ntok": rng.randint(20, 200), "batch": _log(rng, 64, 8192),
            "dtype": rng.choice(["bf16", "bf16", "f32"])}


# ---------------------------------------------------------------------------------------------------- inputs

def _decoder_shapes(c):
    """Shapes of the parameters of the race decoder (embeddings, post-LN blocks with a 4 d MLP, final norm, head), in its order."""
    d, ntok = c["d"], c["ntok"]
    block = [(3 * d, d), (3 * d,), (d, d), (d,), (d,), (d,), (d,), (d,), (4 * d, d), (4 * d,), (d, 4 * d), (d,)]
    return [(ntok, d), (4, d)] + block * c["layers"] + [(d,), (d,), (ntok, d), (ntok,)]


def _muon_shapes(c):
    d, ff = c["d"], c["ff"]
    block = [(3 * d, d), (d, d), (ff, d), (d, ff)] if c["fused_qkv"] else [(d, d)] * 4 + [(ff, d)] * 2 + [(d, ff)]
    return block * c["layers"]


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(g, shape, scale=1.0, dtype=torch.float32):
    return (torch.randn(shape, generator=g, device=DEV) * scale).to(dtype)


def _tensors(shapes, g, dtype):
    """Parameters as a model initialises them (matrices N(0, 1/sqrt(fan in)), vectors near one) and gradients N(0, 1e-3)."""
    ps = []
    for s in shapes:
        p = _randn(g, s, s[-1] ** -0.5) if len(s) == 2 else 1.0 + _randn(g, s, 0.02)
        p = torch.nn.Parameter(p.to(dtype))
        p.grad = _randn(g, s, 1e-3, dtype)
        ps.append(p)
    return ps


def _meta_weights(meta_net, g):
    """A meta-network some way into meta-training: every weight away from the symmetric values it starts from."""
    sd = {}
    for k, v in meta_net.state_dict().items():
        if not v.is_floating_point():
            sd[k] = v.clone()
            continue
        v = _randn(g, v.shape)
        if "A_log" in k:
            v = 0.05 * v + torch.log(torch.arange(1, v.shape[1] + 1, device=DEV, dtype=torch.float32))
        elif k.endswith(".D"):
            v = 1.0 + 0.1 * v
        elif "rope" in k:
            v = 0.05 * v
        elif "expert_W" in k:
            v = 0.2 * v
        elif "bias" in k or "expert_b" in k:
            v = 0.05 * v
        elif "product_keys" in k:
            v = 0.3 * v
        elif v.dim() == 2:
            v = v * v.shape[1] ** -0.5
        sd[k] = v
    return sd


def _resume(opt, ps, g, v2):
    """Puts ``opt`` where a checkpoint of step 149 leaves it (moments, sharpness and, for v2, GRU and scan states)."""
    state = {}
    for i, p in enumerate(ps):
        n = p.numel()
        st = {"step": 149, "exp_avg": _randn(g, (n,), 3e-4), "exp_avg_sq": _randn(g, (n,), 1e-3).square(), "mu": _randn(g, (n,), 1e-4),
              "sharpness": _randn(g, (n,), 1e-3).abs()}
        if v2:
            st["gru_state"] = _randn(g, (n, 4), 0.1)
            st["mamba_fwd_state"], st["mamba_bwd_state"] = _randn(g, (16, 16), 0.01), _randn(g, (16, 16), 0.01)
        state[i] = st
    extra = {"global_step": 149, "cached_alpha": 0.97, "cached_train_acc": 0.5, "flat_steps": [149] * len(ps)}
    if v2:
        extra.update(step_counter=149, meta_net=_meta_weights(opt.meta_net, g))
    opt.load_state_dict({"state": state, "param_groups": opt.state_dict()["param_groups"], "extra": extra})


def _v2_optimizer(ps, g, **kw):
    from supergrok15_b200 import SuperGrok2
    opt = SuperGrok2(ps, recycle_interval=0, **kw)      # without the periodic expert recycling, which draws at random
    opt.meta_net.to(DEV)
    _resume(opt, ps, g, True)
    return opt


def _prepare_v2(c, seed):
    g = _gen(seed)
    ps = _tensors(_decoder_shapes(c), g, DT[c["dtype"]])
    opt = _v2_optimizer(ps, g)
    return {"opt": opt, "ps": ps}


def _prepare_element(c, seed):
    from supergrok15_b200 import AdamW, GrokAdamW, SuperGrok15
    g = _gen(seed)
    ps = _tensors(_decoder_shapes(c), g, DT[c["dtype"]])
    if c["opt"] == "supergrok15":
        torch.manual_seed(int(seed))
        opt = SuperGrok15(ps)
        with torch.no_grad():
            for p in opt.meta_net.parameters():
                p.copy_(_randn(g, p.shape, 0.1))
        _resume(opt, ps, g, False)
    else:
        opt = (AdamW if c["opt"] == "adamw" else GrokAdamW)(ps)
        names = ("exp_avg", "exp_avg_sq", "ema") if c["opt"] == "grokadamw" else ("exp_avg", "exp_avg_sq")
        for p in ps:
            st = opt.state[p]
            st["step"] = 149
            for k in names:
                v = _randn(g, p.shape, 1e-3)
                st[k] = v.square() if k == "exp_avg_sq" else 0.3 * v
    return {"opt": opt, "ps": ps}


def _prepare_muon(c, seed):
    from supergrok15_b200 import Muon
    g = _gen(seed)
    ps = _tensors(_muon_shapes(c), g, torch.float32)
    opt = Muon(ps)
    for p in ps:
        opt.state[p]["momentum_buffer"] = _randn(g, p.shape, 1e-3)
    return {"opt": opt, "ps": ps}


def _decoder(c, g, dtype):
    from supergrok15_b200.models import Transformer
    m = Transformer(c["layers"], c["d"], c.get("heads", 4), c["ntok"], 4).to(DEV)
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(_randn(g, p.shape, p.shape[-1] ** -0.5 if p.dim() == 2 else 0.02))
        for mod in m.modules():
            if isinstance(mod, torch.nn.LayerNorm):
                mod.weight.add_(1.0)
    return m.to(dtype)


def _prepare_bilevel(c, seed):
    g = _gen(seed)
    model = _decoder(c, g, torch.float32)
    ps = list(model.parameters())
    for p in ps:
        p.grad = _randn(g, p.shape, 1e-3)
    opt = _v2_optimizer(ps, g, bilevel_checkpoint_interval=c["interval"])
    meta = torch.optim.Adam(opt.meta_net.parameters(), lr=1e-4)
    ids = [torch.randint(0, c["ntok"], (c["batch"], 4), generator=g, device=DEV) for _ in range(2)]
    ys = [torch.randint(0, c["ntok"], (c["batch"],), generator=g, device=DEV) for _ in range(2)]
    return {"opt": opt, "model": model, "meta": meta, "x": ids, "y": ys}


def _prepare_norm(c, seed):
    g, dt, shape = _gen(seed), DT[c["dtype"]], (c["rows"], c["d"])
    s = {"x": _randn(g, shape, 1.0, dt).requires_grad_(), "r": _randn(g, shape, 1.0, dt).requires_grad_(),
         "w": (1.0 + _randn(g, (c["d"],), 0.1)).to(dt).requires_grad_(), "dy": _randn(g, shape, 1.0, dt), "rms": c["rms"]}
    if c["rms"]:
        s["dz"] = _randn(g, shape, 1.0, dt)
    else:
        s["b"] = _randn(g, (c["d"],), 0.1, dt).requires_grad_()
    return s


def _prepare_attn(c, seed):
    g, dt, d = _gen(seed), DT[c["dtype"]], c["heads"] * c["hd"]
    return {"qkv": _randn(g, (c["batch"], c["seq"], 3 * d), 1.0, dt).requires_grad_(), "do": _randn(g, (c["batch"], c["seq"], d), 1.0, dt), "heads": c["heads"]}


def _prepare_ce(c, seed):
    g = _gen(seed)
    t = torch.randint(0, c["vocab"], (c["rows"],), generator=g, device=DEV)
    t[torch.rand(c["rows"], generator=g, device=DEV) < 0.02] = -100        # padding
    t[0] = 1
    return {"x": _randn(g, (c["rows"], c["vocab"]), 2.0, DT[c["dtype"]]).requires_grad_(), "t": t}


def _prepare_flash(c, seed):
    g, shape = _gen(seed), (c["batch"], c["seq"], c["heads"], c["hd"])
    q, k, v, do = (_randn(g, shape, 1.0, torch.bfloat16) for _ in range(4))
    return {"q": q.requires_grad_(), "k": k.requires_grad_(), "v": v.requires_grad_(), "do": do, "causal": c["causal"]}


def _prepare_model(c, seed):
    g = _gen(seed)
    return {"model": _decoder(c, g, DT[c["dtype"]]), "x": torch.randint(0, c["ntok"], (c["batch"], 4), generator=g, device=DEV),
            "y": torch.randint(0, c["ntok"], (c["batch"],), generator=g, device=DEV)}


def prepare(case, seed):
    s = {"v2": _prepare_v2, "element": _prepare_element, "muon": _prepare_muon, "bilevel": _prepare_bilevel, "norm": _prepare_norm, "attn": _prepare_attn,
         "ce": _prepare_ce, "flash": _prepare_flash, "model": _prepare_model}[case["kind"]](case, seed)
    s["kind"] = case["kind"]
    return s


# ---------------------------------------------------------------------------------------------------- one pass

def _flat(ts):
    return torch.cat([t.detach().reshape(-1) for t in ts])


class _Later(dict):
    """Outputs of an optimizer step: the state's own buffers, put together per kind of state when they are looked at.  A training
    loop does not gather them, so this stays out of the pass."""

    def __init__(self, groups):
        super().__init__({k: None for k in groups})
        self.groups = groups

    def __getitem__(self, k):
        return _flat(self.groups[k])

    def items(self):
        return [(k, self[k]) for k in self.groups]

    def values(self):
        return [self[k] for k in self.groups]


def _states(opt, ps, names):
    out = {"p": ps}
    for n in names:
        out[n] = [opt.state[p][n] for p in ps]
    return _Later(out)


def run(s):
    from supergrok15_b200.ops import nn_ops
    kind = s["kind"]
    if kind == "v2":
        s["opt"].step(train_acc=0.5)
        return _states(s["opt"], s["ps"], ("exp_avg", "exp_avg_sq", "mu", "gru_state", "mamba_fwd_state", "mamba_bwd_state"))
    if kind == "element":
        opt = s["opt"]
        if hasattr(opt, "meta_net"):
            opt.step(train_acc=0.5)
            return _states(opt, s["ps"], ("exp_avg", "exp_avg_sq", "mu"))
        opt.step()
        return _states(opt, s["ps"], [k for k in opt.state[s["ps"][0]] if k != "step"])
    if kind == "muon":
        s["opt"].step()
        return _states(s["opt"], s["ps"], ("momentum_buffer",))
    if kind == "bilevel":
        loss = s["opt"].bilevel_step(s["model"], s["x"][0], s["y"][0], s["x"][1], s["y"][1], F.cross_entropy, s["meta"])
        return {"loss": loss, "grads": {k: p.grad for k, p in s["opt"].meta_net.named_parameters()}}
    if kind == "norm":
        if s["rms"]:
            y, z = nn_ops.norm_residual(s["x"], s["r"], s["w"], None, 1e-5, rms=True)
            return [y, z, *torch.autograd.grad((y, z), (s["x"], s["r"], s["w"]), (s["dy"], s["dz"]))]
        y = nn_ops.layer_norm(s["x"], s["r"], s["w"], s["b"])
        return [y, *torch.autograd.grad(y, (s["x"], s["r"], s["w"], s["b"]), s["dy"])]
    if kind == "attn":
        o = nn_ops.attention_small(s["qkv"], s["heads"])
        return [o, torch.autograd.grad(o, s["qkv"], s["do"])[0]]
    if kind == "ce":
        loss = nn_ops.cross_entropy(s["x"], s["t"])
        return [loss, torch.autograd.grad(loss, s["x"])[0]]
    if kind == "flash":
        o = nn_ops.attention(s["q"], s["k"], s["v"], s["causal"], impl="tcgen05")
        return [o, *torch.autograd.grad(o, (s["q"], s["k"], s["v"]), s["do"])]
    m = s["model"]
    m.zero_grad(set_to_none=True)
    logits = m(s["x"])
    loss = nn_ops.cross_entropy(logits, s["y"])
    loss.backward()
    return {"logits": logits, "loss": loss, "grads": _Later({"all": [p.grad for p in m.parameters()]})}


# ---------------------------------------------------------------------------------------------------- what a pass cannot do without

def _numel(shapes):
    return sum(math.prod(x) for x in shapes)


def work(case):
    kind = case["kind"]
    if kind in ("v2", "element"):
        n = _numel(_decoder_shapes(case))
        e = 4 if case["dtype"] == "f32" else 2
        if kind == "v2":      # p, m, v, mu, four GRU states read and written; gradient and sharpness read; scan ~2 x 16 x 8 pairs of ~26, GRU / routing / experts ~2.4 k
            return {"bytes": n * (3 * e + 4 * (2 * 7 + 1)), "flops": n * (2 * 16 * 8 * 26 + 2 * 16 * 40 + 2400)}
        states = {"adamw": 2, "grokadamw": 3, "supergrok15": 3}[case["opt"]]
        clip = 0 if case["opt"] == "adamw" else e          # the clipped gradient goes back to where it came from
        return {"bytes": n * (3 * e + clip + 8 * states + (4 if case["opt"] == "supergrok15" else 0)), "flops": n * (400 if case["opt"] == "supergrok15" else 25)}
    if kind == "muon":
        sh = _muon_shapes(case)
        return {"bytes": _numel(sh) * 4 * 5, "flops": sum(5 * (4.0 * a * b * min(a, b) + 2.0 * min(a, b) ** 3) for a, b in sh)}
    if kind == "bilevel":
        n = _numel(_decoder_shapes(case))
        return {"bytes": n * 4 * 12, "flops": n * 3 * (2 * 16 * 8 * 26 + 2 * 16 * 40 + 4 * 1700) + 8.0 * case["batch"] * 4 * n}
    e = 4 if case.get("dtype") == "f32" else 2
    if kind == "norm":       # x, r in, y out (and z for the residual stream); z and dy (and its own gradient) in, one gradient out
        n = case["rows"] * case["d"]
        return {"bytes": n * e * 8, "flops": n * 25}
    if kind == "attn":
        n = case["batch"] * case["seq"] * case["heads"] * case["hd"]
        return {"bytes": n * e * (3 + 1 + 3 + 1 + 3), "flops": n * case["seq"] * 14}
    if kind == "ce":
        return {"bytes": case["rows"] * case["vocab"] * e * 3, "flops": case["rows"] * case["vocab"] * 10}
    if kind == "flash":
        n = case["batch"] * case["seq"] * case["heads"] * case["hd"]
        return {"bytes": n * 2 * 12, "flops": 14.0 * n * case["seq"] * (0.5 if case["causal"] else 1.0)}
    n, t = _numel(_decoder_shapes(case)), case["batch"] * 4
    act = case["layers"] * t * case["d"] * 40              # activations of a block written once and read once
    return {"bytes": e * (4 * n + act), "flops": 6.0 * t * (n - 2 * case["ntok"] * case["d"])}


# ---------------------------------------------------------------------------------------------------- how far another correct implementation may be

def tolerance(case):
    kind = case["kind"]
    if kind == "v2":       # 32-bit sums over scans of many steps; a near tie in the routing may pick another expert for single elements
        return {"rel": 2e-4, "max": 0.5} if case["dtype"] == "f32" else {"rel": 5e-3, "max": 0.5}
    if kind == "element":
        return {"rel": 1e-5, "max": 1e-3} if case["dtype"] == "f32" else {"rel": 5e-3, "max": 0.2}
    if kind == "muon":     # the update is iterated in bf16; parameters move by 0.4 % of the orthogonal factor
        return {"rel": 1e-4, "max": 5e-3}
    if kind == "bilevel":  # sums over all elements of terms of either sign, behind a top-4 selection
        return {"rel": 3e-3, "max": 0.1}
    if kind in ("norm", "attn", "ce"):
        return {"rel": 1e-5, "max": 1e-3} if case["dtype"] == "f32" else {"rel": 5e-3, "max": 0.1}
    if kind == "flash":
        return {"rel": 1e-2, "max": 0.3}
    return {"rel": 1e-4, "max": 0.02} if case["dtype"] == "f32" else {"rel": 2e-2, "max": 0.9}


# ---------------------------------------------------------------------------------------------------- the same in 64 bits

def _adam64(p, grad, m, v, lr, b1, b2, eps, wd, step):
    m = b1 * m + (1 - b1) * grad
    v = b2 * v + (1 - b2) * grad * grad
    p = p * (1 - lr * wd) - lr / (1 - b1 ** step) * m / ((v / (1 - b2 ** step)).sqrt() + eps)
    return p, m, v


def _scan64(x, W, pre, h0):
    """Selective scan of one direction: x [n, 8] -> contexts [n, 8] and the last state.  The 2 x 2 affine maps of all steps are
    combined by doubling (inclusive prefixes), so the depth is log2 n."""
    n = x.shape[0]
    xz = x @ W[pre + "in_proj.weight"].T
    xb, z = xz[:, :16], xz[:, 16:]
    dt = F.softplus(xb @ W[pre + "dt_proj.weight"].T + W[pre + "dt_proj.bias"])
    B, C = xb @ W[pre + "B_proj.weight"].T, xb @ W[pre + "C_proj.weight"].T
    a = dt.unsqueeze(-1) * -torch.exp(W[pre + "A_log"]) / 2
    abar = (1 + a) / (1 - a + 1e-8)
    ang = dt.unsqueeze(-1) * W[pre + "rope_freq"]
    cs, sn = ang.cos(), ang.sin()
    ae, ao = abar[..., 0::2], abar[..., 1::2]
    bx = (dt * xb).unsqueeze(-1) * B.unsqueeze(1)
    m = [ae * cs, -ae * sn, ao * sn, ao * cs]
    b = [bx[..., 0::2], bx[..., 1::2]]
    he, ho = h0[:, 0::2], h0[:, 1::2]
    b = [torch.cat([b[0][:1] + m[0][:1] * he + m[1][:1] * ho, b[0][1:]]), torch.cat([b[1][:1] + m[2][:1] * he + m[3][:1] * ho, b[1][1:]])]
    step = 1
    while step < n:
        hi, lo = slice(step, None), slice(None, n - step)
        nb = [m[0][hi] * b[0][lo] + m[1][hi] * b[1][lo] + b[0][hi], m[2][hi] * b[0][lo] + m[3][hi] * b[1][lo] + b[1][hi]]
        nm = [m[0][hi] * m[0][lo] + m[1][hi] * m[2][lo], m[0][hi] * m[1][lo] + m[1][hi] * m[3][lo],
              m[2][hi] * m[0][lo] + m[3][hi] * m[2][lo], m[2][hi] * m[1][lo] + m[3][hi] * m[3][lo]]
        b = [torch.cat([b[i][:step], nb[i]]) for i in range(2)]
        m = [torch.cat([m[i][:step], nm[i]]) for i in range(4)]
        step *= 2
    y = (b[0] * C[:, None, 0::2]).sum(-1) + (b[1] * C[:, None, 1::2]).sum(-1)
    y = y * F.silu(z) + W[pre + "D"] * xb
    last = torch.stack([b[0][-1], b[1][-1]], -1).reshape(16, 16)
    return y @ W[pre + "out_proj.weight"].T, last


def _meta64(W, g, s, gru, hf, hb, soft):
    """The meta-network on one tensor: (rewritten gradient, GRU states, scan states); ``soft``: top-4 routing instead of top-1."""
    order = torch.argsort(g.float().abs(), stable=True)
    x = torch.stack([g, s], -1)[order] @ W["input_proj.weight"].T + W["input_proj.bias"]
    cf, hf = _scan64(x, W, "mamba_fwd.", hf)
    cb, hb = _scan64(x.flip(0), W, "mamba_bwd.", hb)
    back = torch.argsort(order)
    cf, cb = cf[back], cb.flip(0)[back]
    gs = torch.stack([g, s], -1)
    xin = torch.cat([gs, cf, cb], -1)
    xh = torch.cat([xin, gru], -1)
    z = torch.sigmoid(xh @ W["gru.W_z.weight"].T + W["gru.W_z.bias"])
    r = torch.sigmoid(xh @ W["gru.W_r.weight"].T + W["gru.W_r.bias"])
    gru = (1 - z) * gru + z * torch.tanh(torch.cat([xin, r * gru], -1) @ W["gru.W_h.weight"].T + W["gru.W_h.bias"])
    pin = torch.cat([gru, cf, cb, gs], -1)
    W1, b1, W2, b2 = W["expert_W1"].squeeze(-1), W["expert_b1"], W["expert_W2"].squeeze(1), W["expert_b2"].squeeze(-1)
    out = (torch.relu(g.view(-1, 1, 1) * W1 + b1) * W2).sum(-1) + b2 if g.numel() <= 1 << 17 else None     # [n, experts]
    total = torch.zeros_like(g)
    for h in range(4):
        q = pin @ W["peer_queries.%d.weight" % h].T
        sa, sb = q[:, :4] @ W["product_keys_A.%d" % h].T, q[:, 4:] @ W["product_keys_B.%d" % h].T
        k = 4 if soft else 1
        (ta, ia), (tb, ib) = sa.topk(k), sb.topk(k)
        wa, wb = torch.softmax(10 * ta, -1), torch.softmax(10 * tb, -1)
        e = (ia.unsqueeze(2) * 12 + ib.unsqueeze(1)).reshape(g.numel(), -1)
        w = (wa.unsqueeze(2) * wb.unsqueeze(1)).reshape(g.numel(), -1)
        o = out.gather(1, e) if out is not None else (torch.relu(g.view(-1, 1, 1) * W1[e] + b1[e]) * W2[e]).sum(-1) + b2[e]
        total = total + (w * o).sum(-1)
    return g + 0.1 * total / 4, gru, hf, hb


def _exact_v2(c, seed):
    if _numel(_decoder_shapes(c)) > 4_000_000:
        return None                                  # minutes in 64 bits
    s = _prepare_v2(c, seed)
    opt, ps = s["opt"], s["ps"]
    W = {k: v.double() for k, v in opt.meta_net.state_dict().items() if v.is_floating_point()}
    acc = 0.5
    lamb = 2.0 * 0.5 / (1 + math.exp(-20 * (acc - 0.8)))                      # the ramp is half way at step 150
    wd = 1.0 * (1 + 4.0 / (1 + math.exp(-20 * (acc - 0.9))))
    names = ("p", "exp_avg", "exp_avg_sq", "mu", "gru_state", "mamba_fwd_state", "mamba_bwd_state")
    out = {k: [] for k in names}
    for i, p in enumerate(ps):
        st = {k: opt.state[p][k].double() for k in ("sharpness",) + names[1:]}
        g = p.grad.double().reshape(-1)
        norm = g.norm()
        g = g * (1.0 / (norm + 1e-12)) if norm > 1.0 else g
        smart, gru, hf, hb = _meta64(W, g, st["sharpness"], st["gru_state"], st["mamba_fwd_state"], st["mamba_bwd_state"], False)
        mu = 0.97 * st["mu"] + 0.03 * g
        new, m, v = _adam64(p.detach().double().reshape(-1), smart + lamb * mu, st["exp_avg"], st["exp_avg_sq"], 1e-3, 0.9 * 0.9 ** i, 0.999, 1e-8, wd, 150)
        for k, t in zip(names, (new, m, v, mu, gru, hf, hb)):
            out[k].append(t)
    return {k: _flat(v) for k, v in out.items()}


def _exact_element(c, seed):
    s = _prepare_element(c, seed)
    opt, ps = s["opt"], s["ps"]
    gs = [p.grad.double().reshape(-1) for p in ps]
    out = {}

    def put(k, t):
        out.setdefault(k, []).append(t)
    if c["opt"] != "adamw":
        norm = torch.sqrt(sum(g.square().sum() for g in gs))
        if norm > 1.0:
            gs = [g * (1.0 / (norm + 1e-6)) for g in gs]
    for i, p in enumerate(ps):
        st = {k: v.double().reshape(-1) for k, v in opt.state[p].items() if torch.is_tensor(v)}
        x, g = p.detach().double().reshape(-1), gs[i]
        if c["opt"] == "adamw":
            new = _adam64(x, g, st["exp_avg"], st["exp_avg_sq"], 1e-3, 0.9, 0.999, 1e-8, 1e-2, 150)
        elif c["opt"] == "grokadamw":
            e = 0.98 * st["ema"] + 0.02 * g
            put("ema", e)
            new = _adam64(x, g + 5.0 * e, st["exp_avg"], st["exp_avg_sq"], 1e-3, 0.9, 0.98, 1e-8, 1.0, 150)
        else:
            net = {k: v.double() for k, v in opt.meta_net.state_dict().items()}
            acc = 0.5
            lamb = 2.0 * 0.5 / (1 + math.exp(-20 * (acc - 0.8)))
            wd = 1.0 * (1 + 4.0 / (1 + math.exp(-20 * (acc - 0.9))))
            mu = 0.97 * st["mu"] + 0.03 * g
            put("mu", mu)
            mlp = []
            for a in range(0, g.numel(), 1 << 20):
                h = torch.stack([g[a:a + (1 << 20)], st["sharpness"][a:a + (1 << 20)]], -1) @ net["net.0.weight"].T + net["net.0.bias"]
                mlp.append((F.gelu(h) @ net["net.2.weight"].T + net["net.2.bias"])[:, 0])
            smart = g + net["rescale"] * torch.cat(mlp)
            new = _adam64(x, smart + lamb * mu, st["exp_avg"], st["exp_avg_sq"], 1e-3, 0.9 * 0.9 ** i, 0.999, 1e-8, wd, 150)
        for k, t in zip(("p", "exp_avg", "exp_avg_sq"), new):
            put(k, t)
    return {k: _flat(v) for k, v in out.items()}


def _exact_muon(c, seed):
    s = _prepare_muon(c, seed)
    a, b, k = 3.4445, -4.7750, 2.0315
    ps, bufs = [], []
    for p in s["ps"]:
        buf = 0.95 * s["opt"].state[p]["momentum_buffer"].double() + p.grad.double()
        X = buf / (buf.norm() + 1e-7)
        tall = X.shape[0] > X.shape[1]
        X = X.T if tall else X
        for _ in range(5):
            A = X @ X.T
            X = a * X + (b * A + k * A @ A) @ X
        ps.append((p.detach().double() - 0.2 * 0.02 * (X.T if tall else X)) * (1 - 0.02))
        bufs.append(buf)
    return {"p": _flat(ps), "momentum_buffer": _flat(bufs)}


def _decoder64(P, x, heads, layers):
    """Logits of the post-LN decoder for its parameters ``P`` (name -> tensor)."""
    h = P["tok.weight"][x] + P["pos.weight"][: x.shape[1]]
    b, t, d = h.shape

    def ln(z, n):
        return F.layer_norm(z, (d,), P[n + ".weight"], P[n + ".bias"])
    mask = torch.full((t, t), float("-inf"), device=h.device, dtype=h.dtype).triu(1)
    for i in range(layers):
        n = "layers.%d." % i
        qkv = (h @ P[n + "attn.in_proj_weight"].T + P[n + "attn.in_proj_bias"]).view(b, t, 3, heads, d // heads)
        q, k, v = (qkv[:, :, j].transpose(1, 2) for j in range(3))
        o = torch.softmax(q @ k.transpose(-1, -2) * (d // heads) ** -0.5 + mask, -1) @ v
        o = o.transpose(1, 2).reshape(b, t, d) @ P[n + "attn.out_proj.weight"].T + P[n + "attn.out_proj.bias"]
        h = ln(h + o, n + "n1")
        u = F.gelu(h @ P[n + "ff.0.weight"].T + P[n + "ff.0.bias"])
        h = ln(h + u @ P[n + "ff.2.weight"].T + P[n + "ff.2.bias"], n + "n2")
    return ln(h[:, -1], "norm") @ P["out.weight"].T + P["out.bias"]


def _exact_model(c, seed):
    s = _prepare_model(c, seed)
    P = {k: v.detach().double().requires_grad_() for k, v in s["model"].named_parameters()}
    logits = _decoder64(P, s["x"], c["heads"], c["layers"])
    loss = F.cross_entropy(logits, s["y"])
    return {"logits": logits.detach(), "loss": loss.detach(), "grads": {"all": _flat(torch.autograd.grad(loss, list(P.values())))}}


def _exact_bilevel(c, seed):
    s = _prepare_bilevel(c, seed)
    opt, names = s["opt"], [n for n, _ in s["model"].named_parameters()]
    P = {k: v.detach().double().requires_grad_() for k, v in s["model"].named_parameters()}
    loss = F.cross_entropy(_decoder64(P, s["x"][1], 4, c["layers"]), s["y"][1])
    vgs = torch.autograd.grad(loss, list(P.values()))
    W = {k: v.detach().double().requires_grad_() for k, v in opt.meta_net.named_parameters()}
    for n, p, vg in zip(names, s["model"].parameters(), vgs):
        st = {k: opt.state[p][k].double() for k in ("sharpness", "gru_state", "mamba_fwd_state", "mamba_bwd_state")}
        smart = _meta64(W, p.grad.double().reshape(-1), st["sharpness"], st["gru_state"], st["mamba_fwd_state"], st["mamba_bwd_state"], True)[0]
        (-(smart * vg.reshape(-1) / vg.norm()).sum()).backward()
    return {"loss": float(loss), "grads": {k: v.grad for k, v in W.items()}}


def _exact_layer(c, s):
    kind = c["kind"]
    if kind == "norm":
        x, r, w = (s[k].detach().double().requires_grad_() for k in ("x", "r", "w"))
        z = x + r
        if c["rms"]:
            y = z * torch.rsqrt(z.square().mean(-1, keepdim=True) + 1e-5) * w
            return [y.detach(), z.detach(), *torch.autograd.grad((y, z), (x, r, w), (s["dy"].double(), s["dz"].double()))]
        b = s["b"].detach().double().requires_grad_()
        y = F.layer_norm(z, (c["d"],), w, b, 1e-5)
        return [y.detach(), *torch.autograd.grad(y, (x, r, w, b), s["dy"].double())]
    if kind == "attn":
        qkv = s["qkv"].detach().double().requires_grad_()
        B, S, H = c["batch"], c["seq"], c["heads"]
        q, k, v = (t.transpose(1, 2) for t in qkv.view(B, S, 3, H, c["hd"]).unbind(2))
        mask = torch.full((S, S), float("-inf"), device=DEV, dtype=torch.float64).triu(1)
        o = (torch.softmax(q @ k.transpose(-1, -2) * c["hd"] ** -0.5 + mask, -1) @ v).transpose(1, 2).reshape(B, S, H * c["hd"])
        return [o.detach(), torch.autograd.grad(o, qkv, s["do"].double())[0]]
    if kind == "ce":
        x = s["x"].detach().double().requires_grad_()
        loss = F.cross_entropy(x, s["t"])
        return [loss.detach(), torch.autograd.grad(loss, x)[0]]
    outs = [[], [], [], []]
    for b in range(c["batch"]):                       # one sequence at a time: the scores are [heads, seq, seq] in 64 bits
        q, k, v = (s[n][b].detach().double().transpose(0, 1).requires_grad_() for n in ("q", "k", "v"))
        sc = q @ k.transpose(-1, -2) * c["hd"] ** -0.5
        if c["causal"]:
            sc = sc + torch.full((c["seq"], c["seq"]), float("-inf"), device=DEV, dtype=torch.float64).triu(1)
        o = torch.softmax(sc, -1) @ v
        for t, got in zip(outs, [o.detach(), *torch.autograd.grad(o, (q, k, v), s["do"][b].double().transpose(0, 1))]):
            t.append(got.transpose(0, 1))
    return [torch.stack(t) for t in outs]


def exact(case, seed):
    whole = {"v2": _exact_v2, "element": _exact_element, "muon": _exact_muon, "bilevel": _exact_bilevel, "model": _exact_model}.get(case["kind"])
    return whole(case, seed) if whole else _exact_layer(case, prepare(case, seed))
