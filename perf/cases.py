"""Performance cases: the layers, the objective and the whole model, as training and packed prefill call them.

Widths are those of the presets q38_c1 .. q38_c4 (their training sequence is 4096 tokens, micro batch 2 or 4); token counts run from
one 64-token block to 32768.  A training case is forward and backward with the fp32 gradient buffers that a training
program keeps; the others run under ``no_grad``.

    gdn     Gated DeltaNet layer (three of four token mixers, and the next-token head's)
    qsa     gated attention with the indexer: dense in the warm-up phase, block-sparse afterwards, with the indexer's KL in training
    moe     routed experts with the shared expert
    mhc     the residual-stream pair around a sub-layer
    head    fused vocabulary projection and cross-entropy
    model   whole model, prefill to logits
"""
import math

import torch
import torch.nn.functional as F
import torch.utils.checkpoint

from q38 import ops
from q38.losses import linear_cross_entropy
from q38.models import modeling
from q38.presets import load_preset, model_config

VOCAB, EOS, BLOCK, EXPERTS, TOPK = 10112, 53, 64, 64, 5
WIDTHS = dict(
    q38_c1=dict(hidden=448, heads=16, kv_heads=2, k_heads=6, v_heads=18, ffn=112),
    q38_c2=dict(hidden=576, heads=22, kv_heads=2, k_heads=7, v_heads=21, ffn=144),
    q38_c3=dict(hidden=768, heads=28, kv_heads=2, k_heads=10, v_heads=30, ffn=192),
    q38_c4=dict(hidden=1024, heads=38, kv_heads=2, k_heads=13, v_heads=39, ffn=256))
PARAMS = dict(q38_c1=(9, 49152))          # layers, rows per n-gram table (whole-model cases)


def _case(name, kind, preset, batch, seq, train, dense=False):
    case = dict(kind=kind, preset=preset, batch=batch, seq=seq, train=train, dense=dense, **WIDTHS[preset])
    return case if name is None else dict(name=name, **case)


def listed():
    return [
        # a short prompt: four blocks, latency of the layer's dozen launches
        _case("gdn_infer_short", "gdn", "q38_c1", 1, 256, False),
        # the micro batch of the flagship preset
        _case("gdn_train", "gdn", "q38_c2", 4, 4096, True),
        # one long prompt in a wide model: few sequences, long chain of chunks
        _case("gdn_infer_long", "gdn", "q38_c4", 1, 8192, False),
        # ragged micro batch: an odd number of blocks and sequences
        _case("gdn_train_odd", "gdn", "q38_c3", 3, 2112, True),
        # attention after the warm-up phase, with the indexer's distillation term
        _case("qsa_train_sparse", "qsa", "q38_c2", 4, 4096, True),
        # attention in the warm-up phase
        _case("qsa_train_dense", "qsa", "q38_c1", 2, 4096, True, dense=True),
        # prefill of a long prompt: block selection from the first query of each block
        _case("qsa_infer_long", "qsa", "q38_c3", 1, 8192, False),
        # experts of the flagship micro batch
        _case("moe_train", "moe", "q38_c2", 4, 4096, True),
        # residual streams of the flagship micro batch (the largest activations of the model)
        _case("mhc_train", "mhc", "q38_c2", 4, 4096, True),
        # vocabulary projection and loss of the flagship micro batch
        _case("head_train", "head", "q38_c2", 4, 4096, True),
        # packed prefill of the small preset to logits
        _case("model_prefill", "model", "q38_c1", 4, 4096, False),
    ]


def draw(rng):
    kind = rng.choice(["gdn", "gdn", "gdn", "qsa", "qsa", "moe", "mhc", "head", "model"])
    log_int = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    train = rng.random() < 0.6
    if kind == "model":
        preset, train = "q38_c1", False
        batch, seq = rng.choice([1, 2, 3]), log_int(65, 4096)          # the model pads a ragged prompt to whole blocks itself
    else:
        preset = rng.choice(sorted(WIDTHS))
        top = 8192 if preset == "q38_c4" else 16384
        tokens = log_int(BLOCK, top)
        if kind in ("gdn", "qsa"):
            batch = rng.choice([b for b in (1, 2, 3, 4) if b * BLOCK <= tokens])
            seq = min(8192 if not train else 4096, max(1, tokens // batch // BLOCK) * BLOCK)
        else:
            batch, seq = 1, tokens
    return _case(None, kind, preset, batch, seq, train, dense=kind == "qsa" and train and rng.random() < 0.4)


# ---- inputs -----------------------------------------------------------------------------------------------------------------
def _shapes(c):
    """Parameter shapes of a layer, by the names the module gives them."""
    h, kd, vd, H = c["hidden"], 64 * c["k_heads"], 64 * c["v_heads"], c["v_heads"]
    if c["kind"] == "gdn":
        conv = 2 * kd + vd
        return {"dt_bias": (H,), "A_log": (H,), "conv1d.weight": (conv, 1, 4), "norm.weight": (64,), "out_proj.weight": (h, vd),
                "in_proj_qkv.weight": (conv, h), "in_proj_z.weight": (vd, h), "in_proj_b.weight": (H, h), "in_proj_a.weight": (H, h)}
    if c["kind"] == "qsa":
        nq, nkv = c["heads"] * 64, c["kv_heads"] * 64
        return {"attn.q_proj.weight": (2 * nq, h), "attn.k_proj.weight": (nkv, h), "attn.v_proj.weight": (nkv, h), "attn.o_proj.weight": (h, nq),
                "attn.q_norm.weight": (64,), "attn.k_norm.weight": (64,),
                "indexer.wq.weight": (256, h), "indexer.wk.weight": (64, h), "indexer.ww.weight": (4, h)}
    if c["kind"] == "moe":
        f = c["ffn"]
        return {"gate.weight": (EXPERTS, h), "experts.gate_up_proj": (EXPERTS, 2 * f, h), "experts.down_proj": (EXPERTS, h, f),
                "shared_expert.gate_proj.weight": (f, h), "shared_expert.up_proj.weight": (f, h), "shared_expert.down_proj.weight": (h, f),
                "shared_expert_gate.weight": (1, h)}
    if c["kind"] == "mhc":
        r = max(1, round(h / 8))
        return {"mhc.A.weight": (r, 4 * h), "mhc.B.weight": (24, r), "mhc.b_pre": (4,), "mhc.b_post": (4,), "mhc.b_res": (4, 4),
                "mhc.alphas": (3,), "norm.weight": (h,)}
    return {"weight": (VOCAB, h)}


def _tensors(c, seed):
    """Weights, activations and upstream gradients of a layer case, from the seed alone."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    randn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    rand = lambda *s: torch.rand(*s, device="cuda", generator=gen)
    w = {}
    for name, shape in _shapes(c).items():
        if name == "dt_bias":
            w[name] = rand(*shape) * 7 - 6                               # heads that remember for a long time and heads that forget
        elif name == "A_log":
            w[name] = (rand(*shape) * 15.99 + 0.01).log()
        elif name == "conv1d.weight":
            w[name] = rand(*shape) - 0.5
        elif name == "mhc.b_res":
            w[name] = 8 * torch.eye(4, device="cuda") - 8 + randn(*shape)
        elif name == "mhc.alphas":
            w[name] = 0.1 + 0.05 * rand(*shape)
        elif c["kind"] == "gdn" and name == "norm.weight":
            w[name] = 1 + 0.1 * randn(*shape)
        elif name.startswith("mhc.b_"):
            w[name] = randn(*shape)
        elif len(shape) == 1:
            w[name] = 0.1 * randn(*shape)
        else:
            w[name] = 0.02 * randn(*shape)
    B, S, h = c["batch"], c["seq"], c["hidden"]
    out = dict(weights=w)
    if c["kind"] == "mhc":
        out["x"] = randn(B, S, 4, h)
        out["dy"] = randn(B, S, 4, h) * 1e-3
    elif c["kind"] == "head":
        out["x"] = randn(B * S, h).to(torch.bfloat16)
        out["target"] = torch.randint(0, VOCAB, (B * S,), device="cuda", generator=gen)
    else:
        out["x"] = randn(B, S, h).to(torch.bfloat16)
        out["dy"] = (randn(B, S, h) * 1e-2).to(torch.bfloat16)
    return out


class _Pair(torch.nn.Module):
    """Two modules that one call uses together."""

    def __init__(self, **parts):
        super().__init__()
        for name, part in parts.items():
            setattr(self, name, part)


def _config(c, layers=4):
    shape = dict(layers=layers, hidden=c["hidden"], heads=c["heads"], kv_heads=c["kv_heads"], lin_k_heads=c["k_heads"], lin_v_heads=c["v_heads"],
                 experts=EXPERTS, topk=TOPK, moe_ffn=c["ffn"], shared_ffn=c["ffn"], ngram_rows=1024)
    return model_config(shape, VOCAB, c["seq"], bos_token_id=1, eos_token_id=EOS, pad_token_id=0)


def _module(c):
    cfg = _config(c)
    if c["kind"] == "gdn":
        return modeling.Qwen3_8MoeGatedDeltaNet(cfg, 0)
    if c["kind"] == "qsa":
        return _Pair(attn=modeling.Qwen3_8MoeAttention(cfg, 3), indexer=modeling.Indexer(c["hidden"], cfg.indexer_heads, cfg.indexer_head_dim))
    if c["kind"] == "moe":
        return modeling.Qwen3_8MoeSparseMoeBlock(cfg)
    if c["kind"] == "mhc":
        return _Pair(mhc=modeling.MHC(c["hidden"]), norm=modeling.Qwen3_8MoeRMSNorm(c["hidden"]))
    return torch.nn.Linear(c["hidden"], VOCAB, bias=False)


def _flat_grads(module):
    """One zeroed fp32 buffer with every parameter's gradient as a view (256-byte aligned), as a training program keeps it."""
    sizes = [(p, (p.numel() + 63) // 64 * 64) for p in module.parameters()]
    flat = torch.zeros(sum(n for _, n in sizes), device="cuda")
    at = 0
    for p, n in sizes:
        p.grad = flat[at:at + p.numel()].view_as(p)
        at += n
    return flat


def prepare(case, seed):
    ops.install()
    c = case
    if c["kind"] == "model":
        torch.manual_seed(seed)
        cfg = model_config(load_preset(c["preset"])["model"], VOCAB, max(4096, c["seq"]), bos_token_id=1, eos_token_id=EOS, pad_token_id=0)
        with torch.device("cuda"):
            model = modeling.Q38ForCausalLM(cfg)
        model.model.compute_dtype = torch.bfloat16
        model.eval()
        gen = torch.Generator(device="cuda").manual_seed(seed)
        ids = torch.randint(1, VOCAB, (c["batch"], c["seq"]), device="cuda", generator=gen)
        ids[torch.rand(ids.shape, device="cuda", generator=gen) < 1 / 1024] = EOS
        return dict(case=c, module=model, x=ids)
    t = _tensors(c, seed)
    with torch.device("cuda"):
        module = _module(c)
    module.load_state_dict(t["weights"])
    state = dict(case=c, module=module, x=t["x"], dy=t.get("dy"), target=t.get("target"))
    if c["kind"] == "qsa":
        state["rope"] = modeling.rope_tables(torch.arange(c["seq"], device="cuda")[None], 16, 1e7, torch.float32)
    if c["train"]:
        state["flat"] = _flat_grads(module)
    else:
        module.requires_grad_(False)
    return state


def _forward(state, x):
    c, m = state["case"], state["module"]
    if c["kind"] == "qsa":
        return modeling.qsa_attention(m.attn, x, *state["rope"], m.indexer, 8, c["dense"], c["train"])
    if c["kind"] == "mhc":
        backend = modeling.get_backend()
        xin, link = backend.mhc_pre_norm(m.mhc, m.norm, x, torch.bfloat16)
        return backend.mhc_post(m.mhc, xin, link), None
    if c["kind"] == "head":
        return linear_cross_entropy(m.weight, x, state["target"]), None
    return m(x), None


def run(state):
    c = state["case"]
    if not c["train"]:
        with torch.no_grad():
            if c["kind"] == "model":
                return {"logits": state["module"](state["x"]).logits}
            y, kl = _forward(state, state["x"])
            return {"y": y}
    state["flat"].zero_()
    x = state["x"].detach().requires_grad_()
    y, kl = _forward(state, x)
    if c["kind"] == "head":
        y.backward()
    elif kl is not None:
        torch.autograd.backward([y, kl], [state["dy"], torch.ones_like(kl)])
    else:
        y.backward(state["dy"])
    out = {"y": y.detach(), "dx": x.grad}
    if kl is not None:
        out["kl"] = kl.detach()
    out.update({"d " + name: p.grad for name, p in state["module"].named_parameters()})
    return out


# ---- what a pass cannot do without -------------------------------------------------------------------------------------------------
def work(case):
    c = case
    T, S, h, f = c["batch"] * c["seq"], c["seq"], c["hidden"], c["ffn"]
    if c["kind"] == "model":
        layers, rows = PARAMS[c["preset"]]
        kinds = [i % 4 == 3 for i in range(layers)]
        flops = sum(_forward_flops({**c, "kind": "qsa" if q else "gdn"}) + _forward_flops({**c, "kind": "moe"}) + 2 * _forward_flops({**c, "kind": "mhc"})
                    for q in kinds) + _forward_flops({**c, "kind": "head"})
        params = sum(_params({**c, "kind": "qsa" if q else "gdn"}) + _params({**c, "kind": "moe"}) + 2 * _params({**c, "kind": "mhc"}) for q in kinds)
        params += VOCAB * h + 2 * rows * h
        return {"bytes": 4 * params + 2 * T * VOCAB, "flops": flops}
    flops, params = _forward_flops(c), _params(c)
    row = 16 * h if c["kind"] == "mhc" else 2 * h
    if c["kind"] == "head":
        passes = 3 if c["train"] else 1
        return {"bytes": T * ((2 if c["train"] else 1) * row + 8) + (8 if c["train"] else 4) * params, "flops": passes * flops}
    if c["train"]:
        return {"bytes": 4 * T * row + 8 * params, "flops": 3 * flops}
    return {"bytes": 2 * T * row + 4 * params, "flops": flops}


def _params(c):
    return sum(math.prod(s) for s in _shapes(c).values())


def _forward_flops(c):
    T, S, h = c["batch"] * c["seq"], c["seq"], c["hidden"]
    if c["kind"] == "moe":
        return 2 * T * (EXPERTS * h + (TOPK + 1) * 3 * h * c["ffn"])
    dense = 2 * T * (_params(c))
    if c["kind"] == "gdn":
        return dense + T * c["v_heads"] * 8 * 64 * 64                    # read, correct and write a 64 x 64 state per token and head
    if c["kind"] == "qsa":
        keys = (S / 2 if c["dense"] else min(S / 2, 8 * BLOCK))
        pairs = 4 * 64 * c["heads"] * keys
        if c["train"]:
            pairs += 2 * 64 * (c["heads"] + 4) * S / 2 / 3                  # block masses and indexer scores
        else:
            pairs += 2 * 64 * 4 * S / 2 / BLOCK
        return dense + T * pairs
    return dense


# ---- tolerances ----------------------------------------------------------------------------------------------------------------
def tolerance(case):
    """bf16 activations and tensor-core operands throughout (one rounding is 2e-3).  Against 64 bits the gdn outputs are 1e-2 off, the qsa
    outputs 7e-3 with 4e-2 in the indexer's tiny gradients, mhc 3e-3, head 2.5e-3, moe 5e-3 with 8e-2 where a token's fifth expert changes."""
    return {"rel": {"gdn": 0.03, "qsa": 0.03, "moe": 0.02, "mhc": 0.012, "head": 0.01, "model": 0.03}[case["kind"]]}


# ---- 64-bit results ---------------------------------------------------------------------------------------------------------------
def exact(case, seed):
    c = case
    if c["kind"] == "model" or (c["kind"] == "qsa" and not c["train"]):
        return None                                                       # whole model: no short form; block selection: discrete
    t = _tensors(c, seed)
    w = {k: v.double().requires_grad_(c["train"]) for k, v in t["weights"].items()}
    x = t["x"].double().requires_grad_(c["train"])
    with torch.set_grad_enabled(c["train"]):
        kl = None
        if c["kind"] == "qsa":
            y, kl = _exact_qsa(c, w, x)
        elif c["kind"] == "head":
            y = F.cross_entropy(x @ w["weight"].t(), t["target"])
        else:
            y = {"gdn": _exact_gdn, "moe": _exact_moe, "mhc": _exact_mhc}[c["kind"]](c, w, x)
    if not c["train"]:
        return {"y": y}
    sparse = c["kind"] == "qsa" and not c["dense"]
    if c["kind"] == "head":
        y.backward()
    elif sparse:
        kl.backward()
    elif kl is not None:
        torch.autograd.backward([y, kl], [t["dy"].double(), torch.ones_like(kl)])
    else:
        y.backward(t["dy"].double())
    out = {"y": None if sparse else y.detach(), "dx": None if sparse else x.grad}
    if kl is not None:
        out["kl"] = kl.detach()
    # behind the discrete block selection only the KL and the indexer's gradients are a function of the inputs alone
    out.update({"d " + k: None if sparse and not k.startswith("indexer.") else p.grad for k, p in w.items()})
    return out


def _exact_gdn(c, w, x):
    B, S, _ = x.shape
    Hk, Hv, n = c["k_heads"], c["v_heads"], S // BLOCK
    qkv = F.conv1d((x @ w["in_proj_qkv.weight"].t()).transpose(1, 2), w["conv1d.weight"], None, padding=3, groups=w["conv1d.weight"].shape[0])
    qkv = F.silu(qkv[..., :S]).transpose(1, 2)
    q, k, v = qkv.split([64 * Hk, 64 * Hk, 64 * Hv], -1)
    unit = lambda t: t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6)
    chunks = lambda t, H: t.view(B, n, BLOCK, H, -1).permute(0, 3, 1, 2, 4)
    q = chunks(unit(q.reshape(B, S, Hk, 64)) / 8, Hk).repeat_interleave(Hv // Hk, 1)
    k = chunks(unit(k.reshape(B, S, Hk, 64)), Hk).repeat_interleave(Hv // Hk, 1)
    v = chunks(v.reshape(B, S, Hv, 64), Hv)
    beta = chunks((x @ w["in_proj_b.weight"].t()).sigmoid()[..., None], Hv)
    g = -w["A_log"].exp() * F.softplus(x @ w["in_proj_a.weight"].t() + w["dt_bias"])
    gc = chunks(g[..., None], Hv).cumsum(-2)
    low = torch.ones(BLOCK, BLOCK, dtype=torch.bool, device=x.device).tril()
    decay = (gc - gc.transpose(-1, -2)).masked_fill(~low, float("-inf")).exp()
    system = (beta * k) @ k.transpose(-1, -2) * decay
    u = torch.linalg.solve_triangular(system, beta * v, upper=False, unitriangular=True)
    ww = torch.linalg.solve_triangular(system, beta * gc.exp() * k, upper=False, unitriangular=True)
    P, qg, kg = (q @ k.transpose(-1, -2)) * decay, q * gc.exp(), k * (gc[..., -1:, :] - gc).exp()
    state, outs = x.new_zeros(B, Hv, 64, 64), []
    for i in range(n):
        fresh = u[:, :, i] - ww[:, :, i] @ state
        outs.append(qg[:, :, i] @ state + P[:, :, i] @ fresh)
        state = gc[:, :, i, -1:, :].exp() * state + kg[:, :, i].transpose(-1, -2) @ fresh
    o = torch.stack(outs, 2).reshape(B, Hv, S, 64).transpose(1, 2)
    o = o * torch.rsqrt(o.pow(2).mean(-1, keepdim=True) + 1e-6) * w["norm.weight"]
    o = o.reshape(B, S, -1) * F.silu(x @ w["in_proj_z.weight"].t())
    return o @ w["out_proj.weight"].t()


def _exact_moe(c, w, x):
    f = c["ffn"]
    x2 = x.reshape(-1, x.shape[-1])
    top_p, top_i = (x2 @ w["gate.weight"].t()).softmax(-1).topk(TOPK, -1)
    top_p = top_p / top_p.sum(-1, keepdim=True)
    y = (F.silu(x2 @ w["shared_expert.gate_proj.weight"].t()) * (x2 @ w["shared_expert.up_proj.weight"].t())) @ w["shared_expert.down_proj.weight"].t()
    y = y * torch.sigmoid(x2 @ w["shared_expert_gate.weight"].t())
    for e in range(EXPERTS):
        rows, slot = (top_i == e).nonzero(as_tuple=True)
        gu = x2[rows] @ w["experts.gate_up_proj"][e].t()
        part = (F.silu(gu[:, :f]) * gu[:, f:]) @ w["experts.down_proj"][e].t()
        y = y.index_add(0, rows, part * top_p[rows, slot][:, None])
    return y.view_as(x)


def _exact_mhc(c, w, X):
    xf = X.flatten(2)
    xf = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-6)
    z = torch.tanh(xf @ w["mhc.A.weight"].t() @ w["mhc.B.weight"].t())
    a = w["mhc.alphas"]
    pre = torch.sigmoid(w["mhc.b_pre"] + a[0] * z[..., :4])
    post = 2 * torch.sigmoid(w["mhc.b_post"] + a[1] * z[..., 4:8])
    logits = w["mhc.b_res"] + a[2] * z[..., 8:].unflatten(-1, (4, 4))
    res = torch.exp(logits - logits.amax((-2, -1), keepdim=True))
    for _ in range(20):
        res = res / res.sum(-1, keepdim=True).clamp(min=1e-9)
        res = res / res.sum(-2, keepdim=True).clamp(min=1e-9)
    xin = (pre[..., None] * X).sum(2)
    xin = xin * torch.rsqrt(xin.pow(2).mean(-1, keepdim=True) + 1e-6) * (1 + w["norm.weight"])
    return res @ X + post[..., None] * xin[:, :, None]


def _exact_qsa(c, w, x):
    B, S, _ = x.shape
    nq, nkv = c["heads"], c["kv_heads"]
    freq = 1.0 / (1e7 ** (torch.arange(0, 16, 2, device=x.device).float() / 16))
    ang = (torch.arange(S, device=x.device).float()[:, None] * freq).double()
    cos, sin = torch.cat([ang, ang], -1).cos(), torch.cat([ang, ang], -1).sin()

    def rope(t):                                                          # [B, H, S, 64]: the first 16 dims are rotated
        r = t[..., :16]
        return torch.cat([r * cos + torch.cat([-r[..., 8:], r[..., :8]], -1) * sin, t[..., 16:]], -1)

    norm = lambda t, g: t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + 1e-6) * (1 + g)
    qg = (x @ w["attn.q_proj.weight"].t()).view(B, S, nq, 128)
    q, gate = rope(norm(qg[..., :64], w["attn.q_norm.weight"]).transpose(1, 2)), qg[..., 64:].reshape(B, S, -1)
    k = rope(norm((x @ w["attn.k_proj.weight"].t()).view(B, S, nkv, 64), w["attn.k_norm.weight"]).transpose(1, 2))
    v = (x @ w["attn.v_proj.weight"].t()).view(B, S, nkv, 64).transpose(1, 2)
    xd = x.detach()
    qi = rope((xd @ w["indexer.wq.weight"].t()).view(B, S, 4, 64).transpose(1, 2))
    ki = rope((xd @ w["indexer.wk.weight"].t()).view(B, S, 1, 64).transpose(1, 2))[:, 0]
    wi = (xd @ w["indexer.ww.weight"].t()) / 2

    def rows(q, k, v, qi, ki, wi, t0):                                    # one sequence, queries t0 .. t0 + len(q)
        hide = torch.arange(k.shape[1], device=x.device)[None] > (t0 + torch.arange(q.shape[1], device=x.device))[:, None]
        p = (q.unflatten(0, (nkv, -1)) @ k[:, None].transpose(-1, -2) / 8).masked_fill(hide, float("-inf")).softmax(-1)
        o = (p @ v[:, None]).flatten(0, 1)
        mass = p.detach().unflatten(-1, (-1, BLOCK)).sum(-1).mean((0, 1))
        score = (F.relu(qi @ ki.t()) / 8 * wi.t()[..., None]).sum(0).masked_fill(hide, -1e9)
        lp = score.log_softmax(-1).unflatten(-1, (-1, BLOCK)).logsumexp(-1)
        return o, torch.where(mass > 0, mass * (mass.clamp(min=1e-300).log() - lp), torch.zeros_like(lp)).sum()

    outs, kl = [], 0
    for b in range(B):
        parts = []
        for t0 in range(0, S, 256):
            t1 = min(S, t0 + 256)
            o, term = torch.utils.checkpoint.checkpoint(rows, q[b, :, t0:t1], k[b, :, :t1], v[b, :, :t1], qi[b, :, t0:t1], ki[b, :t1], wi[b, t0:t1], t0,
                                                        use_reentrant=False)
            parts.append(o)
            kl = kl + term
        outs.append(torch.cat(parts, 1))
    o = torch.stack(outs).transpose(1, 2).reshape(B, S, -1) * torch.sigmoid(gate)
    return o @ w["attn.o_proj.weight"].t(), kl / (B * S)
