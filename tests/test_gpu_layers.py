"""Layer calls (one native call per pass) against the op-by-op path of the same hook: the same launches, so the same bits.

Sums whose order varies are compared to 1e-3 of their norm (one bf16 rounding of such a sum): the key and value gradients of the attention and the
indexer's key gradient (fp32 atomics), what is computed from them, the small parameters' gradients, and split weight gradients.  Where a gradient is added to a buffer, what was
added is compared, not the sum, and the buffer's content is of the gradient's own size."""
import pytest
import torch

pytestmark = pytest.mark.gpu
HIDDEN, S = 64, 128
# hidden width, tokens per sequence (an even, a single and an odd number of blocks), heads, KV heads, key and value heads of the delta rule
SHAPES = {"even": (64, 128, 6, 2, 2, 6), "single": (192, 64, 5, 1, 3, 3), "odd": (128, 192, 4, 4, 1, 4)}


@pytest.fixture(scope="module")
def modeling():
    from q38 import ops
    from q38.models import modeling
    ops.install()
    return modeling


def build(modeling, kind, shape="even"):
    from q38.presets import model_config
    hidden, seq, heads, kv_heads, k_heads, v_heads = SHAPES[shape]
    cfg = model_config(dict(layers=4, hidden=hidden, heads=heads, kv_heads=kv_heads, lin_k_heads=k_heads, lin_v_heads=v_heads, experts=8, topk=2, moe_ffn=32, shared_ffn=32,
                            ngram_rows=64), 512, seq, bos_token_id=1, eos_token_id=2, pad_token_id=0)
    torch.manual_seed(0)
    with torch.device("cuda"):
        if kind == "gdn":
            module = modeling.Qwen3_8MoeGatedDeltaNet(cfg, 0)
        elif kind == "moe":
            module = modeling.Qwen3_8MoeSparseMoeBlock(cfg)
            torch.nn.init.normal_(module.experts.gate_up_proj, std=0.1)
            torch.nn.init.normal_(module.experts.down_proj, std=0.1)
        elif kind == "mhc":
            module = torch.nn.ModuleDict(dict(mhc=modeling.MHC(hidden), norm=modeling.Qwen3_8MoeRMSNorm(hidden)))
        elif kind == "head":
            module = torch.nn.Linear(hidden, 512, bias=False)
        else:
            module = torch.nn.ModuleDict(dict(attn=modeling.Qwen3_8MoeAttention(cfg, 3), indexer=modeling.Indexer(hidden, 4, 64)))
    return module


def run(modeling, module, kind, x, target, parts):
    if kind == "gdn" or kind == "moe":
        return [module(x)]
    if kind == "mhc":
        backend = modeling.get_backend()
        xin, link = backend.mhc_pre_norm(module["mhc"], module["norm"], x, torch.bfloat16)
        return [backend.mhc_post(module["mhc"], xin, link)]
    if kind == "head":
        from q38.losses import linear_cross_entropy
        return [linear_cross_entropy(module.weight, x.reshape(-1, x.shape[-1]), target)]
    cos, sin = modeling.rope_tables(torch.arange(x.shape[1], device="cuda")[None], 16, 1e7, torch.float32)
    train = x.requires_grad or any(p.requires_grad for p in module.parameters())
    y, kl = modeling.qsa_attention(module["attn"], x, cos, sin, None if "plain" in kind else module["indexer"], 1, "dense" in kind, train and "kl" in kind)
    return [out for name, out in (("y", y), ("kl", kl)) if out is not None and name in parts and (not train or out.requires_grad)]


KINDS = ["gdn", "moe", "mhc", "head", "qsa kl", "qsa kl dense", "qsa dense", "qsa", "qsa plain dense"]
MODES = ["infer", "buffers", "fresh", "side stream", "frozen input", "frozen weights", "y alone", "kl alone"]
CASES = [(mode, "even") for mode in MODES] + [(mode, shape) for shape in ("single", "odd") for mode in ("infer", "buffers", "fresh")]
# results with sums whose order varies, besides weight gradients that are added to a buffer
ANY_ORDER = {"gdn": ("conv1d.weight", "A_log", "dt_bias", "norm.weight"), "moe": (), "mhc": ("mhc.B.weight", "mhc.b_pre", "mhc.b_post", "mhc.b_res", "mhc.alphas", "norm.weight"), "head": (),
             "qsa": ("dx", "attn.k_proj.weight", "attn.v_proj.weight", "attn.q_norm.weight", "attn.k_norm.weight", "indexer.wk.weight")}


class Library:
    """The kernel library, with the names of the operators that were called."""

    def __init__(self, lib):
        self.lib, self.called = lib, set()

    def __getattr__(self, name):
        self.called.add(name)
        return getattr(self.lib, name)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("mode,shape", CASES)
def test_layer_call_matches_its_ops(modeling, kind, mode, shape, monkeypatch):
    from q38.ops import backend as ops_backend
    from q38.ops.backend import WGRAD_STREAM
    if "alone" in mode and "kl" not in kind:
        pytest.skip("one output")
    backend = modeling.get_backend()
    hidden, seq = SHAPES[shape][:2]
    gen = torch.Generator(device="cuda").manual_seed(1)
    x0 = torch.randn((2, seq, 4, hidden) if kind == "mhc" else (2, seq, hidden), device="cuda", generator=gen)
    x0 = x0 if kind == "mhc" else x0.to(torch.bfloat16)
    target = torch.randint(0, 512, (2 * seq,), device="cuda", generator=gen)
    parts = {"y alone": ("y",), "kl alone": ("kl",)}.get(mode, ("y", "kl"))
    op = {"gdn": "gdn_layer", "moe": "moe_layer", "mhc": "mhc_layer", "head": "linear_ce"}.get(kind, "qsa_layer")

    def once(native, buffers):
        """Outputs and gradients; `buffers`: what the gradient buffers hold before, by name."""
        module = build(modeling, kind, shape)
        library = Library(ops_backend.load())
        x = x0.clone().requires_grad_(mode not in ("infer", "frozen input"))
        for i, (name, p) in enumerate(module.named_parameters()):
            p.requires_grad_(mode != "infer" and not (mode == "frozen weights" and i % 2))
            if name in buffers and p.requires_grad:
                p.grad = buffers[name].clone()
        WGRAD_STREAM.enabled = mode == "side stream"
        with monkeypatch.context() as patch, torch.set_grad_enabled(mode != "infer"):
            patch.setattr(ops_backend, "load", lambda: library)
            if not native:
                patch.setattr(backend, "native_layers", lambda hidden: False)
            outs = run(modeling, module, kind, x, target, parts)
            if mode != "infer":
                torch.autograd.backward(outs, [torch.ones_like(o) * 0.5 for o in outs])
                WGRAD_STREAM.join()
        WGRAD_STREAM.enabled = False
        used = {name for name in library.called if "_layer_" in name or name.startswith("linear_ce_")}
        assert used == ({op + "_fwd"} | ({op + "_bwd"} if mode != "infer" else set()) if native else set())
        added = {n: p.grad if n not in buffers or p.grad is None else p.grad - buffers[n] for n, p in module.named_parameters()}
        return {**{f"out {i}": o.detach() for i, o in enumerate(outs)}, "dx": x.grad, **added}

    buffers = {}
    if mode not in ("infer", "fresh"):
        own = once(False, {})
        noise = lambda g: torch.randn(g.shape, device="cuda", generator=gen) * (g.double().pow(2).mean().sqrt().float() if bool(g.any()) else 1e-3)
        buffers = {n: noise(torch.zeros_like(p) if own[n] is None else own[n]) for n, p in build(modeling, kind, shape).named_parameters()}
    got, want = once(True, buffers), once(False, buffers)
    assert got.keys() == want.keys()
    for name in got:
        a, b = got[name], want[name]
        assert (a is None) == (b is None), name
        if a is None:
            continue
        assert a.dtype == b.dtype and a.shape == b.shape
        if buffers and name in buffers:
            assert bool(b.any()) == (own[name] is not None and bool(own[name].any())), (name, "nothing was added")
            if own[name] is not None:
                assert (a.double() - own[name].double()).norm() <= 1e-3 * own[name].double().norm(), (name, "not the gradient that is returned without a buffer")
        err = (a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30)
        varies = name in ANY_ORDER[kind.split()[0]] or name in buffers
        assert err <= (1e-3 if varies else 0), (name, float(err))


def test_layer_call_under_activation_checkpointing(modeling):
    module, x = build(modeling, "gdn"), torch.randn(1, S, HIDDEN, device="cuda").to(torch.bfloat16)
    grads = []
    for wrap in (lambda f, t: f(t), lambda f, t: torch.utils.checkpoint.checkpoint(f, t, use_reentrant=False)):
        leaf = x.clone().requires_grad_()
        wrap(module, leaf).sum().backward()
        grads.append(leaf.grad)
    assert torch.equal(*grads)


def test_layer_call_refuses_forward_mode(modeling):
    module, x = build(modeling, "gdn"), torch.randn(1, S, HIDDEN, device="cuda").to(torch.bfloat16)
    with torch.autograd.forward_ad.dual_level():
        with pytest.raises(RuntimeError):
            module(torch.autograd.forward_ad.make_dual(x, torch.ones_like(x)))


@pytest.mark.parametrize("kind", ["gdn", "moe", "mhc", "head", "qsa kl"])
@pytest.mark.parametrize("mode", ["frozen", "fresh", "buffers"])
def test_side_stream_is_joined_where_it_was_used(modeling, kind, mode):
    """A pass whose weight gradients are not wanted, or are returned, puts nothing on the second stream; a join there would make a capture wait for a
    stream that never entered it."""
    from q38.ops.backend import WGRAD_STREAM
    module = build(modeling, kind).requires_grad_(mode != "frozen")
    for p in module.parameters():
        p.grad = torch.zeros_like(p) if mode == "buffers" else None
    x = torch.randn((1, S, 4, HIDDEN) if kind == "mhc" else (1, S, HIDDEN), device="cuda").to(torch.float32 if kind == "mhc" else torch.bfloat16).requires_grad_()
    target = torch.randint(0, 512, (S,), device="cuda")
    WGRAD_STREAM.enabled = True
    try:
        assert not WGRAD_STREAM.pending
        outs = run(modeling, module, kind, x, target, ("y",) if mode == "frozen" else ("y", "kl"))
        torch.autograd.backward(outs, [torch.ones_like(o) for o in outs])
        assert WGRAD_STREAM.pending == (mode == "buffers")
    finally:
        WGRAD_STREAM.join()
        WGRAD_STREAM.enabled = False


@pytest.mark.parametrize("kind", ["gdn", "moe", "mhc", "qsa kl", "qsa"])
def test_layer_results_are_memory_of_their_own(modeling, kind, monkeypatch):
    """The operators' schemas declare no result that shares memory with an argument, or with another result."""
    from q38.ops import backend as ops_backend
    lib, checked = ops_backend.load(), []

    def own(call):
        def wrapped(*args):
            results = call(*args)
            flat = [t for a in args for t in (a if isinstance(a, (list, tuple)) else [a]) if isinstance(t, torch.Tensor) and t.numel()]
            seen = {t.untyped_storage().data_ptr() for t in flat}
            for t in results:
                if t is not None and t.numel():
                    assert t.untyped_storage().data_ptr() not in seen, t.shape
                    seen.add(t.untyped_storage().data_ptr())
            checked.append(1)
            return results
        return wrapped

    class Library:
        def __getattr__(self, name):
            return own(getattr(lib, name)) if name.endswith("_layer_fwd") else getattr(lib, name)

    monkeypatch.setattr(ops_backend, "load", lambda: Library())
    x = torch.randn((1, S, 4, HIDDEN) if kind == "mhc" else (1, S, HIDDEN), device="cuda").to(torch.float32 if kind == "mhc" else torch.bfloat16).requires_grad_()
    run(modeling, build(modeling, kind), kind, x, None, ("y", "kl"))
    assert checked
