"""Layer calls (one native call per pass) against the op-by-op path of the same hook: the same launches, so the same bits.

The key and value gradients of the attention and the indexer's key gradient are added with fp32 atomics in both, and so are split weight
gradients: these are compared to 1e-3 of their norm (one bf16 rounding of a sum whose order varies)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
HIDDEN, S = 64, 128


@pytest.fixture(scope="module")
def modeling():
    from q38 import ops
    from q38.models import modeling
    ops.install()
    return modeling


def build(modeling, kind):
    from q38.presets import model_config
    shape = dict(layers=4, hidden=HIDDEN, heads=6, kv_heads=2, lin_k_heads=2, lin_v_heads=6, experts=8, topk=2, moe_ffn=32, shared_ffn=32, ngram_rows=64)
    cfg = model_config(shape, 512, S, bos_token_id=1, eos_token_id=2, pad_token_id=0)
    torch.manual_seed(0)
    with torch.device("cuda"):
        if kind == "gdn":
            module = modeling.Qwen3_8MoeGatedDeltaNet(cfg, 0)
        elif kind == "moe":
            module = modeling.Qwen3_8MoeSparseMoeBlock(cfg)
            torch.nn.init.normal_(module.experts.gate_up_proj, std=0.1)
            torch.nn.init.normal_(module.experts.down_proj, std=0.1)
        elif kind == "mhc":
            module = torch.nn.ModuleDict(dict(mhc=modeling.MHC(HIDDEN), norm=modeling.Qwen3_8MoeRMSNorm(HIDDEN)))
        elif kind == "head":
            module = torch.nn.Linear(HIDDEN, 512, bias=False)
        else:
            module = torch.nn.ModuleDict(dict(attn=modeling.Qwen3_8MoeAttention(cfg, 3), indexer=modeling.Indexer(HIDDEN, 4, 64)))
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
        return [linear_cross_entropy(module.weight, x.reshape(-1, HIDDEN), target)]
    cos, sin = modeling.rope_tables(torch.arange(S, device="cuda")[None], 16, 1e7, torch.float32)
    train = x.requires_grad or any(p.requires_grad for p in module.parameters())
    y, kl = modeling.qsa_attention(module["attn"], x, cos, sin, None if "plain" in kind else module["indexer"], 1, "dense" in kind, train and "kl" in kind)
    return [out for name, out in (("y", y), ("kl", kl)) if out is not None and name in parts and (not train or out.requires_grad)]


KINDS = ["gdn", "moe", "mhc", "head", "qsa kl", "qsa kl dense", "qsa dense", "qsa", "qsa plain dense"]
MODES = ["infer", "buffers", "fresh", "side stream", "frozen input", "frozen weights", "y alone", "kl alone"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("mode", MODES)
def test_layer_call_matches_its_ops(modeling, kind, mode, monkeypatch):
    from q38.ops.backend import WGRAD_STREAM
    if "alone" in mode and "kl" not in kind:
        pytest.skip("one output")
    backend = modeling.get_backend()
    gen = torch.Generator(device="cuda").manual_seed(1)
    shape = (2, S, 4, HIDDEN) if kind == "mhc" else (2, S, HIDDEN)
    x0 = torch.randn(shape, device="cuda", generator=gen)
    x0 = x0 if kind == "mhc" else x0.to(torch.bfloat16)
    target = torch.randint(0, 512, (2 * S,), device="cuda", generator=gen)
    parts = {"y alone": ("y",), "kl alone": ("kl",)}.get(mode, ("y", "kl"))
    results = []
    for native in (True, False):
        module = build(modeling, kind)
        if not native:
            monkeypatch.setattr(backend, "native_layers", lambda hidden: False)
        calls = []
        if native and kind != "head":
            from q38.ops import backend as ops_backend
            lib = ops_backend.load()
            monkeypatch.setattr(ops_backend, "load", lambda: calls.append(1) or lib)
        x = x0.clone().requires_grad_(mode not in ("infer", "frozen input"))
        names = [n for n, _ in module.named_parameters()]
        for i, p in enumerate(module.parameters()):
            p.requires_grad_(mode != "infer" and not (mode == "frozen weights" and i % 2))
            if mode not in ("fresh", "infer") and p.requires_grad:
                p.grad = torch.full_like(p, 0.25)
        WGRAD_STREAM.enabled = mode == "side stream"
        with torch.set_grad_enabled(mode != "infer"):
            outs = run(modeling, module, kind, x, target, parts)
            if mode != "infer":
                torch.autograd.backward(outs, [torch.ones_like(o) * 0.5 for o in outs])
                WGRAD_STREAM.join()
        WGRAD_STREAM.enabled = False
        if native and kind != "head":
            assert len(calls) <= 4, "the op-by-op path ran"
            monkeypatch.undo()
        results.append([("out", o.detach()) for o in outs] + [("dx", x.grad)] + [(n, p.grad) for n, p in zip(names, module.parameters())])
    for (name, got), (_, want) in zip(*results):
        assert (got is None) == (want is None), name
        if got is not None:
            assert got.dtype == want.dtype and got.shape == want.shape
            err = (got.double() - want.double()).norm() / want.double().norm().clamp_min(1e-30)
            assert err <= (0 if name == "out" else 1e-3), (name, float(err))


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
