"""Attention, indexer and convolution kernels at the edges of their splits, against the same sums in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from q38 import ops as q38_ops
    q38_ops.install()
    return q38_ops


def rel(a, b):
    return ((a.double() - b).norm() / b.norm().clamp_min(1e-30)).item()


# head counts that leave the second group of warps with zero, one and two heads; one block, and an odd number above the key pass's split of eight
@pytest.mark.parametrize("NI", [1, 2, 3, 4])
@pytest.mark.parametrize("B,nb", [(1, 1), (2, 3), (1, 11)])
def test_indexer_backward(ops, NI, B, nb):
    S, scale = 64 * nb, 0.125
    gen = torch.Generator(device="cuda").manual_seed(7 * NI + nb)
    qi = torch.randn(B, NI, S, 64, device="cuda", generator=gen).to(torch.bfloat16)
    ki = torch.randn(B, S, 64, device="cuda", generator=gen).to(torch.bfloat16)
    wi = torch.randn(B, S, NI, device="cuda", generator=gen) / 2
    lib = ops.load()
    blse = lib.qsa_indexer_fwd(qi, ki, wi, scale)
    dblse = torch.randn(B, S, nb, device="cuda", generator=gen)
    dqi, dki, dwi = lib.qsa_indexer_bwd(qi, ki, wi, blse, dblse, 0.5, scale)
    q, k, w = (t.double().requires_grad_() for t in (qi, ki, wi))
    score = (torch.relu(q @ k[:, None].transpose(-1, -2)) * scale * w.transpose(1, 2)[..., None]).sum(1)
    causal = torch.ones(S, S, dtype=torch.bool, device="cuda").tril()
    lse = score.masked_fill(~causal, float("-inf")).unflatten(-1, (nb, 64)).logsumexp(-1)
    own = torch.arange(S, device="cuda")[:, None] // 64 >= torch.arange(nb, device="cuda")[None]
    (torch.where(own, lse, torch.zeros_like(lse)) * dblse.double() * 0.5).sum().backward()
    # q.k is rounded to bf16 before the relu (scores move by 2e-3 of |q.k| ~ 8, the softmax weights by 1 %), dS once more before its products
    assert rel(dqi, q.grad) < 2e-2 and rel(dki, k.grad) < 2e-2 and rel(dwi, w.grad) < 2e-2


# query blocks with one to four shares of their key blocks
def test_indexer_query_gradients_have_the_same_bits_in_every_run(ops):
    B, NI, nb = 4, 4, 24
    S = 64 * nb
    gen = torch.Generator(device="cuda").manual_seed(0)
    qi = torch.randn(B, NI, S, 64, device="cuda", generator=gen).to(torch.bfloat16)
    ki = torch.randn(B, S, 64, device="cuda", generator=gen).to(torch.bfloat16)
    wi = torch.randn(B, S, NI, device="cuda", generator=gen) / 2
    lib = ops.load()
    blse = lib.qsa_indexer_fwd(qi, ki, wi, 0.125)
    dblse = torch.randn(B, S, nb, device="cuda", generator=gen)
    first = lib.qsa_indexer_bwd(qi, ki, wi, blse, dblse, 0.5, 0.125)
    for _ in range(20):
        again = lib.qsa_indexer_bwd(qi, ki, wi, blse, dblse, 0.5, 0.125)
        assert torch.equal(again[0], first[0]) and torch.equal(again[2], first[2])


def test_indexer_backward_refuses_what_its_tiles_do_not_hold(ops):
    B, S, nb = 1, 128, 2
    lib = ops.load()
    make = lambda NI: (torch.zeros(B, NI, S, 64, device="cuda", dtype=torch.bfloat16), torch.zeros(B, S, 64, device="cuda", dtype=torch.bfloat16),
                       torch.zeros(B, S, NI, device="cuda"), torch.zeros(B, S, nb, device="cuda"), torch.zeros(B, S, nb, device="cuda"))
    lib.qsa_indexer_bwd(*make(4), 1.0, 0.125)
    with pytest.raises(RuntimeError, match="at most 4 indexer heads"):
        lib.qsa_indexer_bwd(*make(5), 1.0, 0.125)
    for at, bad in ((1, lambda t: t.float()), (2, lambda t: t.double()), (2, lambda t: t[..., :1].expand_as(t)), (3, lambda t: t[..., :1]),
                    (4, lambda t: t.transpose(1, 2).contiguous().transpose(1, 2))):
        args = list(make(4))
        args[at] = bad(args[at])
        with pytest.raises(RuntimeError, match="required"):
            lib.qsa_indexer_bwd(*args, 1.0, 0.125)


# the own block alone, a list with gaps, every block (dense); the second half of a 64-row tile is what the half-tile loops reach last
@pytest.mark.parametrize("B,nb,nq,nkv,pick", [(1, 1, 2, 1, "dense"), (1, 5, 6, 2, "own"), (2, 7, 4, 2, "gaps"), (1, 33, 2, 1, "dense")])
def test_block_attention(ops, B, nb, nq, nkv, pick):
    S = 64 * nb
    gen = torch.Generator(device="cuda").manual_seed(nb)
    q = torch.randn(B, nq, S, 64, device="cuda", generator=gen).to(torch.bfloat16)
    k = torch.randn(B, nkv, S, 64, device="cuda", generator=gen).to(torch.bfloat16)
    v = torch.randn(B, nkv, S, 64, device="cuda", generator=gen).to(torch.bfloat16)
    do = torch.randn(B, S, nq, 64, device="cuda", generator=gen).to(torch.bfloat16)
    chosen = torch.ones(nb, nb, dtype=torch.bool).tril()
    if pick == "own":
        chosen = torch.eye(nb, dtype=torch.bool)
    elif pick == "gaps":
        chosen = chosen & ((torch.arange(nb)[:, None] - torch.arange(nb)[None]) % 3 == 0)
    count = index = None
    if pick != "dense":
        lists = [row.nonzero().flatten().tolist() for row in chosen]
        width = max(map(len, lists))
        index = torch.tensor([r[::-1] + [0] * (width - len(r)) for r in lists], dtype=torch.int32, device="cuda").expand(B, -1, -1).contiguous()
        count = torch.tensor([len(r) for r in lists], dtype=torch.int32, device="cuda").expand(B, -1).contiguous()
    lib = ops.load()
    o, lse, sel = lib.qsa_attn_fwd(q, k, v, count, index, 0.125)
    grads = lib.qsa_attn_bwd(q, k, v, o, do, lse, sel, 0.125)
    ref = [t.double().requires_grad_() for t in (q, k, v)]
    mask = chosen.cuda().repeat_interleave(64, 0).repeat_interleave(64, 1) & torch.ones(S, S, dtype=torch.bool, device="cuda").tril()
    s = (ref[0] @ ref[1].repeat_interleave(nq // nkv, 1).transpose(-1, -2) * 0.125).masked_fill(~mask, float("-inf"))
    ro = (s.softmax(-1) @ ref[2].repeat_interleave(nq // nkv, 1)).transpose(1, 2)
    ro.backward(do.double())
    # bf16 probabilities and score gradients (2e-3 rms each) and a bf16 output
    assert rel(o, ro.detach()) < 1e-2
    for got, want in zip(grads, ref):
        assert rel(got, want.grad) < 1.5e-2


# one thread and several blocks of channels; sequences below, at and above the runs of 32 and 128 tokens
@pytest.mark.parametrize("C", [2, 258])
@pytest.mark.parametrize("S", [1, 32, 128, 133])
def test_conv_silu(ops, C, S):
    gen = torch.Generator(device="cuda").manual_seed(C + S)
    x = torch.randn(2, S, C, device="cuda", generator=gen).to(torch.bfloat16)
    w = (torch.rand(C, 4, device="cuda", generator=gen) - 0.5).to(torch.bfloat16).float()
    dy = torch.randn(2, S, C, device="cuda", generator=gen).to(torch.bfloat16)
    lib = ops.load()
    y = lib.conv_silu_fwd(x, w)
    dx, dw = lib.conv_silu_bwd(x, w, dy)
    xr, wr = x.double().requires_grad_(), w.double().requires_grad_()
    yr = torch.nn.functional.silu(torch.nn.functional.conv1d(xr.transpose(1, 2), wr[:, None], None, padding=3, groups=C)[..., :S].transpose(1, 2))
    yr.backward(dy.double())
    # the convolution output is bf16 before the activation, and so are y and dx
    assert rel(y, yr.detach()) < 6e-3 and rel(dx, xr.grad) < 6e-3 and rel(dw, wr.grad) < 6e-3


def test_head_preparation_of_views(ops):
    """A contiguous view may start anywhere; other strides are refused wherever they start."""
    B, S, H = 1, 64, 3
    gen = torch.Generator(device="cuda").manual_seed(0)
    flat = torch.randn(B * S * H * 64 + 8, device="cuda", generator=gen).to(torch.bfloat16)
    cos, sin = (f(torch.rand(1, S, 8, device="cuda", generator=gen)).repeat(1, 1, 2) for f in (torch.cos, torch.sin))
    lib = ops.load()
    for first in (0, 1, 2, 8):
        view = flat[first:first + B * S * H * 64].view(B, S, H, 64)
        out = lib.qsa_headprep_fwd(view, None, cos, sin, 0.0, False)
        again = lib.qsa_headprep_fwd(view.clone(), None, cos, sin, 0.0, False)
        assert torch.equal(out[0], again[0])
    wide = torch.zeros(B, S, H, 72, device="cuda", dtype=torch.bfloat16)
    for first in (0, 1):
        with pytest.raises(RuntimeError, match="contiguous bf16"):
            lib.qsa_headprep_fwd(wide[..., first:first + 64], None, cos, sin, 0.0, False)
        with pytest.raises(RuntimeError, match="bad inputs"):
            lib.qsa_headprep_bwd(torch.zeros(B, H, S, 64, device="cuda", dtype=torch.bfloat16), None, wide[..., first:first + 64], None, cos, sin, torch.zeros(0, S, H, device="cuda"))


@pytest.mark.parametrize("norm", [False, True])
def test_head_preparation_weight_gradient_has_the_norm_s_shape(ops, norm):
    """64 values, zeros without a norm."""
    B, S, H = 1, 64, 3
    src, dout = torch.randn(B, S, H, 64, device="cuda").to(torch.bfloat16), torch.randn(B, H, S, 64, device="cuda").to(torch.bfloat16)
    cos, sin = (torch.rand(1, S, 16, device="cuda") for _ in range(2))
    w = torch.randn(64, device="cuda") if norm else None
    rstd = ops.load().qsa_headprep_fwd(src, w, cos, sin, 1e-6, False)[2]
    dw = ops.load().qsa_headprep_bwd(dout, None, src, w, cos, sin, rstd)[1]
    assert dw.shape == (64,) and dw.dtype == torch.float32 and bool(dw.any()) == norm
