"""Delta-rule kernels at the edges of their dispatch and pipelines, against the recurrences in 64 bits."""
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


def chunk_operands(BH, NT, seed):
    """Operands with the sizes the preparation kernel gives them: w, kg of unit-norm rows, P and qg scaled by 1/8, decays in (0, 1)."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    t = [torch.randn(BH, NT, 64, 64, device="cuda", generator=gen) for _ in range(5)]
    w, u, P, qg, kg = (t[0] / 16, t[1], t[2].tril() / 64, t[3] / 64, t[4] / 16)
    return [x.to(torch.bfloat16) for x in (w, u, P, qg, kg)] + [torch.rand(BH, NT, device="cuda", generator=gen)]


# 1 and 37 pairs: four CTAs per pair; 38 and 74: two; 75: one; 156: more pairs than SMs; chunk counts below, at and above the three and four pipeline stages
@pytest.mark.parametrize("B,H", [(1, 1), (1, 37), (2, 19), (2, 37), (5, 15), (4, 39)])
@pytest.mark.parametrize("NT", [1, 2, 3, 4, 5, 9])
def test_scan_forward(ops, B, H, NT):
    BH = B * H
    w, u, P, qg, kg, d = chunk_operands(BH, NT, 10 * NT + BH)
    lib = ops.load()
    o, vnew, states = lib.gdn_scan_fwd(w, u, P, qg, kg, d, B, H, ops.error_flag())
    o2, v2, s2 = lib.gdn_scan_fwd(w, u, P, qg, kg, d, B, H, ops.error_flag(), False)
    ops.check_errors()
    assert torch.equal(o, o2) and v2.numel() == s2.numel() == 0
    S = torch.zeros(BH, 64, 64, device="cuda", dtype=torch.float64)
    f = [x.double() for x in (w, u, P, qg, kg)]
    for c in range(NT):
        v = f[1][:, c] - f[0][:, c] @ S
        out = (f[3][:, c] @ S + f[2][:, c] @ v).view(B, H, 64, 64).transpose(1, 2)
        # bf16 operands of every product (2^-9 each) carried along the chunks: three roundings of 2e-3 (rms) and their propagation
        assert rel(states[:, c], S) < 1e-2 and rel(vnew[:, c], v) < 1e-2 and rel(o[:, 64 * c:64 * c + 64], out) < 1e-2, c
        S = d[:, c, None, None].double() * S + f[4][:, c].transpose(-1, -2) @ v


def recurrence(qkv, g, beta, Hk, Hv):
    B, S, _ = qkv.shape
    q, k, v = qkv.split([64 * Hk, 64 * Hk, 64 * Hv], -1)
    unit = lambda t: t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6)
    q = (unit(q.reshape(B, S, Hk, 64)) / 8).repeat_interleave(Hv // Hk, 2)
    k = unit(k.reshape(B, S, Hk, 64)).repeat_interleave(Hv // Hk, 2)
    v = v.reshape(B, S, Hv, 64)
    state, outs = qkv.new_zeros(B, Hv, 64, 64), []
    for t in range(S):
        state = state * g[:, t].exp()[..., None, None]
        fresh = (v[:, t] - torch.einsum("bhkv,bhk->bhv", state, k[:, t])) * beta[:, t][..., None]
        state = state + k[:, t][..., None] * fresh[..., None, :]
        outs.append(torch.einsum("bhkv,bhk->bhv", state, q[:, t]))
    return torch.stack(outs, 1)


# one and three value heads per key head; one chunk, an odd number of chunks; heads that forget at once and heads that keep everything
# (the reverse scan runs one warp per CTA up to 37 pairs, then two)
@pytest.mark.parametrize("B,S,Hk,Hv", [(1, 64, 1, 1), (2, 192, 2, 6), (1, 320, 13, 39)])
@pytest.mark.parametrize("decay", [0.0, 0.05, 20.0])
def test_delta_rule_gradients(ops, B, S, Hk, Hv, decay):
    from q38.ops.backend import _DeltaRule
    gen = torch.Generator(device="cuda").manual_seed(S + Hv)
    qkv = torch.randn(B, S, (2 * Hk + Hv) * 64, device="cuda", generator=gen).to(torch.bfloat16).requires_grad_()
    g = (-decay * torch.rand(B, S, Hv, device="cuda", generator=gen)).requires_grad_()
    beta = torch.rand(B, S, Hv, device="cuda", generator=gen).to(torch.bfloat16)
    beta[:, ::7] = 0                                           # tokens that write nothing still have a beta gradient
    beta.requires_grad_()
    do = torch.randn(B, S, Hv, 64, device="cuda", generator=gen).to(torch.bfloat16)
    o = _DeltaRule.apply(qkv, g, beta, Hk, Hv)
    o.backward(do)
    ops.check_errors()
    ref = [t.detach().double().requires_grad_() for t in (qkv, g, beta)]
    ro = recurrence(*ref, Hk, Hv)
    ro.backward(do.double())
    # bf16 chunk operands (2e-3 rms each); the gate gradients are differences of row and column sums of those products
    assert rel(o, ro.detach()) < 1.5e-2 and rel(qkv.grad, ref[0].grad) < 2e-2 and rel(beta.grad, ref[2].grad) < 2e-2
    if decay:
        assert rel(g.grad, ref[1].grad) < 2.5e-2
    zero = beta.detach() == 0
    assert rel(beta.grad[zero], ref[2].grad[zero]) < 2e-2


def test_delta_rule_gradients_with_negative_beta(ops):
    """The rule is defined for any beta; a sigmoid never gives a negative one, a caller of the rule may."""
    from q38.ops.backend import _DeltaRule
    B, S, Hk, Hv = 1, 192, 2, 6
    gen = torch.Generator(device="cuda").manual_seed(3)
    qkv = torch.randn(B, S, (2 * Hk + Hv) * 64, device="cuda", generator=gen).to(torch.bfloat16).requires_grad_()
    g = (-0.1 * torch.rand(B, S, Hv, device="cuda", generator=gen)).requires_grad_()
    beta = (torch.rand(B, S, Hv, device="cuda", generator=gen) - 0.5).to(torch.bfloat16)
    beta[:, ::7] = 0
    beta.requires_grad_()
    do = torch.randn(B, S, Hv, 64, device="cuda", generator=gen).to(torch.bfloat16)
    _DeltaRule.apply(qkv, g, beta, Hk, Hv).backward(do)
    ops.check_errors()
    ref = [t.detach().double().requires_grad_() for t in (qkv, g, beta)]
    recurrence(*ref, Hk, Hv).backward(do.double())
    # the bounds of the positive case: bf16 chunk operands, 2e-3 rms each
    assert rel(qkv.grad, ref[0].grad) < 2e-2 and rel(beta.grad, ref[2].grad) < 2e-2 and rel(g.grad, ref[1].grad) < 2.5e-2
    for part in (beta.detach() < 0, beta.detach() == 0):
        assert rel(beta.grad[part], ref[2].grad[part]) < 2e-2


def test_beta_gradient_is_summed_in_32_bits(ops):
    """Every factor is exact in bf16 and only the gradient of the triangular system, an integer of up to sixteen bits, is not: beta's gradient comes
    from its fp32 form.  Only token 0 writes (beta = 0 elsewhere) and only token 63 has an upstream gradient."""
    gen = torch.Generator(device="cuda").manual_seed(5)
    sign = lambda *s: torch.randint(0, 2, s, device="cuda", generator=gen).float() * 2 - 1
    q, k, v = sign(1, 64, 64), sign(1, 64, 64), torch.zeros(1, 64, 64, device="cuda")
    v[:, 0] = torch.randint(-15, 16, (64,), device="cuda", generator=gen).float()
    qkv = torch.cat([q, k, v], -1).to(torch.bfloat16)
    g, beta = torch.zeros(1, 64, 1, device="cuda"), torch.zeros(1, 64, 1, device="cuda", dtype=torch.bfloat16)
    beta[:, 0] = 0.5
    do = torch.zeros(1, 64, 1, 64, device="cuda", dtype=torch.bfloat16)
    do[:, 63] = sign(1, 64).to(torch.bfloat16)
    lib = ops.load()
    _, *saved = lib.gdn_rule_fwd(qkv, g, beta, 1, 1, ops.error_flag(), True)
    dbeta = lib.gdn_rule_bwd(qkv, g, beta, saved, do, 1, 1, ops.error_flag())[2]
    ops.check_errors()
    ref = [t.double().requires_grad_() for t in (qkv, g, beta)]
    recurrence(*ref, 1, 1).backward(do.double())
    # rounded to bf16 before the sum it is 1e-3 off; what is left is the 1e-6 in the norms against 64 and fp32 sums
    assert rel(dbeta[:, 1:], ref[2].grad[:, 1:]) < 1e-5
