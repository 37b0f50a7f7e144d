"""Residual-stream coefficients with few tokens and the smallest and largest Sinkhorn depths, against the same formulas in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def rel(a, b):
    return ((a.double() - b).norm() / b.norm().clamp_min(1e-30)).item()


# one token, one CTA of 32 tokens and one more; one iteration, the presets' twenty, the largest depth
@pytest.mark.parametrize("T", [1, 32, 33])
@pytest.mark.parametrize("iters", [1, 20, 32])
def test_coefficients_and_gradients(T, iters):
    from q38 import ops
    from q38.models import modeling
    ops.install()
    backend = modeling.get_backend()
    torch.manual_seed(T + iters)
    h = 64
    mhc, norm = modeling.MHC(h, iters=iters).cuda(), modeling.Qwen3_8MoeRMSNorm(h).cuda()
    with torch.no_grad():
        mhc.B.weight.normal_(0, 0.3)
        mhc.b_res.add_(torch.randn_like(mhc.b_res))
    X = torch.randn(1, T, 4, h, device="cuda", requires_grad=True)
    dY = torch.randn(1, T, 4, h, device="cuda")
    x, state = backend.mhc_pre_norm(mhc, norm, X, torch.float32)
    Y = backend.mhc_post(mhc, x.to(torch.bfloat16), state)
    Y.backward(dY)
    ops.check_errors()
    ref = {n: p.detach().double().requires_grad_() for n, p in mhc.named_parameters()}
    w, Xr = norm.weight.detach().double().requires_grad_(), X.detach().double().requires_grad_()
    xf = Xr.flatten(2)
    xf = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-6)
    z = torch.tanh(xf @ ref["A.weight"].t() @ ref["B.weight"].t())
    a = ref["alphas"]
    pre, post = torch.sigmoid(ref["b_pre"] + a[0] * z[..., :4]), 2 * torch.sigmoid(ref["b_post"] + a[1] * z[..., 4:8])
    logits = ref["b_res"] + a[2] * z[..., 8:].unflatten(-1, (4, 4))
    res = torch.exp(logits - logits.amax((-2, -1), keepdim=True))
    for _ in range(iters):
        res = res / res.sum(-1, keepdim=True).clamp(min=1e-9)
        res = res / res.sum(-2, keepdim=True).clamp(min=1e-9)
    xin = (pre[..., None] * Xr).sum(2)
    xin = xin * torch.rsqrt(xin.pow(2).mean(-1, keepdim=True) + norm.eps) * (1 + w)
    Yr = res @ Xr + post[..., None] * xin[:, :, None]
    Yr.backward(dY.double())
    # tf32 projection (1e-3) behind tanh, bf16 sub-layer output (2e-3); the coefficient gradients pass through bf16 copies of dL and X
    assert rel(state[1][:, 8:24].view(1, T, 4, 4), res.detach()) < 1e-3
    assert rel(Y, Yr.detach()) < 5e-3 and rel(X.grad, Xr.grad) < 1e-2
    for name in ("b_res", "b_pre", "b_post"):
        assert rel(dict(mhc.named_parameters())[name].grad, ref[name].grad) < 2e-2, name


def sinkhorn_gradient(logits, d, iters):
    """d(logits) of the iterated row and column normalisation, from kept iterates, in the dtype of the arguments."""
    p0 = p = torch.exp(logits - logits.amax((-2, -1), keepdim=True))
    kept = []
    for _ in range(iters):
        for dim in (-1, -2):
            s = p.sum(dim, keepdim=True).clamp(min=1e-9)
            p = p / s
            kept.append((p, s, dim))
    for y, s, dim in reversed(kept):
        d = (d - (d * y).sum(dim, keepdim=True)) / s
    return d * p0


# residual logits that span some 25 and some 70
@pytest.mark.parametrize("spread,mean,tail", [(4, 3.0e-7, 2.5e-6), (12, 6.5e-7, 1.0e-5)])
def test_sinkhorn_gradient_per_token(spread, mean, tail):
    """The gradient is as good as iterates kept in 32 bits give it; iterates rebuilt on the way back are a quarter to a third worse."""
    from q38 import ops
    ops.install()
    T, h, iters, a2 = 65536, 64, 20, 64.0
    gen = torch.Generator(device="cuda").manual_seed(0)
    z = (torch.randn(T, 24, device="cuda", generator=gen) * (spread / a2)).clamp(-0.9, 0.9)
    dcoef = torch.randn(T, 24, device="cuda", generator=gen)
    dcoef[:, :8] = 0
    zeros = lambda *s: torch.zeros(*s, device="cuda")
    alphas = torch.tensor([0.0, 0.0, a2], device="cuda")
    logits, d = (a2 * z[:, 8:]).view(T, 4, 4), dcoef[:, 8:].clone().view(T, 4, 4)
    # with an identity as the second projection and unit norms, dL_raw is d(logits) alphas (1 - z^2) of every token
    dL = ops.load().mhc_pre_bwd_a(zeros(T, h), zeros(T, 4, h), zeros(T, 24), torch.eye(24, device="cuda"), zeros(4), zeros(4), zeros(16), alphas, zeros(h),
                                  zeros(T, 24), z, zeros(T) + 1, zeros(T) + 1, dcoef, iters)[0]
    factor = (a2 * (1 - z[:, 8:].double() ** 2)).view(T, 4, 4)
    ref = sinkhorn_gradient(logits.double(), d.double(), iters) * factor
    err = lambda x: (x.double().view(T, 16) - ref.view(T, 16)).norm(dim=1) / ref.view(T, 16).norm(dim=1)
    good = err(sinkhorn_gradient(logits, d, iters) * factor.float()) < 1e-5       # some tokens' gradients are ill-conditioned in any 32-bit arithmetic
    assert good.float().mean() > 0.999
    got = err(dL[:, 8:])[good]
    # forty divisions of 2^-23 each way and an exponential of 2^-22: with kept iterates 2.6e-7 and 5.8e-7 in the mean, 1.5e-6 and 6.8e-6 for one token in
    # a thousand; with rebuilt ones 3.5e-7 and 7.4e-7, 1.6e-6 and 1.5e-5
    assert got.mean() < mean and got.quantile(0.999) < tail, (got.mean().item(), got.quantile(0.999).item())
