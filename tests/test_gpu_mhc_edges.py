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
