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


# 1 and 37 pairs: four CTAs per pair; 38 and 74: two; 75: one; chunk counts below, at and above the three and four pipeline stages
@pytest.mark.parametrize("B,H", [(1, 1), (1, 37), (2, 19), (2, 37), (5, 15)])
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
