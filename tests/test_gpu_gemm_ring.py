"""Products whose K blocks are fewer than, as many as and more than the stages of the ring (eight for narrow tiles, four for wide ones)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
@pytest.mark.parametrize("N", [40, 256])
@pytest.mark.parametrize("blocks", [1, 4, 8, 19])
def test_gemm_ring(layout, N, blocks):
    from q38 import ops
    ops.install()
    M, K = 40000 if layout != "tn" else 136, 64 * blocks - 8          # many tiles per SM: the ring runs on from tile to tile; a ragged last block
    gen = torch.Generator(device="cuda").manual_seed(blocks)
    a = torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16)
    b = torch.randn(N, K, device="cuda", generator=gen).to(torch.bfloat16)
    got = ops.gemm(a.t().contiguous() if layout == "tn" else a, b if layout == "nt" else b.t().contiguous(), a_mn_major=layout == "tn", b_mn_major=layout != "nt",
                   out_dtype=torch.float32)
    want = a.double() @ b.double().t()
    # exact bf16 products, fp32 sums of at most 1208 terms in steps of sixteen
    assert (got.double() - want).norm() <= 2e-6 * want.norm()
    assert int(ops.error_flag().item()) == 0
