"""Row kernels of the expert block, the head preparation and the loss at the edges of their pieces, against PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    from q38 import ops
    ops.install()
    return ops.load()


# one pair, one block of 1024 pairs and one more, enough blocks that the scan's sixteen segments hold one and two of them
@pytest.mark.parametrize("T,k,E", [(1, 1, 1), (1024, 1, 3), (205, 5, 64), (16 * 1024, 1, 64), (4 * 1024 + 1, 4, 7)])
def test_sort_and_row_sums(lib, T, k, E):
    gen = torch.Generator(device="cuda").manual_seed(T)
    top = torch.randint(0, E, (T, k), device="cuda", generator=gen, dtype=torch.int32)
    perm, inv, offsets, sched = lib.moe_sort(top, E, None)
    order = torch.sort(top.flatten().long(), stable=True).indices
    assert torch.equal(perm.long(), order) and torch.equal(inv.long()[order], torch.arange(T * k, device="cuda"))
    counts = torch.bincount(top.flatten().long(), minlength=E)
    assert torch.equal(offsets.long(), torch.cat([counts.new_zeros(1), counts.cumsum(0)]))
    tiles = [(e, int(offsets[e]) + r, min(128, int(counts[e]) - r)) for e in range(E) for r in range(0, int(counts[e]), 128)]
    got = sched[1:].view(-1, 3)
    assert int(sched[0]) == len(tiles) and got[:len(tiles)].tolist() == [list(t) for t in tiles] and not got[len(tiles):, 2].any()
    for h in (8, 36, 264):                                     # one 16-byte piece, no whole pieces, more pieces than a warp
        rows = torch.randn(T * k, h, device="cuda", generator=gen).to(torch.bfloat16)
        w = torch.rand(T, k, device="cuda", generator=gen)
        pairs = rows[inv.long()].view(T, k, h)
        want, plain = torch.zeros(T, h, device="cuda"), torch.zeros(T, h, device="cuda")
        for j in range(k):                                     # slot order, each weighted row rounded to bf16 first
            want += (pairs[:, j].float() * w[:, j, None]).to(torch.bfloat16).float()
            plain += pairs[:, j].float()
        assert torch.equal(lib.moe_combine_fwd(rows, inv, w), want.to(torch.bfloat16))
        assert torch.equal(lib.moe_unpermute_sum(rows, inv, T, k), plain.to(torch.bfloat16))


# one CTA of eight tokens, a ragged second one, more CTAs than fit the chip at once
@pytest.mark.parametrize("T,E,k", [(1, 1, 1), (9, 64, 8), (16384, 64, 5), (5000, 33, 2)])
def test_router_sums(lib, T, E, k):
    gen = torch.Generator(device="cuda").manual_seed(T)
    logits = (2 * torch.randn(T, E, device="cuda", generator=gen)).to(torch.bfloat16)
    _, idx, probs, counts, prob_sum = lib.moe_route_fwd(logits, k)
    assert torch.equal(counts, torch.bincount(idx.flatten().long(), minlength=E).float())
    want = logits.double().softmax(-1)
    # an approximate exponential and quotient (2^-21); a sum has seven roundings within a CTA, 2^-37 per CTA and one rounding at the end
    assert ((probs.double() - want).norm() / want.norm()).item() < 1e-6
    assert ((prob_sum.double() - probs.double().sum(0)).norm() / want.sum(0).norm()).item() < 3e-7
    for _ in range(20):
        again = lib.moe_route_fwd(logits, k)
        assert torch.equal(again[4], prob_sum) and torch.equal(again[3], counts)
    logits[T // 2, 0] = float("nan")
    assert lib.moe_route_fwd(logits, k)[4].isnan().all()
    empty = lib.moe_route_fwd(logits[:0], k)
    assert not empty[3].any() and not empty[4].any()


def test_row_sums_of_empty_rows(lib):
    top = torch.tensor([[0, 1], [1, 0]], device="cuda", dtype=torch.int32)
    inv = lib.moe_sort(top, 2, None)[1]
    rows = torch.zeros(4, 0, device="cuda", dtype=torch.bfloat16)
    assert lib.moe_combine_fwd(rows, inv, torch.ones(2, 2, device="cuda")).shape == (2, 0)
    assert lib.moe_unpermute_sum(rows, inv, 2, 2).shape == (2, 0)


@pytest.mark.parametrize("B,S,H", [(1, 1, 1), (2, 3, 5), (1, 1000, 2)])
def test_rotary_with_rounded_products(lib, B, S, H):
    from q38.models import modeling
    gen = torch.Generator(device="cuda").manual_seed(S)
    x = torch.randn(B, S, H, 64, device="cuda", generator=gen).to(torch.bfloat16)
    cos, sin = modeling.rope_tables(torch.arange(S, device="cuda")[None], 16, 1e7, torch.float32)
    out = lib.qsa_headprep_fwd(x, None, cos, sin, 0.0, False, True)[0]
    assert torch.equal(out, modeling.apply_rope(x.transpose(1, 2), cos, sin))
    shifted = torch.empty(x.numel() + 1, device="cuda", dtype=torch.bfloat16)[1:].view_as(x).copy_(x)      # contiguous, but not on 16 bytes
    assert torch.equal(lib.qsa_headprep_fwd(shifted, None, cos, sin, 0.0, False, True)[0], out)


@pytest.mark.parametrize("n", [8, 2048, 2056])
def test_scale(lib, n):
    from q38.ops.backend import scale_bf16
    x = torch.randn(n, device="cuda").to(torch.bfloat16)
    f = torch.tensor(0.37, device="cuda").to(torch.bfloat16)
    assert torch.equal(scale_bf16(x, f), x * f) and torch.equal(scale_bf16(x[1:], f), x[1:] * f)


@pytest.mark.parametrize("rows", [0, 1, 8192, 8193])
def test_loss_over_chunk_edges(lib, rows):
    from q38.models import modeling
    V, h = 128, 64
    gen = torch.Generator(device="cuda").manual_seed(rows)
    hid = torch.randn(rows, h, device="cuda", generator=gen).to(torch.bfloat16).requires_grad_()
    w = (torch.randn(V, h, device="cuda", generator=gen) / 4).requires_grad_()
    tgt = torch.randint(0, V, (rows,), device="cuda", generator=gen)
    loss = modeling.get_backend().linear_cross_entropy(w, hid, tgt, "sum")
    loss.backward()
    hr, wr = hid.detach().double().requires_grad_(), w.detach().to(torch.bfloat16).double().requires_grad_()
    ref = torch.nn.functional.cross_entropy(hr @ wr.t(), tgt, reduction="sum")
    ref.backward()
    assert hid.grad.shape == hid.shape
    if rows:
        # logits of rms 2 rounded to bf16 (3e-3, so the probabilities move by 0.3 %), then their bf16 gradients and the bf16 outputs (2e-3 rms each)
        rel = lambda a, b: ((a.double() - b).norm() / b.norm()).item()
        assert abs(loss.item() - ref.item()) < 5e-3 * abs(ref.item()) + 5e-2 and rel(hid.grad, hr.grad) < 2e-2 and rel(w.grad, wr.grad) < 2e-2


@pytest.mark.parametrize("E,k", [(8, 2), (32, 5), (64, 5)])
def test_routing_of_rows_without_probabilities(lib, E, k):
    """A NaN or +infinity among a row's logits, or nothing above -infinity: all slots name expert 0 with weight NaN, and other rows are as they were."""
    gen = torch.Generator(device="cuda").manual_seed(E)
    logits = torch.randn(77, E, device="cuda", generator=gen).to(torch.bfloat16)
    want = lib.moe_route_fwd(logits, k)
    bad = torch.tensor([0, 9, 40, 76], device="cuda")
    logits[0, E - 1], logits[9], logits[40, 3], logits[76] = float("nan"), float("nan"), float("inf"), float("-inf")
    top_w, top_idx, probs, counts, prob_sum = lib.moe_route_fwd(logits, k)
    good = torch.ones(77, dtype=torch.bool, device="cuda")
    good[bad] = False
    assert (top_idx[bad] == 0).all() and top_w[bad].isnan().all() and probs[bad].isnan().all() and prob_sum.isnan().all()
    assert torch.equal(top_idx[good], want[1][good]) and torch.equal(top_w[good], want[0][good])
    assert torch.equal(counts, torch.bincount(top_idx.flatten(), minlength=E).float())


# CTAs of one, two, three and four rounds of eight tokens, with a last round that is not full
@pytest.mark.parametrize("T", [1, 9, 2360, 2361, 3546, 4733])
def test_routing_over_its_grids(lib, T):
    gen = torch.Generator(device="cuda").manual_seed(T)
    logits = torch.randn(T, 64, device="cuda", generator=gen).to(torch.bfloat16)
    top_w, top_idx, probs, counts, prob_sum = lib.moe_route_fwd(logits, 5)
    want = logits.double().softmax(-1)
    # fp32: an exponential of 2^-21, a sum and a division
    assert ((probs - want).abs() <= 2 ** -19 * want).all()
    best = probs.topk(5, -1).values
    assert torch.equal(probs.gather(1, top_idx.long()), best) and (top_idx.sort(-1).values.diff(dim=-1) > 0).all()
    assert torch.equal(counts, torch.bincount(top_idx.flatten(), minlength=64).float())
    # sums of eight tokens in fp32, rounded to multiples of 2^-36, and one rounding at the end
    assert ((prob_sum - probs.double().sum(0)).abs() <= 2 ** -21 * probs.double().sum(0)).all()


# whole and half warps per pair (few pairs, the last and the first count on either side; rows that fill a warp), one piece, no whole pieces
@pytest.mark.parametrize("T,k", [(1, 1), (473, 5), (474, 5), (2000, 2)])
@pytest.mark.parametrize("h", [8, 36, 264, 448, 512])
def test_combine_backward(lib, T, k, h):
    gen = torch.Generator(device="cuda").manual_seed(T + h)
    inv = torch.randperm(T * k, device="cuda", generator=gen).to(torch.int32)
    y, dout = (torch.randn(n, h, device="cuda", generator=gen).to(torch.bfloat16) for n in (T * k, T))
    w = torch.rand(T, k, device="cuda", generator=gen)
    dy, dw = lib.moe_combine_bwd(dout, y, inv, w)
    spread = dout.float().repeat_interleave(k, 0)
    assert torch.equal(dy[inv.long()], (spread * w.view(-1, 1)).to(torch.bfloat16))
    want = (spread.double() * y[inv.long()].double())
    # fp32 sums of h products in some order
    assert ((dw.flatten() - want.sum(-1)).abs() <= h * 2 ** -24 * want.abs().sum(-1) + 1e-30).all()
