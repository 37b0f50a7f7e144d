"""Attention and indexer kernels on the tcgen05 path at the edges of their tiles, against the same sums in 64 bits."""
import pytest
import torch

from test_gpu_kernels import test_first_query_indexer_log_probabilities as first_query
from test_gpu_qsa_edges import ops, test_block_attention as block_attention, test_indexer_backward as indexer_backward  # noqa: F401
from test_kernel_sources import test_waits_of_whole_warps_are_voted as waits_are_voted

gpu = pytest.mark.gpu


# one and an odd number of heads per group (a half-empty tile of the dQ pass; an odd last (query block, head) pair of the dK / dV pass), one tile, fewer
# tiles than a part has, and key blocks split over several parts of unequal length
@gpu
@pytest.mark.parametrize("B,nb,nq,nkv,pick", [(1, 1, 1, 1, "dense"), (1, 1, 3, 1, "dense"), (2, 9, 11, 1, "gaps"), (1, 21, 10, 2, "dense"), (1, 24, 22, 2, "gaps")])
def test_block_attention_tiles(ops, B, nb, nq, nkv, pick):  # noqa: F811
    block_attention(ops, B, nb, nq, nkv, pick)


# one, three, fifteen and sixteen tiles per part, the latter in as many parts as allowed and in fewer
@gpu
@pytest.mark.parametrize("B,nb,nq,nkv", [(1, 4, 16, 2), (1, 8, 22, 2), (1, 19, 24, 2), (1, 20, 24, 2), (4, 20, 20, 2)])
def test_block_attention_parts(ops, B, nb, nq, nkv):  # noqa: F811
    block_attention(ops, B, nb, nq, nkv, "dense")


# enough query blocks for one CTA each (no slices): a half-empty key tile, one and a half key tiles; heads that do not exist
@gpu
@pytest.mark.parametrize("B,nb,NI", [(150, 1, 4), (50, 3, 3)])
def test_indexer_backward_without_slices(ops, B, nb, NI):  # noqa: F811
    indexer_backward(ops, NI, B, nb)


# half a query tile, an odd last one, a CTA for every key block and for two; several blocks per CTA; fewer heads than the kernel holds
@gpu
@pytest.mark.parametrize("B,nb,NI", [(1, 1, 4), (2, 3, 1), (1, 16, 4), (1, 21, 3), (12, 21, 4)])
def test_indexer_forward(ops, B, nb, NI):  # noqa: F811
    S = 64 * nb
    gen = torch.Generator(device="cuda").manual_seed(nb)
    qi = torch.randn(B, NI, S, 64, device="cuda", generator=gen).to(torch.bfloat16)
    ki = torch.randn(B, S, 64, device="cuda", generator=gen).to(torch.bfloat16)
    wi = torch.randn(B, S, NI, device="cuda", generator=gen) / 2
    blse = ops.load().qsa_indexer_fwd(qi, ki, wi, 0.125).double()
    causal = torch.ones(S, S, dtype=torch.bool, device="cuda").tril()
    dots = (qi.double() @ ki.double()[:, None].transpose(-1, -2)).to(torch.bfloat16).double()
    score = (torch.relu(dots) * 0.125 * wi.double().transpose(1, 2)[..., None]).sum(1).masked_fill(~causal, float("-inf"))
    want = score.unflatten(-1, (nb, 64)).logsumexp(-1)
    own = (torch.arange(S, device="cuda")[:, None] // 64 >= torch.arange(nb, device="cuda")[None]).expand_as(want)
    assert (blse[~own] == -1e9).all()
    # fp32 sums; a product that lies on a rounding boundary of bf16 may fall to the other side: 2^-8 of |q.k| <= 40, times scale and |w| <= 2
    assert (blse - want)[own].abs().max() < 2 ** -8 * 40 * 0.125 * 2
    assert (blse - want)[own].pow(2).mean().sqrt() < 1e-3


@pytest.mark.parametrize("name", ["qsa_attn.cu", "qsa_attn_bwd.cu", "qsa_index_fwd.cu", "qsa_index_bwd.cu"])
def test_waits_of_whole_warps(name):
    waits_are_voted(name)


@gpu
@pytest.mark.parametrize("nkv", [1, 2])
def test_values_as_a_transposed_view(ops, nkv):  # noqa: F811
    """Values may be the transposed view of a projection's output: the same results, and their gradient in that layout."""
    B, nq, S = 2, 4, 192
    gen = torch.Generator(device="cuda").manual_seed(nkv)
    q, k, do = (torch.randn(s, device="cuda", generator=gen).to(torch.bfloat16) for s in ((B, nq, S, 64), (B, nkv, S, 64), (B, S, nq, 64)))
    v = torch.randn(B, S, nkv, 64, device="cuda", generator=gen).to(torch.bfloat16).transpose(1, 2)
    lib = ops.load()
    results = []
    for values in (v, v.contiguous()):
        o, lse, sel = lib.qsa_attn_fwd(q, k, values, None, None, 0.125)
        results.append((o, lse, *lib.qsa_attn_bwd(q, k, values, o, do, lse, sel, 0.125)))
    assert results[0][4].stride() == v.stride()
    for i, (a, b) in enumerate(zip(*results)):
        # key and value gradients: fp32 sums whose order varies, rounded to bf16 once
        assert torch.equal(a, b) if i < 3 else ((a.float() - b.float()).norm() <= 4e-3 * b.float().norm())
    with pytest.raises(RuntimeError, match="contiguous bf16"):
        lib.qsa_attn_fwd(q, k, v.expand(B, nkv, S, 64)[..., ::1].transpose(2, 3).contiguous().transpose(2, 3), None, None, 0.125)


def block_stats(ops, q, k):  # noqa: F811
    stats = ops.load().qsa_block_stats_tc(q, k, 0.125, ops.error_flag()).double()
    return stats[..., 0], stats[..., 1]


@gpu
@pytest.mark.parametrize("at", range(8))
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_block_statistics_show_a_bad_key(ops, at, bad):  # noqa: F811
    """Full blocks take two of every eight exponentials through a polynomial: a key whose scores are NaN or infinite shows in the sum wherever it stands."""
    gen = torch.Generator(device="cuda").manual_seed(at)
    q, k = (torch.randn(1, h, 256, 64, device="cuda", generator=gen).to(torch.bfloat16) for h in (2, 1))
    k[0, 0, 8 * at + at] = bad
    m, total = block_stats(ops, q, k)
    assert not total[0, :, 64:, 0].isfinite().any() and not total[0, :, 8 * at + at:64, 0].isfinite().any()
    assert total[0, :, 192:, 1:3].isfinite().all()


@gpu
@pytest.mark.parametrize("alone", [False, True])
def test_block_statistics_accuracy(ops, alone):  # noqa: F811
    """Against 64 bits, with all keys and with the sums left to the keys that go through the polynomial (`alone`: the others score 60 lower)."""
    gen = torch.Generator(device="cuda").manual_seed(7)
    q, k = (torch.randn(1, h, 1024, 64, device="cuda", generator=gen).to(torch.bfloat16) for h in (4, 1))
    if alone:
        q[..., 0], k[..., 0] = 8, 0
        k.view(1, 1, 128, 8, 64)[:, :, :, :6, 0] = -60
    m, total = block_stats(ops, q, k)
    score = (q.double() @ k.double().transpose(-1, -2) / 8).unflatten(-1, (16, 64))
    full = torch.arange(1024, device="cuda")[:, None] // 64 > torch.arange(16, device="cuda")[None]
    err = ((m + total.log()) - score.logsumexp(-1))[:, :, full].abs()
    # fp32 throughout: 64 products of at most 500 in all (2^-24 each), an argument of the exponential of at most 200 (2^-24), an exponential of 2^-21
    assert err.max() < 500 / 8 * 2 ** -23 + 200 * 2 ** -24 + 2 ** -21


@gpu
@pytest.mark.parametrize("block", [0, 1, 2, 3])
def test_indexer_backward_keeps_a_nan_in_its_blocks(ops, block):  # noqa: F811
    """Key tiles hold two blocks.  A key that is not finite reaches the gradients of no earlier query block, a query none of later keys."""
    gen = torch.Generator(device="cuda").manual_seed(block)
    qi, ki = (torch.randn(s, device="cuda", generator=gen).to(torch.bfloat16) for s in ((1, 4, 320, 64), (1, 320, 64)))
    wi, dblse = torch.randn(1, 320, 4, device="cuda", generator=gen), torch.randn(1, 320, 5, device="cuda", generator=gen)
    lib, later = ops.load(), slice(64 * block + 64, None)
    clean = lib.qsa_indexer_bwd(qi, ki, wi, lib.qsa_indexer_fwd(qi, ki, wi, 0.125), dblse, 1.0, 0.125)
    for bad in (float("nan"), float("inf")):
        k = ki.clone()
        k[:, later] = bad
        dq, _, dw = lib.qsa_indexer_bwd(qi, k, wi, lib.qsa_indexer_fwd(qi, k, wi, 0.125), dblse, 1.0, 0.125)
        assert torch.equal(dq[:, :, :64 * block + 64], clean[0][:, :, :64 * block + 64]) and torch.equal(dw[:, :64 * block + 64], clean[2][:, :64 * block + 64])
        q = qi.clone()
        q[:, :, :64 * block + 64] = bad
        dk = lib.qsa_indexer_bwd(q, ki, wi, lib.qsa_indexer_fwd(q, ki, wi, 0.125), dblse, 1.0, 0.125)[1]
        # fp32 sums whose order varies, rounded to bf16 once
        assert (dk[:, later].float() - clean[1][:, later].float()).norm() <= 4e-3 * clean[1][:, later].float().norm()


@gpu
@pytest.mark.parametrize("B,nb", [(1, 1), (1, 21), (4, 64)])
def test_indexer_weight_gradient_sees_more_than_bf16(ops, B, nb):  # noqa: F811
    """dw = scale sum_s dI relu(q.k) against 64 bits, with the scores inside dI rounded to bf16 as the kernels do.  dI enters with sixteen bits: 2^-17 per term,
    2^-20 from the exponential's argument, and where a score falls to the other side of a rounding boundary 2^-8 of it, once in ten thousand: 2^-13 in
    all.  (dI in one bf16: 5e-4.)"""
    S = 64 * nb
    gen = torch.Generator(device="cuda").manual_seed(nb)
    qi, ki = (torch.randn(s, device="cuda", generator=gen).to(torch.bfloat16) for s in ((B, 4, S, 64), (B, S, 64)))
    wi, dblse = torch.randn(B, S, 4, device="cuda", generator=gen) / 2, torch.randn(B, S, nb, device="cuda", generator=gen)
    lib = ops.load()
    dw = lib.qsa_indexer_bwd(qi, ki, wi, lib.qsa_indexer_fwd(qi, ki, wi, 0.125), dblse, 1.0, 0.125)[2].double()
    want = torch.zeros_like(dw)
    for b in range(B):
        for t0 in range(0, S, 512):
            t1 = min(S, t0 + 512)
            dots = torch.relu(qi[b, :, t0:t1].double() @ ki[b, :t1].double().t())
            hide = torch.arange(t1, device="cuda")[None] > torch.arange(t0, t1, device="cuda")[:, None]
            score = (dots.to(torch.bfloat16).double() * 0.125 * wi[b, t0:t1].double().t()[..., None]).sum(0).masked_fill(hide, float("-inf"))
            spread = lambda t: t.repeat_interleave(64, -1)
            dI = torch.where(hide, 0.0, torch.exp(score - spread(score.unflatten(-1, (-1, 64)).logsumexp(-1))) * spread(dblse[b, t0:t1, :(t1 + 63) // 64].double()))
            want[b, t0:t1] = (dI * dots).sum(-1).t() * 0.125
    assert (dw - want).norm() <= 2 ** -13 * want.norm()


# one, two and four queries per CTA, the last CTA of the latter two with one query
@gpu
@pytest.mark.parametrize("B,nb,NI", [(1, 1, 4), (1, 17, 3), (1, 37, 4), (3, 41, 2)])
def test_first_query_grids(ops, B, nb, NI):  # noqa: F811
    first_query(ops, B, 64 * nb, NI)


@gpu
@pytest.mark.parametrize("nb,nq,nkv,pick", [(1, 1, 1, "dense"), (3, 5, 1, "dense"), (9, 11, 1, "gaps"), (37, 4, 1, "dense")])
@pytest.mark.parametrize("tokens", [False, True])
def test_block_attention_is_the_same_on_both_kernels(ops, nb, nq, nkv, pick, tokens):  # noqa: F811
    """Up to one CTA per SM the warp-MMA kernel runs, above it the tensor-memory one: a sequence alone, and among copies that make the grid large, gives the
    same bits.  Values as a transposed view too."""
    S, copies = 64 * nb, 150
    gen = torch.Generator(device="cuda").manual_seed(nb)
    q, k, v = (torch.randn(1, h, S, 64, device="cuda", generator=gen).to(torch.bfloat16) for h in (nq, nkv, nkv))
    count = index = None
    if pick == "gaps":
        index = torch.tensor([[j for j in range(nb) if j <= i and (i - j) % 3 == 0][::-1] + [0] * (i - i // 3 + nb - 1 - i) for i in range(nb)], dtype=torch.int32, device="cuda")[None]
        count = torch.tensor([[i // 3 + 1 for i in range(nb)]], dtype=torch.int32, device="cuda")
    lay = lambda t: t.transpose(1, 2).contiguous().transpose(1, 2) if tokens else t
    many = lambda t: None if t is None else t.expand(copies, *t.shape[1:]).contiguous()
    alone = ops.load().qsa_attn_fwd(q, k, lay(v), count, index, 0.125)
    among = ops.load().qsa_attn_fwd(many(q), many(k), lay(many(v)), many(count), many(index), 0.125)
    for a, b in zip(alone, among):
        assert torch.equal(a[0], b[0]) and torch.equal(a[0], b[copies - 1])


@gpu
@pytest.mark.parametrize("B", [1, 150])
def test_block_attention_refuses_unaligned_operands(ops, B):  # noqa: F811
    flat = torch.randn(B * 64 * 64 + 1, device="cuda").to(torch.bfloat16)
    q, odd = flat[:-1].view(B, 1, 64, 64), flat[1:].view(B, 1, 64, 64)
    for operands in ((odd, q, q), (q, odd, q), (q, q, odd)):
        with pytest.raises(RuntimeError):
            ops.load().qsa_attn_fwd(*operands, None, None, 0.125)


@gpu
@pytest.mark.parametrize("copies", [1, 60])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("where", ["query", "key", "value", "upstream"])
def test_block_attention_keeps_bad_values_to_what_they_reach(ops, copies, bad, where):  # noqa: F811
    """One element that is not finite, on both forward kernels (grids below and above one CTA per SM): what does not depend on it keeps its bits, although
    tiles hold two heads, accumulators two gradients and blocks masked positions; what does shows it."""
    B, nq, nkv, S, at = copies, 5, 1, 192, 70
    gen = torch.Generator(device="cuda").manual_seed(3)
    clean = {n: torch.randn(s, device="cuda", generator=gen).to(torch.bfloat16)
             for n, s in dict(query=(B, nq, S, 64), key=(B, nkv, S, 64), value=(B, nkv, S, 64), upstream=(B, S, nq, 64)).items()}
    dirty = dict(clean, **{where: clean[where].clone()})
    if where == "upstream":
        dirty[where][0, at, 1, 5] = bad
    else:
        dirty[where][0, 1 if where == "query" else 0, at, 5] = bad
    results = []
    for t in (clean, dirty):
        o, lse, sel = ops.load().qsa_attn_fwd(t["query"], t["key"], t["value"], None, None, 0.125)
        results.append((o, *ops.load().qsa_attn_bwd(t["query"], t["key"], t["value"], o, t["upstream"], lse, sel, 0.125)))
    (o, dq, dk, dv), (o2, dq2, dk2, dv2) = results
    one_row = where in ("query", "upstream")                             # else all heads' rows from the key's block on (hidden positions of it weigh zero times the bad value)
    touched = torch.zeros(B, nq, S, dtype=torch.bool, device="cuda")
    touched[0, 1 if one_row else slice(None), at if one_row else slice(at // 64 * 64, None)] = True
    if where != "upstream":
        assert torch.equal(o.transpose(1, 2)[~touched], o2.transpose(1, 2)[~touched]) and not o2[0, at, 1].isfinite().all()
    else:
        assert torch.equal(o, o2)
    assert torch.equal(dq[~touched], dq2[~touched]) and not dq2[0, 1, at].isfinite().all()
    last = (at // 64 + 1) * 64 if one_row else S                         # keys after the query's block get nothing from it
    for a, b in ((dk, dk2), (dv, dv2)):
        if copies > 1:
            assert (a[1:].float() - b[1:].float()).norm() <= 4e-3 * a[1:].float().norm()
        if last < S:
            assert (a[0, :, last:].float() - b[0, :, last:].float()).norm() <= 4e-3 * a[0, :, last:].float().norm()
    assert not dk2[0].isfinite().all()
