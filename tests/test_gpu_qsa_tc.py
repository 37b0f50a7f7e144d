"""Attention and indexer kernels on the tcgen05 path at the edges of their tiles, against the same sums in 64 bits."""
import pytest
import torch

from test_gpu_qsa_edges import ops, test_block_attention as block_attention, test_indexer_backward as indexer_backward  # noqa: F401
from test_kernel_sources import test_waits_of_whole_warps_are_voted as waits_are_voted

gpu = pytest.mark.gpu


# one and an odd number of heads per group (a half-empty tile of the dQ pass; an odd last (query block, head) pair of the dK / dV pass), one tile, fewer
# tiles than a part has, and key blocks split over several parts of unequal length
@gpu
@pytest.mark.parametrize("B,nb,nq,nkv,pick", [(1, 1, 1, 1, "dense"), (1, 1, 3, 1, "dense"), (2, 9, 11, 1, "gaps"), (1, 21, 10, 2, "dense"), (1, 24, 22, 2, "gaps")])
def test_block_attention_tiles(ops, B, nb, nq, nkv, pick):  # noqa: F811
    block_attention(ops, B, nb, nq, nkv, pick)


# enough query blocks for one CTA each (no slices): a half-empty key tile, one and a half key tiles; heads that do not exist
@gpu
@pytest.mark.parametrize("B,nb,NI", [(150, 1, 4), (50, 3, 3)])
def test_indexer_backward_without_slices(ops, B, nb, NI):  # noqa: F811
    indexer_backward(ops, NI, B, nb)


@pytest.mark.parametrize("name", ["qsa_attn.cu", "qsa_attn_bwd.cu", "qsa_index_bwd.cu"])
def test_waits_of_whole_warps(name):
    waits_are_voted(name)
