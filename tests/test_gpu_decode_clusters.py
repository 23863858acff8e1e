"""Decode attention where the number of CTAs that share a group of heads changes: as many groups as clusters of eight, four
and two CTAs fit the chip at once, for one and for several heads a CTA, and one more."""
import pytest
import torch

import test_gpu_few_rows as few

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads", [1, 4])
@pytest.mark.parametrize("sequences", [15, 16, 33, 34, 71, 72, 74, 75, 148, 149])
def test_groups_around_the_resident_clusters(sequences, heads):
    few.test_decode_attention_shapes(torch.device("cuda:0"), sequences, 1, heads, 1, 64, 9)


def test_a_captured_call_asks_for_the_resident_clusters_too():
    from memory_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(1)
    q = torch.randn(8, 1, 4 * 64, generator=g, device="cuda").bfloat16()
    kv = torch.randn(12 * 64, 2 * 64, generator=g, device="cuda").bfloat16()
    idx = torch.rand(8, 12, generator=g, device="cuda").topk(9, dim=1).indices.int()
    w = torch.rand(8, 9, generator=g, device="cuda")
    want = ops.decode_attn(q, kv, idx, w, 4, 1, 64, 0.125)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = ops.decode_attn(q, kv, idx, w, 4, 1, 64, 0.125)
    out.zero_()
    graph.replay()
    assert torch.equal(out, want)
