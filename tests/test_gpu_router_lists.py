"""Token routing with lists on both sides of the 32 entries that one warp finishes, with and without shared chapters, chapter
counts that end in the middle of a thread's columns, and more ties than that warp takes."""
import pytest
import torch

import test_gpu_few_rows as few

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows, chapters, k, shared", [(592, 4352, 32, 0), (600, 4351, 32, 1), (600, 4097, 31, 1), (592, 257, 1, 0),
                                                       (136, 2049, 33, 0), (608, 4607, 16, 0), (600, 4609, 128, 0)])
def test_list_lengths(rows, chapters, k, shared):
    few.test_token_router_shapes(torch.device("cuda:0"), rows, chapters, 64, k, shared)


@pytest.mark.parametrize("k, shared, distinct", [(16, 0, 5), (32, 0, 40), (17, 2, 5), (40, 0, 5)])
def test_more_ties_than_candidates(k, shared, distinct):
    """Weight rows that are equal give equal probabilities, bit for bit: of them the lowest ids are taken, in ascending order."""
    import memory_b200 as M
    torch.manual_seed(k)
    rows, chapters, d = 600, 3000, 64
    h = torch.randn(1, rows, d, device="cuda").bfloat16()
    w = (torch.randn(1, d, device="cuda") * 0.05).expand(chapters, d).contiguous()
    w[:distinct] = torch.randn(distinct, d, device="cuda") * 0.05
    idx, wt, _ = M.route_tokens(h, w, None, k, shared, False)
    idx = idx[0].cpu()
    for row in idx.tolist():
        tied = [c for c in row if c >= distinct]
        first = max(shared, distinct)
        assert tied == list(range(first, first + len(tied)))
        assert len(set(row)) == k and min(row) >= shared
    assert (wt[0].sum(1) - 1).abs().max() < 1e-5             # k fp32 quotients of one sum
