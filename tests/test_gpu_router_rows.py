"""Token routing over banks of eight thousand chapters: on both sides of the line up to which many rows are selected by CTAs of
256 threads, and at the next power of two with a shared chapter."""
import pytest
import torch

import test_gpu_few_rows as few

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows, chapters, d, k, shared", [(600, 8193, 72, 16, 1), (592, 8448, 64, 5, 0), (600, 8449, 64, 300, 1),
                                                          (584, 8448, 64, 5, 1)])
def test_many_rows_of_large_banks(rows, chapters, d, k, shared):
    few.test_token_router_shapes(torch.device("cuda:0"), rows, chapters, d, k, shared)
