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
