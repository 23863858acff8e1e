"""Sparse attention where the rows of a tile are loaded differently: groups of query heads that are boxes of whole swizzle groups
(8 to 128 heads) and ones that are not (24 leave a tile's last rows empty), with tiles that are not full."""
import pytest

import test_gpu_sparse_tc as sparse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [64, 128])
@pytest.mark.parametrize("group", [8, 16, 24, 32, 64, 128])
def test_groups_of_query_heads(group, rows, monkeypatch):
    shape = dict(B=2, TQ=37, M=5, HQ=2 * group, H=2, S=3, BS=rows)
    monkeypatch.setitem(sparse.SHAPES, "group", shape)
    sparse.test_values_gradients_and_repeats("group")
