"""The kernels' own arithmetic over its whole range, against what it stands in for."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def test_polynomial_exponential():
    from memory_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(1)
    x = torch.cat([torch.empty(1 << 22, device=DEV).uniform_(-126, 12, generator=g),
                   torch.empty(1 << 20, device=DEV).uniform_(-1, 1, generator=g),
                   torch.arange(-126, 13, device=DEV).float(), torch.arange(-251, 25, device=DEV).float() / 2,
                   torch.zeros(1, device=DEV)])
    y, want = ops.exp2_probe(x).double(), x.double().exp2()
    # 2.1e-7 is the polynomial's own error; six fp32 roundings, the last two at full weight, add up to 1e-7
    assert float(((y - want) / want)[x >= -125.5].abs().max()) < 3.2e-7
    assert float((y - want)[x < -125.5].abs().max()) < 2.0 ** -126        # (the exponential unit flushes these to zero)
    small = torch.cat([torch.empty(1 << 16, device=DEV).uniform_(-300, -126, generator=g),
                       torch.tensor([-126.5, -127.0, -127.5, -1e4, -3e38, -math.inf], device=DEV)])
    y = ops.exp2_probe(small)
    assert float(y.min()) >= 0.0 and float(y.max()) <= 2.0 ** -126
    assert float(y[small <= -127].max()) <= 2.0 ** -149 and not y.bfloat16()[small <= -127].any()


def test_a_nan_score_makes_its_row_nan_in_every_column():
    from memory_b200 import _lib as L, ops
    g = torch.Generator(device=DEV).manual_seed(2)
    n_sel, heads = 128, 2
    q = torch.randn(n_sel, 5, heads * 64, generator=g, device=DEV).bfloat16()
    kv = torch.randn(n_sel, n_sel, 2 * heads * 64, generator=g, device=DEV).bfloat16()
    for i in range(n_sel):
        kv[i, i, 3] = math.nan                         # one key of head 0, another one in every item
    o, lse = ops.attn_fwd(q, kv, heads, heads, 0.125)
    L.check_device_status(o.device)
    assert o[..., :64].isnan().all() and lse[:, 0].isnan().all()
    assert o[..., 64:].isfinite().all() and lse[:, 1].isfinite().all()


def test_an_infinite_score_makes_its_row_nan_in_every_column():
    """Infinity against itself, wherever it stands; minus infinity is a key of no weight unless it comes first."""
    from memory_b200 import _lib as L, ops
    n_sel = 1024
    q = torch.ones(n_sel, 3, 64, device=DEV).bfloat16()
    kv = torch.randn(n_sel, n_sel, 128, generator=torch.Generator(device=DEV).manual_seed(6), device=DEV).bfloat16()
    up, down = kv.clone(), kv.clone()
    for i in range(n_sel):
        up[i, i, 5] = math.inf
        down[i, i, 5] = -math.inf
    o, lse = ops.attn_fwd(q, up, 1, 1, 0.125)
    assert o.isnan().all() and lse.isnan().all()
    o, lse = ops.attn_fwd(q, down, 1, 1, 0.125)
    for i in range(0, n_sel, 37):              # alone, an item's key range is shared by a cluster
        alone, alone_lse = ops.attn_fwd(q[i:i + 1], up[i:i + 1], 1, 1, 0.125)
        assert alone.isnan().all() and alone_lse.isnan().all()
    L.check_device_status(o.device)
    ref = torch.softmax((q.double() @ down[..., :64].double().transpose(1, 2)) * 0.125, -1) @ down[..., 64:].double()
    assert float((o.double() - ref).norm() / ref.norm()) < 5e-3 and lse.isfinite().all()


@pytest.mark.parametrize("n_sel", [70, 97, 200])
def test_columns_past_the_end_add_nothing(n_sel):
    """What lies behind an item's last key is the next item's, whatever its size."""
    from memory_b200 import _lib as L, ops
    g = torch.Generator(device=DEV).manual_seed(3)
    q = torch.randn(2, 40, 64, generator=g, device=DEV).bfloat16()
    kv = torch.randn(2, n_sel, 128, generator=g, device=DEV).bfloat16()
    want, want_lse = ops.attn_fwd(q[:1].contiguous(), kv[:1].contiguous(), 1, 1, 0.125)
    kv[1, :, 64:] = 1e38
    o, lse = ops.attn_fwd(q, kv, 1, 1, 0.125)
    L.check_device_status(o.device)
    assert torch.equal(o[:1], want) and torch.equal(lse[:1], want_lse)


def test_router_quotient_is_the_division():
    """Exponentials from 1 down to 2^-100, over sums from the floor of a masked row to a few thousand."""
    from memory_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(4)
    n = 1 << 24
    x = torch.empty(n, device=DEV).uniform_(1, 2, generator=g) * torch.empty(n, device=DEV).uniform_(-100, 0, generator=g).exp2()
    x[: n // 8] = torch.empty(n // 8, device=DEV).uniform_(2.0 ** -20, 1, generator=g)
    d = torch.empty(n, device=DEV).uniform_(-40, 14, generator=g).exp2()
    # (divisors that are all ones but for the last bits are the hard ones for a corrected reciprocal)
    d[::3] = (d[::3].view(torch.int32) | 0x7FFFF8).view(torch.float32)
    x[:3], d[:3] = torch.tensor([0.0, 1.0, 2.0 ** -100], device=DEV), torch.tensor([3.0, 3.0, 7.0], device=DEV)
    want = (x.double() / d.double()).float()         # (all normal numbers: twice rounded is once rounded)
    got = ops.quotient_probe(x, d)
    assert torch.equal(got, want), float((got != want).float().mean())
    assert ops.quotient_probe(torch.tensor([math.nan], device=DEV), torch.ones(1, device=DEV)).isnan().all()


@pytest.mark.parametrize("rows", [2, 4096])
@pytest.mark.parametrize("chapters", [200, 1025, 2000, 4097, 5000, 8193, 9000])
def test_router_probabilities_of_rows_with_a_wide_range_are_divided(rows, chapters):
    """Two rows with the same tiny rest under one large value and under two.  The first row's sum is 1, so its
    probabilities are the exponentials themselves; the second's must be those divided by its sum, to the last bit."""
    from memory_b200 import _lib as L, ops
    g = torch.Generator(device=DEV).manual_seed(chapters)
    logits = torch.empty(chapters, device=DEV).uniform_(-104, -30, generator=g).repeat(rows, 1)
    logits[:, 0], logits[0::2, 1], logits[1::2, 1] = 0.0, -104.0, -0.3
    total = 1.0 + torch.full((1,), -0.3, device=DEV).exp()
    h = torch.zeros(rows, 1, 8, device=DEV)
    r = ops.router_fwd(h, torch.zeros(chapters, 8, device=DEV), None, 4, 1, 1.0, False, pooled=h.view(rows, 8), logits=logits)
    L.check_device_status(h.device)
    e, p = r["probs"][0].cpu().numpy(), r["probs"].cpu().numpy()
    assert e[2:].min() < 1e-44 and e[0] == 1.0
    for row in (1, rows - 1):
        assert p[row, 0] == 1.0 / total.cpu().numpy()[0]
        assert (p[row, 2:] == e[2:] / total.cpu().numpy()[0]).all()


@pytest.mark.parametrize("block", [64, 128])
def test_a_nan_query_stays_nan_in_the_sparse_attention(block):
    """Every listed block of such a token has a NaN sum; a token none of whose blocks exists still gets zeros."""
    import memory_b200 as M
    from memory_b200 import _lib as L
    g = torch.Generator(device=DEV).manual_seed(5)
    q = torch.randn(1, 20, 4, 64, generator=g, device=DEV).bfloat16()
    k, v = (torch.randn(1, 6 * block, 2, 64, generator=g, device=DEV).bfloat16() for _ in range(2))
    bi = torch.rand(40, 6, generator=g, device=DEV).topk(3, dim=1).indices.view(1, 20, 2, 3).int()
    want, want_lse = M.memory_cross_attn_forward(q, k, v, bi, block)
    q[0, 7, 2], bi[0, 11] = math.nan, 6
    o, lse = M.memory_cross_attn_forward(q, k, v, bi, block)
    with pytest.raises(RuntimeError, match="out of range"):
        L.check_device_status(o.device)
    assert o[0, 7, 2].isnan().all() and lse[0, 7, 2].isnan()
    assert not o[0, 11].any() and (lse[0, 11] == -math.inf).all()
    rest = torch.ones(20, 4, dtype=torch.bool, device=DEV)
    rest[7, 2], rest[11] = False, False
    assert torch.equal(o[0][rest], want[0][rest]) and torch.equal(lse[0][rest], want_lse[0][rest])
