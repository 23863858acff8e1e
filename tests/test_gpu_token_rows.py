"""Token mixture: buckets around the sizes where the kernels change what they do (blocks of 16, steps of 32 pairs, tiles of 128) and
both sides of the rule that chooses between them, with lists per token and per KV head, against the fp32 oracle."""
import pytest
import torch

from oracle import moc_oracle as O
from util_cases import assert_close_all_forms

pytestmark = pytest.mark.gpu

# pairs of the first chapters (the rest nobody selects); 256 pairs a chapter on average and more: the 128-row kernels
BUCKETS = {"edges": [1, 2, 15, 16, 17, 31, 32, 33, 48, 49, 64, 65], "one": [1], "tiles": [127, 128, 129, 300],
           "few_rows_side": [255, 255], "tile_side": [256, 256], "bwd_few_rows_side": [170, 170], "bwd_tile_side": [171, 171]}


@pytest.mark.parametrize("heads", [(2, 2), (6, 2)], ids=["mha", "gqa"])
@pytest.mark.parametrize("lists", ["token", "head"])
@pytest.mark.parametrize("name", list(BUCKETS))
def test_bucket_sizes(name, lists, heads):
    from memory_b200 import _lib as L, ops
    dev = torch.device("cuda:0")
    hq, h = heads
    counts = BUCKETS[name]
    m = len(counts) + (2 if len(counts) > 2 else 0)
    g = torch.Generator().manual_seed(sum(counts))
    tokens = sum(counts)                                     # one slot a token, so that the sizes are exact
    order = torch.cat([torch.full((n,), c) for c, n in enumerate(counts)])
    hi = 1 if lists == "token" else h
    bi = torch.stack([order[torch.randperm(tokens, generator=g)] for _ in range(hi)], 1).view(1, tokens, hi, 1).int()
    q, do = (torch.randn(1, tokens, hq, 64, generator=g).bfloat16() for _ in range(2))
    k, v = (torch.randn(1, m * 64, h, 64, generator=g).bfloat16() for _ in range(2))
    w = torch.rand(1, tokens, 1, generator=g) + 0.1
    qc, kc, vc, wc = (t.float().requires_grad_(True) for t in (q, k, v, w))
    ref = 2.5 * O.weighted_chapter_attention(qc, kc, vc, bi.expand(1, tokens, h, 1), wc, 64)
    ref.backward(do.float())
    d = [t.to(dev) for t in (q, k, v, bi, w)]
    o, lse, ws = ops.token_mix_fwd(*d, 0.125, out_scale=2.5)
    dk, dv = (torch.full_like(t, float("nan")) for t in d[1:3])
    dq, dw = ops.token_mix_bwd(*d, lse, do.to(dev), 0.125, 2.5, ws, dk, dv)
    L.check_device_status(dev)
    # bf16 operands: P, dS and the results are rounded once each (2^-9), the sums are fp32
    for got, want, what in ((o, ref, "o"), (dq, qc.grad, "dq"), (dk, kc.grad, "dk"), (dv, vc.grad, "dv"), (dw, wc.grad, "dw")):
        assert_close_all_forms(got, want, 2e-2, what)
    assert not dk[:, len(counts) * 64:].any() and not dv[:, len(counts) * 64:].any()
    again = ops.token_mix_bwd(*d, lse, do.to(dev), 0.125, 2.5, ws, dk2 := torch.empty_like(dk), dv2 := torch.empty_like(dv))
    assert torch.equal(dq, again[0]) and torch.equal(dw, again[1]) and torch.equal(dk, dk2) and torch.equal(dv, dv2)


@pytest.mark.parametrize("pairs", [1, 5, 16, 17, 33, 511, 512, 700])
@pytest.mark.parametrize("heads", [(2, 2), (6, 2)], ids=["mha", "gqa"])
def test_an_infinite_key_stays_with_its_own_gradients(pairs, heads):
    """A key whose score is -inf for every pair has weight 0: forward, dV, dW and the dK of the chapter's other keys are what they are
    without it, whatever stands in the part of a step or tile that holds no pair.  (dQ is NaN by the product 0 * inf.)"""
    from memory_b200 import _lib as L, ops
    dev = torch.device("cuda:0")
    hq, h = heads
    g = torch.Generator().manual_seed(pairs)
    q, do = (torch.randn(1, pairs, hq, 64, generator=g).bfloat16() for _ in range(2))
    k, v = (torch.randn(1, 64, h, 64, generator=g).bfloat16() for _ in range(2))
    q[..., 3] = -q[..., 3].abs() - 0.125
    k[0, 7, :, 3] = float("inf")
    bi, w = torch.zeros(1, pairs, 1, 1, dtype=torch.int32), torch.rand(1, pairs, 1, generator=g) + 0.1
    qc, kc, vc, wc = (t.float().requires_grad_(True) for t in (q, k, v, w))
    ref = O.weighted_chapter_attention(qc, kc, vc, bi.expand(1, pairs, h, 1), wc, 64)
    ref.backward(do.float())
    d = [t.to(dev) for t in (q, k, v, bi, w)]
    o, lse, ws = ops.token_mix_fwd(*d, 0.125)
    dk, dv = (torch.full_like(t, float("nan")) for t in d[1:3])
    dq, dw = ops.token_mix_bwd(*d, lse, do.to(dev), 0.125, 1.0, ws, dk, dv)
    L.check_device_status(dev)
    assert lse.isfinite().all() and dq.isnan().any()
    for got, want, what in ((o, ref, "o"), (dk, kc.grad, "dk"), (dv, vc.grad, "dv"), (dw, wc.grad, "dw")):
        assert want.isfinite().all() and got.isfinite().all(), what
        assert_close_all_forms(got, want, 2e-2, what)           # (bf16 operands, as above)
