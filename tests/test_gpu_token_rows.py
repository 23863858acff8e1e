"""Token mixture: buckets around the sizes where the kernels change what they do (blocks of 16, steps of 32 pairs, tiles of 128) and
both sides of the rule that chooses between them, with lists per token and per KV head, against the fp32 oracle."""
import pytest
import torch

from oracle import moc_oracle as O
from util_cases import assert_close_all_forms

pytestmark = pytest.mark.gpu

# pairs of the first chapters (the rest nobody selects); in the backward, 512 rows (pairs x query heads of a KV head; 256 with lists per head)
# a chapter and more: the 128-row kernel.  So few pairs in all are the other kernel's in the forward: its tiles of up to 128 pairs are what the sizes meet.
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


def _by_chapter(q, k, v, bi, w):
    """Plain fp64 mixture, chapter by chapter: q [T, HQ, 64], k / v [M * 64, H, 64], bi [T, 1 or H, S], w [T, S]."""
    h, per = k.shape[1], q.shape[1] // k.shape[1]
    heads = []
    for kh in range(h):
        ids = bi[:, kh if bi.shape[1] > 1 else 0]
        qh, out = q[:, kh * per:(kh + 1) * per], torch.zeros_like(q[:, :per])
        for c in ids.unique().tolist():
            t, s = (ids == c).nonzero(as_tuple=True)
            p = torch.softmax(torch.einsum("ngd,md->ngm", qh[t], k[c * 64:(c + 1) * 64, kh]) * 0.125, -1)
            out = out.index_add(0, t, w[t, s][:, None, None] * torch.einsum("ngm,md->ngd", p, v[c * 64:(c + 1) * 64, kh]))
        heads.append(out)
    return torch.cat(heads, 1)


@pytest.mark.parametrize("heads,lists", [((2, 2), "token"), ((2, 2), "head"), ((4, 1), "token")], ids=["mha", "lists", "mqa"])
@pytest.mark.parametrize("used", [26, 60, 1000])
def test_the_buckets_decide_between_the_kernels(used, heads, lists):
    """Enough pairs for both kernels and few a chapter on average, all of them in 26 chapters (full tiles, one long item each), in 60, or
    spread: whichever kernel takes the call, the results are the mixture's and repeats are the same bits."""
    from memory_b200 import _lib as L, ops
    dev = torch.device("cuda:0")
    (hq, h), tokens, S, m = heads, 1600, 26, 1000
    g = torch.Generator(device=dev).manual_seed(used + hq)
    rand = lambda *s: torch.randn(*s, generator=g, device=dev).bfloat16()
    hi = 1 if lists == "token" else h
    chosen = torch.randperm(m, generator=g, device=dev)[:used]
    bi = chosen[torch.rand(tokens, hi, used, generator=g, device=dev).topk(S, -1).indices].int()
    q, do, k, v = rand(1, tokens, hq, 64), rand(1, tokens, hq, 64), rand(1, m * 64, h, 64), rand(1, m * 64, h, 64)
    w = torch.rand(1, tokens, S, generator=g, device=dev) + 0.1
    qc, kc, vc, wc = (t[0].double().requires_grad_(True) for t in (q, k, v, w))
    ref = _by_chapter(qc, kc, vc, bi.long(), wc)
    ref.backward(do[0].double())
    runs = []
    for _ in range(2):
        o, lse, ws = ops.token_mix_fwd(q, k, v, bi[None], w, 0.125)
        dk, dv = (torch.full_like(t, float("nan")) for t in (k, v))
        dq, dw = ops.token_mix_bwd(q, k, v, bi[None], w, lse, do, 0.125, 1.0, ws, dk, dv)
        runs.append((o, dq, dk, dv, dw))
    L.check_device_status(dev)
    for got, want, what in zip(runs[0], (ref, qc.grad, kc.grad, vc.grad, wc.grad), ("o", "dq", "dk", "dv", "dw")):
        assert_close_all_forms(got[0], want.float(), 2e-2, what)      # (bf16 operands, as above)
    assert all(torch.equal(a, b) for a, b in zip(*runs))


@pytest.mark.parametrize("heads", [(2, 2), (6, 2)], ids=["mha", "gqa"])
@pytest.mark.parametrize("lists", ["token", "head"])
@pytest.mark.parametrize("B,tokens", [(5, 1801), (2, 75)], ids=["tiles", "few_rows"])
def test_batches_slots_strided_rows_base_and_an_unselected_chapter(B, tokens, lists, heads):
    """Sequences of three slots on six chapters, one that every token selects (a ragged last tile), one that nobody selects, K and V
    halves of one row, a base under the outputs and the query gradients, bit-identical repeats, an id out of range.  27,015 pairs, 900 a
    chapter on average: the 128-row kernels in both passes; 38 a chapter: those for chapters with few pairs."""
    from memory_b200 import _lib as L, ops
    dev = torch.device("cuda:0")
    hq, h = heads
    S, m, rho = 3, 6, 2.5
    g = torch.Generator(device=dev).manual_seed(tokens + hq)
    hi = 1 if lists == "token" else h
    others = 1 + torch.rand(B, tokens, hi, m - 2, generator=g, device=dev).topk(S - 1, -1).indices
    bi = torch.cat([torch.zeros_like(others[..., :1]), others], -1).int()
    q, base, do, dq0 = (torch.randn(B, tokens, hq, 64, generator=g, device=dev).bfloat16() for _ in range(4))
    # A value of dV sums thousands of products that are rounded to 2^-9: six of its standard deviations are 6 * 2^-9 / sqrt(3) of the
    # values' rms, which a quarter of dO keeps near one.
    do = do / 4
    kv = torch.randn(B, m * 64, 2 * h * 64, generator=g, device=dev).bfloat16()
    w = torch.rand(B, tokens, S, generator=g, device=dev) + 0.1
    halves = lambda t: (t[..., :h * 64].unflatten(-1, (h, 64)), t[..., h * 64:].unflatten(-1, (h, 64)))
    qc, kc, vc, wc = (t.double().requires_grad_(True) for t in (q, *halves(kv), w))
    ref = base.double() + rho * torch.stack([_by_chapter(qc[b], kc[b], vc[b], bi[b].long(), wc[b]) for b in range(B)])
    ref.backward(do.double())

    def run():
        o, lse, ws = ops.token_mix_fwd(q, *halves(kv), bi, w, 0.125, base=base, out_scale=rho)
        d_kv = torch.full_like(kv, float("nan"))                 # the call writes every row
        dq, dw = ops.token_mix_bwd(q, *halves(kv), bi, w, lse, do, 0.125, rho, ws, *halves(d_kv), d_q_base=dq0)
        return o, dq, dw, d_kv

    o, dq, dw, d_kv = run()
    L.check_device_status(dev)
    dk, dv = halves(d_kv)
    # (bf16 operands and results, as above; the base's part of dQ is exact up to the rounding of the sum)
    for got, want, what in ((o, ref, "o"), (dq, qc.grad + dq0.double(), "dq"), (dw, wc.grad, "dw"), (dk, kc.grad, "dk"), (dv, vc.grad, "dv")):
        assert_close_all_forms(got, want.float(), 2e-2, what)
    assert not d_kv[:, 5 * 64:].any(), "rows of a chapter nobody selected are zero"
    assert all(torch.equal(a, b) for a, b in zip((o, dq, dw, d_kv), run()))
    bi[1, 7, 0, 1] = m
    o2, _, _ = ops.token_mix_fwd(q, *halves(kv), bi, w, 0.125, base=base, out_scale=rho)
    same = torch.ones(B, tokens, dtype=torch.bool, device=dev)
    same[1, 7] = False
    assert torch.equal(o2[same], o[same])
    with pytest.raises(RuntimeError, match="out of range"):
        L.check_device_status(dev)


@pytest.mark.parametrize("tokens,S,chapters,heads", [(250, 16, 512, (4, 4)), (1200, 4, 300, (4, 2))])
def test_the_weights_gradient_keeps_the_128_row_kernels_precision(tokens, S, chapters, heads):
    """dW leaves in fp32.  From fp64, 2-norm: 2.75e-7 in the kernel of 128-row tiles, 2.7e-7 here, and 3.1e-7 with one chain of products
    over a head's 64 columns."""
    from memory_b200 import _lib as L, ops
    dev = torch.device("cuda:0")
    (hq, h) = heads
    g = torch.Generator(device=dev).manual_seed(tokens)
    q, do, k, v = (torch.randn(1, n, i, 64, generator=g, device=dev).bfloat16()
                   for n, i in ((tokens, hq), (tokens, hq), (chapters * 64, h), (chapters * 64, h)))
    bi = torch.rand(tokens, 1, chapters, generator=g, device=dev).topk(S, -1).indices.int()
    w = torch.softmax(torch.randn(1, tokens, S, generator=g, device=dev), -1)
    wc = w[0].double().requires_grad_(True)
    _by_chapter(q[0].double(), k[0].double(), v[0].double(), bi.long(), wc).backward(do[0].double())
    _, lse, ws = ops.token_mix_fwd(q, k, v, bi[None], w, 0.125)
    _, dw = ops.token_mix_bwd(q, k, v, bi[None], w, lse, do, 0.125, 1.0, ws, torch.empty_like(k), torch.empty_like(v))
    L.check_device_status(dev)
    assert float((dw[0].double() - wc.grad).norm() / wc.grad.norm()) < 2.9e-7
