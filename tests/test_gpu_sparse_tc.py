"""``memory_cross_attn`` on the tensor cores (bf16, head_dim 64, chapters of a multiple of 64 rows) against the oracle:
units of 64 and 128 keys and chapters of several units, groups that fill a row tile unevenly, chapters with no pair, one
pair and several row tiles, buckets cut into several work items."""
import pytest
import torch

from util_cases import assert_close_all_forms
from oracle import moc_oracle as O

pytestmark = pytest.mark.gpu

SHAPES = {
    "unit64_g1": dict(B=2, TQ=77, M=7, HQ=2, H=2, S=3, BS=64),
    "unit64_g3_many_tiles": dict(B=1, TQ=300, M=3, HQ=6, H=2, S=2, BS=64),
    "unit128_g16": dict(B=1, TQ=130, M=5, HQ=16, H=1, S=3, BS=128),
    "three_units_of_64": dict(B=2, TQ=33, M=4, HQ=4, H=1, S=2, BS=192),
    "two_units_of_128": dict(B=1, TQ=40, M=3, HQ=2, H=2, S=1, BS=256),
    "one_token_one_block": dict(B=1, TQ=1, M=9, HQ=1, H=1, S=1, BS=64),
    "all_tokens_one_chapter": dict(B=1, TQ=4100, M=1, HQ=8, H=1, S=1, BS=64),
}


def _problem(B, TQ, M, HQ, H, S, BS, seed=5):
    g = torch.Generator().manual_seed(seed)
    q, k, v, do = (torch.randn(B, n, h, 64, generator=g).bfloat16()
                   for n, h in ((TQ, HQ), (M * BS, H), (M * BS, H), (TQ, HQ)))
    bi = torch.rand(B * TQ * H, M, generator=g).topk(S, dim=1).indices.view(B, TQ, H, S).int()
    return q, k, v, bi, do


@pytest.mark.parametrize("name", list(SHAPES))
def test_values_gradients_and_repeats(name):
    import memory_b200 as M
    from memory_b200 import _lib as L, ops
    dev = torch.device("cuda:0")
    bs = SHAPES[name]["BS"]
    q, k, v, bi, do = _problem(**SHAPES[name])
    qc, kc, vc = (t.float().requires_grad_(True) for t in (q, k, v))
    ref = O.sparse_chapter_attention(qc, kc, vc, bi, bs)
    ref.backward(do.float())
    runs = []
    for _ in range(2):
        qg, kg, vg = (t.to(dev).requires_grad_(True) for t in (q, k, v))
        seen = []
        ops.LAUNCH_HOOK = seen.append
        try:
            o = M.memory_cross_attn(qg, kg, vg, bi.to(dev), bs)
            o.backward(do.to(dev))
        finally:
            ops.LAUNCH_HOOK = None
        assert "sparse_attn_tc_fwd:bf16" in seen and "sparse_attn_tc_bwd:bf16" in seen
        runs.append((o.detach(), qg.grad, kg.grad, vg.grad))
    L.check_device_status(dev)
    for got, want, tol, what in zip(runs[0], (ref, qc.grad, kc.grad, vc.grad), (2e-2, 3e-2, 3e-2, 3e-2), "o dq dk dv".split()):
        assert_close_all_forms(got, want, tol, what)
    if SHAPES[name]["TQ"] * SHAPES[name]["S"] <= 2048:          # longer lists are not sorted
        assert all(torch.equal(a, b) for a, b in zip(*runs))


def test_stand_alone_backward_and_bad_ids():
    import memory_b200 as M
    from memory_b200 import _lib as L
    dev = torch.device("cuda:0")
    q, k, v, bi, do = (t.to(dev) for t in _problem(B=1, TQ=50, M=6, HQ=4, H=2, S=2, BS=64))
    o, lse = M.memory_cross_attn_forward(q, k, v, bi, 64)
    qg, kg, vg = (t.clone().requires_grad_(True) for t in (q, k, v))
    M.memory_cross_attn(qg, kg, vg, bi, 64).backward(do)
    dq, dk, dv = M.memory_cross_attn_backward(q, k, v, o, lse, do, bi, 64)
    L.check_device_status(dev)
    assert torch.equal(dq, qg.grad) and torch.equal(dk, kg.grad) and torch.equal(dv, vg.grad)
    # a listed block that does not exist is reported and contributes nothing; a token with none left gets zeros
    bad = bi.clone()
    bad[0, 3, :, :] = 6
    bad[0, 4, 0, 1] = -1
    o2, _ = M.memory_cross_attn_forward(q, k, v, bad, 64)
    with pytest.raises(RuntimeError, match="out of range"):
        L.check_device_status(dev)
    assert not o2[0, 3].any() and torch.equal(o2[0, 5:], o[0, 5:]) and torch.isfinite(o2).all()
