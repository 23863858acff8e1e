"""``memory_cross_attn`` on the tensor cores in slices: scratch is bounded whatever the problem's size, and the results are
those of smaller calls."""
import ctypes as C

import pytest
import torch

GIB = 1 << 30


def _sizes(batch, tq, tk, hq, h, select, block):
    from memory_b200 import _lib as L, ops
    return ops._sparse_tc_sizes(L.SparseAttnShape(batch, tq, tk, hq, h, 64, select, block, 0.125, L.MOC_BF16))


@pytest.mark.parametrize("batch, tq, tk, hq, h, select, block", [
    (1, 8192, 512 * 128, 16, 1, 8, 128),           # whole
    (1, 16500, 24 * 128, 16, 1, 8, 128), (5, 5000, 24 * 128, 16, 1, 8, 128), (4, 65536, 512 * 128, 16, 1, 8, 128),
    (1024, 16, 64 * 64, 8, 8, 16, 64), (3, 100000, 4096 * 64, 12, 4, 16, 64), (7, 33333, 9 * 192, 128, 1, 3, 192),
    (1, 1 << 24, 64 * 64, 8, 8, 8, 64),            # 2^30 pairs: beyond the ids of one pass
])
def test_scratch_is_bounded(batch, tq, tk, hq, h, select, block):
    from memory_b200.build import build
    build()
    index, fwd, bwd = _sizes(batch, tq, tk, hq, h, select, block)
    sums = 2 * tk * h * 64 * 4                     # fp32 dK / dV of one batch item
    assert 0 < fwd <= GIB and 0 < bwd <= GIB + GIB // 16 + sums and 0 < index <= GIB
    # a slice of this size is worth its launches
    if fwd < batch * tq * hq * select * (block // (128 if block % 128 == 0 else 64)) * 260:
        assert max(fwd, bwd) > GIB // 8


def _run(q, k, v, bi, do, block):
    import memory_b200 as M
    q, k, v = (t.clone().requires_grad_(True) for t in (q, k, v))
    o = M.memory_cross_attn(q, k, v, bi, block)
    o.backward(do)
    return o.detach(), q.grad, k.grad, v.grad


@pytest.mark.gpu
@pytest.mark.parametrize("b, tq, m, hq, h, s, block", [
    (1, 16500, 24, 16, 1, 8, 128),                 # token slices, dK / dV added in fp32, both kinds of buckets
    (1, 66000, 40, 8, 8, 8, 64),
    (2, 17000, 1500, 16, 1, 8, 128),               # token slices of two items, chapters with few pairs or none
    (5, 5000, 24, 16, 1, 8, 128),                  # whole items, a shorter last slice
])
def test_slices_give_the_results_of_smaller_calls(b, tq, m, hq, h, s, block):
    from memory_b200 import _lib as L
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(5)
    rnd = lambda n, heads: torch.randn(b, n, heads, 64, generator=g, device=dev).bfloat16()      # noqa: E731
    q, k, v, do = rnd(tq, hq), rnd(m * block, h), rnd(m * block, h), rnd(tq, hq)
    bi = torch.rand(b * tq * h, m, generator=g, device=dev).topk(s, dim=1).indices.view(b, tq, h, s).int()
    index, fwd, bwd = _sizes(b, tq, m * block, hq, h, s, block)
    assert fwd < b * tq * hq * s * 260             # it is cut
    o, dq, dk, dv = _run(q, k, v, bi, do, block)
    cut = 4001
    dk_sum, dv_sum = torch.zeros_like(k, dtype=torch.float32), torch.zeros_like(v, dtype=torch.float32)
    for i in range(b):
        for t0 in range(0, tq, cut):
            t = slice(t0, min(tq, t0 + cut))
            part = _run(q[i:i + 1, t].contiguous(), k[i:i + 1], v[i:i + 1], bi[i:i + 1, t].contiguous(),
                        do[i:i + 1, t].contiguous(), block)
            assert torch.equal(o[i:i + 1, t], part[0]) and torch.equal(dq[i:i + 1, t], part[1])
            dk_sum[i] += part[2][0].float()
            dv_sum[i] += part[3][0].float()
    L.check_device_status(dev)
    for got, want in ((dk, dk_sum), (dv, dv_sum)):
        # against sums of up to 17 pieces that were rounded to bf16 (2^-9 each of its own size), and one rounding here
        assert float((got.float() - want).norm() / want.norm()) < 1e-2
