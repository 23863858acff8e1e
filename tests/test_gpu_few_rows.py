"""The kernels of a decoding step at the edges of their ranges, against the same arithmetic in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30))


@pytest.fixture(scope="module")
def dev():
    return torch.device("cuda:0")


@pytest.mark.parametrize("b,l,d,c", [(1, 1, 4, 3), (8, 33, 256, 65), (9, 5, 260, 70), (64, 128, 768, 4097), (3, 1024, 1024, 33),
                                     (17, 40, 1028, 41), (2, 1025, 30, 9)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_router_rows(dev, b, l, d, c, dtype):
    """Pooling, logits, d_w and d_pooled for few and many rows, widths that fill the register tile or not, both poolings."""
    from memory_b200 import ops
    torch.manual_seed(b + d)
    h = torch.randn(b, l, d, device=dev).to(dtype)
    w, bias = torch.randn(c, d, device=dev), torch.randn(c, device=dev)
    f = ops.router_fwd(h, w, bias, 2, 1, 1.0, True)
    pooled = h.double().mean(1)
    assert _rel(f["pooled"], pooled) < 1e-6
    assert _rel(f["logits"], pooled @ w.double().t() + bias.double()) < 1e-6
    g = torch.randn_like(f["weights"])
    r = ops.router_bwd((b, l, d), dtype, w, f, 2, 1, 1.0, g, None, torch.ones(4, device=dev), True)
    dl = r["d_logits"].double()
    assert _rel(r["d_w"], dl.t() @ f["pooled"].double()) < 1e-5 and _rel(r["d_bias"], dl.sum(0)) < 1e-5
    assert _rel(r["d_h"], ((dl @ w.double()) / l).unsqueeze(1).expand(b, l, d)) < (1e-5 if dtype == torch.float32 else 5e-3)


@pytest.mark.parametrize("m,n,k", [(1, 1, 8), (8, 768, 768), (9, 7, 264), (63, 100, 1024), (64, 520, 512), (65, 64, 768), (5, 64, 1032)])
@pytest.mark.parametrize("out", [torch.float32, torch.bfloat16])
def test_projection_of_few_rows(dev, m, n, k, out):
    from memory_b200 import ops
    torch.manual_seed(m + n)
    a, w = torch.randn(m, k, device=dev).bfloat16(), torch.randn(n, k, device=dev).bfloat16()
    y = ops.gemm(a, w, out_dtype=out)
    assert y.dtype == out and _rel(y, a.double() @ w.double().t()) < (1e-5 if out == torch.float32 else 4e-3)


@pytest.mark.parametrize("b,nq,h,hk,t,n_ch", [(1, 1, 12, 12, 64, 65), (1, 1, 4, 1, 5, 3), (2, 3, 6, 2, 33, 4), (1, 1, 1, 1, 1, 1),
                                              (40, 1, 8, 4, 16, 9), (3, 2, 5, 1, 70, 2)])
def test_decode_attention_shapes(dev, b, nq, h, hk, t, n_ch):
    """Clusters of one to eight CTAs, one to four query heads a CTA, chapters that fill no run of 32 rows."""
    from memory_b200 import ops
    torch.manual_seed(b + t)
    c = n_ch + 3
    q = torch.randn(b, nq, h * 64, device=dev).bfloat16()
    kv = torch.randn(c * t, 2 * hk * 64, device=dev).bfloat16()
    idx = torch.stack([torch.randperm(c, device=dev)[:n_ch] for _ in range(b)]).int()
    u = torch.rand(b, n_ch, device=dev) + 0.1
    o, lse = ops.decode_attn(q, kv, idx, u, h, hk, t, 0.125, want_lse=True)
    rows = (idx.long() * t).unsqueeze(-1) + torch.arange(t, device=dev)
    x = kv[rows.view(b, -1)].double() * u.double().repeat_interleave(t, 1).unsqueeze(-1)
    k, v = (y.view(b, n_ch * t, hk, 64).repeat_interleave(h // hk, 2) for y in x.chunk(2, dim=-1))
    s = torch.einsum("bqhd,bkhd->bhqk", q.view(b, nq, h, 64).double(), k) * 0.125
    want = torch.einsum("bhqk,bkhd->bqhd", s.softmax(-1), v).reshape(b, nq, h * 64)
    assert _rel(o, want) < 5e-3 and _rel(lse, torch.logsumexp(s, -1).transpose(1, 2)) < 1e-4


@pytest.mark.parametrize("dtype,d", [(torch.bfloat16, 768), (torch.float32, 12), (torch.bfloat16, 12)])
def test_routing_window_is_the_sliced_concatenation(dev, dtype, d):
    import memory_b200 as M
    torch.manual_seed(d)
    prompt = torch.randn(3, 9, d, device=dev).to(dtype)
    window, want = M.RoutingWindow(6, "hybrid"), prompt[:, -6:]
    window.prefill(prompt)
    for n in (1, 2, 1, 7, 6):
        h = torch.randn(3, n, d, device=dev).to(dtype)
        want = torch.cat([want, h], 1)[:, -6:]
        assert torch.equal(window.step(h), want)
    window = M.RoutingWindow(6, "rolling")
    want = window.prefill(prompt[:, :2])
    for n in (1, 2, 3):
        want = torch.cat([want, prompt[:, :n]], 1)[:, -6:]
        assert torch.equal(window.step(prompt[:, :n]), want)


@pytest.mark.parametrize("rows,c,d,k,s", [(136, 4097, 256, 16, 1), (592, 1280, 256, 300, 0), (600, 1283, 200, 8, 2), (608, 4352, 64, 5, 1),
                                          (616, 4355, 72, 5, 1)])
def test_token_router_shapes(dev, rows, c, d, k, s):
    """Both CTA widths of the selection, chapter counts and widths that fill no tile, the terms of weight and gradient."""
    import memory_b200 as M
    torch.manual_seed(rows + c)
    h = torch.randn(1, rows, d, device=dev).bfloat16().requires_grad_(True)
    w = (torch.randn(c, d, device=dev) * 0.05).requires_grad_(True)
    bias = (torch.randn(c, device=dev) * 0.1).requires_grad_(True)
    idx, wt, losses = M.route_tokens(h, w, bias, k, s, True)
    g = torch.randn_like(wt)
    coef = {"load_balance": 0.3, "z_loss": 0.2, "entropy": 0.1}
    (sum(coef[n] * losses[n] for n in coef) + (wt * g).sum()).backward()
    h64, w64, b64 = (t.detach().double().requires_grad_(True) for t in (h, w, bias))
    z = h64[0] @ w64.t() + b64
    p = z.softmax(-1)
    masked = torch.cat([torch.zeros_like(p[:, :s]), p[:, s:]], 1)
    top = masked.gather(1, idx[0])
    assert (top.min(1).values >= masked.detach().topk(k, 1).values[:, -1] * (1 - 1e-5)).all()
    w_ref = top / top.sum(1, keepdim=True)
    f = torch.zeros_like(p).scatter_(1, idx[0], 1.0).mean(0)
    lb = c * (f * p.mean(0)).sum()
    zl = torch.logsumexp(z, 1).square().mean()
    ent = -(p * p.clamp_min(1e-12).log()).sum(1).mean()
    for name, ref in (("load_balance", lb), ("z_loss", zl), ("entropy", ent)):
        assert abs(float(losses[name]) - float(ref)) < 2e-5 * abs(float(ref)), name
    (0.3 * lb + 0.2 * zl + 0.1 * ent + (w_ref * g[0].double()).sum()).backward()
    assert _rel(wt[0], w_ref) < 1e-5
    assert _rel(w.grad, w64.grad) < 1e-4 and _rel(bias.grad, b64.grad) < 1e-4 and _rel(h.grad, h64.grad) < 1e-2


@pytest.mark.parametrize("rows,k,m,s,h,hk,bank_dtype", [(8, 1, 300, 2, 4, 2, torch.float32), (136, 3, 205, 0, 2, 2, torch.bfloat16),
                                                        (72, 5, 180, 1, 3, 1, torch.float32), (72, 5, 181, 1, 3, 1, torch.bfloat16),
                                                        (600, 2, 7, 1, 2, 1, torch.float32)])
def test_token_attention_over_listed_chapters(dev, rows, k, m, s, h, hk, bank_dtype):
    """Few selections (only the chapters somebody selected are projected) and many, on both sides of the line between them."""
    import memory_b200 as M
    torch.manual_seed(rows + m)
    d, dkv = h * 64, hk * 64
    rnd = lambda *shape, std=1.0, dtype=torch.float32: (torch.randn(*shape, device=dev) * std).to(dtype).requires_grad_(True)
    x = rnd(1, rows, d, dtype=torch.bfloat16)
    shared, routed = (rnd(s * 64, d, dtype=bank_dtype) if s else None), rnd(m * 64, d, dtype=bank_dtype)
    wq, wk, wv, wo = rnd(d, d, std=0.1), rnd(dkv, d, std=0.1), rnd(dkv, d, std=0.1), rnd(d, d, std=0.1)
    idx = torch.rand(rows, m, device=dev).topk(k, 1).indices.int().view(1, rows, k)
    u = torch.rand(1, rows, k, device=dev).requires_grad_(True)
    leaves = [t for t in (x, shared, routed, u, wq, wk, wv, wo) if t is not None]
    g = torch.randn(1, rows, d, device=dev).bfloat16()

    def grads(out):
        return [out] + list(torch.autograd.grad(out, leaves, g.to(out.dtype)))

    got = grads(M.token_routed_attention(x, shared, routed, idx, u, wq, wk, wv, wo, num_heads=h, num_kv_heads=hk,
                                         tokens_per_chapter=64, routed_scale=2.5, compute_dtype=torch.bfloat16))
    q = (x[0].float() @ wq.t()).view(rows, h, 64)

    def heads(mem):
        kv = [(mem.float() @ w.t()).view(-1, hk, 64).repeat_interleave(h // hk, 1) for w in (wk, wv)]
        return kv

    out = torch.zeros(rows, h, 64, device=dev)
    if s:
        ks, vs = heads(shared)
        out = torch.einsum("thn,nhd->thd", (torch.einsum("thd,nhd->thn", q, ks) * 0.125).softmax(-1), vs)
    kr, vr = (t.view(m, 64, h, 64) for t in heads(routed))
    for j in range(k):
        c = idx[0, :, j].long()
        p = (torch.einsum("thd,tnhd->thn", q, kr[c]) * 0.125).softmax(-1)
        out = out + 2.5 * u[0, :, j, None, None] * torch.einsum("thn,tnhd->thd", p, vr[c])
    want = grads((out.reshape(rows, d) @ wo.t()).view(1, rows, d))
    for i, (a, b) in enumerate(zip(got, want)):
        assert _rel(a, b) < 2e-2, i
    from memory_b200 import _lib as L
    L.check_device_status(dev)


@pytest.mark.parametrize("rows,d", [(1, 4), (17, 256), (33, 260), (100, 768), (16, 772), (31, 1024), (9, 1028)])
@pytest.mark.parametrize("kind", ["rms", "layernorm"])
def test_norm_backward_widths(dev, rows, d, kind):
    """Rows in registers (every width class and its edge) and in two passes."""
    from memory_b200 import ops
    torch.manual_seed(rows + d)
    x, dy, res = (torch.randn(rows, d, device=dev) for _ in range(3))
    w, b = torch.rand(d, device=dev) + 0.5, torch.randn(d, device=dev)
    x64, w64, b64 = (t.double().requires_grad_(True) for t in (x, w, b))
    mu = x64.mean(-1, keepdim=True) if kind == "layernorm" else 0.0
    y = (x64 - mu) / ((x64 - mu).square().mean(-1, keepdim=True) + 1e-5).sqrt() * w64
    (y + b64 if kind == "layernorm" else y).backward(dy.double())
    _, stats = ops.norm_fwd(x, w, b if kind == "layernorm" else None, kind, 1e-5, torch.float32)
    dx, dw, db = ops.norm_bwd(dy, x, w, stats, res, kind, kind == "layernorm")
    assert _rel(dx, x64.grad + res.double()) < 1e-5 and _rel(dw, w64.grad) < 1e-5
    if kind == "layernorm":
        assert _rel(db, b64.grad) < 1e-5
