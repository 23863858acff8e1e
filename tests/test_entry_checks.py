"""What the entry points refuse before a native pass gets raw pointers: shapes that contradict the sizes of its descriptor.
The refusals come ahead of the look at the device, so CPU tensors show them; the accepted odd shapes are compared on the GPU."""
import pytest
import torch

D, HEADS = 128, 2


def _attn_args(**over):
    a = dict(h=torch.zeros(2, 8, D), memory=torch.zeros(2, 24, D), wq=torch.zeros(D, D), wk=torch.zeros(D, D),
             wv=torch.zeros(D, D), wo=torch.zeros(D, D), num_heads=HEADS, num_kv_heads=None)
    a.update(over)
    return a


@pytest.mark.parametrize("over, message", [
    # grouped weights with the group count left out: the likeliest mistake
    (dict(wk=torch.zeros(64, D), wv=torch.zeros(64, D)), "num_kv_heads"),
    (dict(wv=torch.zeros(64, D)), "num_kv_heads"),
    (dict(num_kv_heads=1), "num_kv_heads"),
    (dict(wq=torch.zeros(D, 64)), "inner dimensions differ: wq"),
    (dict(wk=torch.zeros(D, 64)), "inner dimensions differ: wk"),
    (dict(wv=torch.zeros(D, 64)), "inner dimensions differ: wv"),
    (dict(wo=torch.zeros(D, 64)), "inner dimensions differ: wo"),
    (dict(memory=torch.zeros(2, 24, 64)), "inner dimensions differ: wk"),
    (dict(memory=torch.zeros(3, 24, D)), "batch size"),
    (dict(num_heads=3), "heads"),
    (dict(wo=torch.zeros(64, D), add_residual=True), "residual"),
    (dict(pre_norm="rms", norm_weight=torch.ones(64)), "norm_weight"),
    (dict(pre_norm="layernorm", norm_weight=torch.ones(D), norm_bias=torch.ones(64)), "norm_bias"),
    ({}, "CUDA"),
])
def test_cross_attention_refuses(over, message):
    from memory_b200 import functional as F
    with pytest.raises(ValueError, match=message):
        F.cross_attention(**_attn_args(**over))


def _dense_attention(h, memory, wq, wk, wv, wo, heads, kv_heads):
    """Plain fp64 form; the softmax scale is that of the hidden width."""
    b, l, d = h.shape
    q = (h @ wq.T).view(b, l, heads, -1).transpose(1, 2)
    k, v = ((memory @ w.T).view(b, -1, kv_heads, q.shape[-1]).transpose(1, 2).repeat_interleave(heads // kv_heads, dim=1)
            for w in (wk, wv))
    p = torch.softmax(q @ k.transpose(-1, -2) * (d // heads) ** -0.5, dim=-1)
    return (p @ v).transpose(1, 2).reshape(b, l, -1) @ wo.T


# widths of Q and of the result that are not the hidden width; d_model, attention width, result width, heads, KV heads
@pytest.mark.gpu
@pytest.mark.parametrize("dtype, dims", [
    (torch.float32, (96, 64, 96, 4, 2)), (torch.float32, (96, 128, 40, 2, 1)), (torch.float32, (96, 96, 64, 3, 3)),
    (torch.bfloat16, (192, 128, 64, 2, 1)), (torch.bfloat16, (128, 256, 128, 4, 2)),
])
def test_cross_attention_takes_rectangular_projections(dtype, dims):
    from memory_b200 import _lib as L, functional as F
    d, hd, od, heads, kv = dims
    dkv, g = kv * (hd // heads), torch.Generator().manual_seed(3)
    shapes = {"h": (2, 64, d), "memory": (2, 76, 72), "wq": (hd, d), "wk": (dkv, 72), "wv": (dkv, 72), "wo": (od, hd)}
    x = {n: (torch.randn(*s, generator=g) * (1.0 if n in ("h", "memory") else s[-1] ** -0.5)).to(dtype)
         for n, s in shapes.items()}
    ref = {n: t.double().requires_grad_(True) for n, t in x.items()}
    want = _dense_attention(*ref.values(), heads, kv)
    grad = torch.randn(want.shape, generator=g)
    want.backward(grad.to(dtype).double())
    mine = {n: t.cuda().requires_grad_(True) for n, t in x.items()}
    out = F.cross_attention(*mine.values(), heads, kv)
    out.backward(grad.to(dtype).cuda())
    L.check_device_status(out.device)
    # fp32: sums of at most a few hundred fp32 products; bf16: a handful of bf16 roundings (2^-9 each) on the way
    tol = 2e-5 if dtype == torch.float32 else 2e-2
    for name, a, b in [("out", out, want)] + [(n, mine[n].grad, ref[n].grad) for n in x]:
        assert a.shape == b.shape, name
        err = (a.detach().double().cpu() - b.detach()).norm() / b.detach().norm()
        assert float(err) < tol, (name, float(err))


# ---- the whole layer ---------------------------------------------------------------------------------------------
def _layer_args(**over):
    a = dict(h_router=torch.zeros(2, 8, D, dtype=torch.bfloat16), h_attn=torch.zeros(2, 8, D, dtype=torch.bfloat16),
             bank=torch.zeros(9 * 64, D), router_weight=torch.zeros(9, D), router_bias=torch.zeros(9), wq=torch.zeros(D, D),
             wk=torch.zeros(D, D), wv=torch.zeros(D, D), wo=torch.zeros(D, D), num_heads=HEADS, num_kv_heads=None,
             tokens_per_chapter=64, top_k=2)
    a.update(over)
    return a


@pytest.mark.parametrize("over, message", [
    (dict(wk=torch.zeros(64, D), wv=torch.zeros(64, D)), "num_kv_heads"),
    (dict(wv=torch.zeros(64, D)), "num_kv_heads"),
    (dict(wq=torch.zeros(D, 64)), "inner dimensions differ: wq"),
    (dict(wk=torch.zeros(D, 64)), "inner dimensions differ: wk"),
    (dict(wo=torch.zeros(D, 64)), "inner dimensions differ: wo"),
    (dict(h_router=torch.zeros(1, 8, D, dtype=torch.bfloat16)), "share the batch"),
    (dict(h_router=torch.zeros(2, 8, 64, dtype=torch.bfloat16)), "inner dimensions differ: router_weight"),
    (dict(router_weight=torch.zeros(9, 64)), "inner dimensions differ: router_weight"),
    (dict(router_bias=torch.zeros(8)), "router_bias"),
    (dict(pre_norm="rms", pre_norm_weight=torch.ones(64)), "pre_norm_weight"),
    (dict(pre_norm="layernorm", pre_norm_weight=torch.ones(D), pre_norm_bias=torch.ones(64)), "pre_norm_bias"),
    ({}, "CUDA"),
])
def test_memory_layer_refuses(over, message):
    from memory_b200 import functional as F
    with pytest.raises(ValueError, match=message):
        F.memory_layer(**_layer_args(**over))


def _layer_run(two_stream, h_router, h_attn, seed=7):
    """(outputs, gradients) of a small layer; router and attention may look at different states."""
    from memory_b200 import _lib as L, functional as F
    g = torch.Generator().manual_seed(seed)
    dr = h_router.shape[2]
    p = {"bank": torch.randn(9 * 64, D, generator=g), "router_w": torch.randn(9, dr, generator=g) * 0.3,
         "router_b": torch.randn(9, generator=g) * 0.1, **{n: torch.randn(D, D, generator=g) * D ** -0.5
                                                          for n in ("wq", "wk", "wv", "wo")}}
    p = {n: t.cuda().requires_grad_(True) for n, t in p.items()}
    same = h_router is h_attn
    ha = h_attn.cuda().requires_grad_(True)
    hr = ha if same else h_router.cuda().requires_grad_(True)
    out, losses, info = F.memory_layer(hr, ha, *p.values(), num_heads=HEADS, num_kv_heads=None, tokens_per_chapter=64,
                                       top_k=3, two_stream=two_stream, compute_dtype=torch.bfloat16)
    torch.autograd.backward([out, losses.vector], [torch.randn(out.shape, generator=g).to(out.dtype).cuda(),
                                                   torch.tensor([1.0, 0.5, 0.1, 0.2], device="cuda")])
    L.check_device_status(out.device)
    return {"out": out, "idx": info["indices"], "h_attn": ha.grad, "h_router": hr.grad, **{n: t.grad for n, t in p.items()}}


@pytest.mark.gpu
@pytest.mark.parametrize("width, seq", [(64, 50), (200, 64), (72, 1500)])
def test_router_states_of_another_width_than_the_attention(width, seq):
    g = torch.Generator().manual_seed(1)
    h_router, h_attn = (torch.randn(2, n, w, generator=g).bfloat16() for n, w in ((seq, width), (64, D)))
    one, chain = (_layer_run(two, h_router, h_attn) for two in (True, False))
    assert torch.equal(one.pop("idx"), chain.pop("idx"))
    for n in one:        # the same bf16 operators in one call or in three; gradients may round once more between nodes
        err = (one[n].detach().float() - chain[n].detach().float()).norm() / chain[n].detach().float().norm()
        assert one[n].dtype == chain[n].dtype and float(err) < 2e-2, (n, float(err))


@pytest.mark.gpu
def test_fp16_states_get_fp16_gradients():
    """States the kernels do not take themselves go through bf16, and so do their gradients."""
    h = torch.randn(2, 64, D, generator=torch.Generator().manual_seed(2)).bfloat16()
    want, got = (_layer_run(True, x, x) for x in (h, h.half()))
    assert got["h_attn"].dtype == torch.float16
    err = (got["h_attn"].float() - want["h_attn"].float()).norm() / want["h_attn"].float().norm()
    assert float(err) < 1e-2, float(err)      # two bf16 roundings (2^-9) of the sum of both branches against one


# ---- routers -----------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("over, message", [
    (dict(weight=torch.zeros(9, 64)), "inner dimensions differ"),
    (dict(weight=torch.zeros(9, 256)), "inner dimensions differ"),
    (dict(bias=torch.zeros(8)), "bias"),
    ({}, "CUDA"),
])
def test_routers_refuse(over, message):
    from memory_b200 import functional as F, ops
    a = dict(dict(weight=torch.zeros(9, D), bias=torch.zeros(9)), **over)
    h = torch.zeros(2, 8, D, dtype=torch.bfloat16)
    with pytest.raises(ValueError, match=message):
        F.route(h, a["weight"], a["bias"], 2, 1)
    with pytest.raises(ValueError, match=message):
        F.route_tokens(h, a["weight"], a["bias"], 2, 1)
    with pytest.raises(ValueError, match=message):
        ops.token_route_fwd(h.view(16, D), a["weight"], a["bias"], 2, 1, True)


def test_route_refuses_pooling_coefficients_of_another_length():
    from memory_b200 import functional as F
    with pytest.raises(ValueError, match="pos_weight"):
        F.route(torch.zeros(2, 8, D), torch.zeros(9, D), torch.zeros(9), 2, 1, pos_weight=torch.zeros(7))


# ---- token-routed attention --------------------------------------------------------------------------------------
def test_token_attention_refuses_projections_of_another_size():
    from memory_b200 import functional as F, ops
    h, routed = torch.zeros(1, 8, D, dtype=torch.bfloat16), torch.zeros(4 * 64, D)
    idx, w = torch.zeros(1, 8, 2, dtype=torch.int32), torch.zeros(1, 8, 2)
    good = {"wq": (D, D), "wk": (64, D), "wv": (64, D), "wo": (D, D)}

    def native(**over):
        return F._TokenRoutedAttention._native(h, None, routed, idx, *(torch.zeros(*s) for s in dict(good, **over).values()),
                                               HEADS, 1, 64, torch.bfloat16)
    assert native()
    for name, shape in (("wv", (128, D)), ("wv", (64, 64)), ("wk", (128, D)), ("wo", (D, 64)), ("wq", (64, D))):
        assert not native(**{name: shape}), (name, shape)
        ws = [torch.zeros(*s) for s in dict(good, **{name: shape}).values()]
        with pytest.raises(ValueError, match="inner dimensions differ"):
            ops.token_attn_fwd(h.view(8, D), None, routed, idx, w, *ws, HEADS, 1, 1.0, False)


def test_listed_chapters_are_read_from_16_byte_rows(monkeypatch):
    """A bank slice that starts anywhere is copied: its rows are converted with 16-byte loads."""
    from types import SimpleNamespace
    from memory_b200 import _lib as L, ops
    seen = []
    fake = SimpleNamespace(moc_token_attn_arena_bytes=lambda s: 16, moc_token_attn_fwd_scratch_bytes=lambda s: 16,
                           moc_token_attn_fwd=lambda s, scratch: seen.append(s._obj.routed) or 0)
    for name, fn in (("lib", lambda: fake), ("stream_ptr", lambda dev: 1), ("require_cuda", lambda *t: None),
                     ("status_word", lambda dev: torch.zeros(1, dtype=torch.int32))):
        monkeypatch.setattr(L, name, fn)
    h, idx, w = torch.zeros(8, D, dtype=torch.bfloat16), torch.zeros(1, 8, 2, dtype=torch.int32), torch.zeros(1, 8, 2)
    ws = [torch.zeros(n, D) for n in (D, 64, 64, D)]
    for bank in (_off_by(torch.zeros(4 * 64, D), 1), _off_by(torch.zeros(4 * 64, D).bfloat16(), 3), torch.zeros(4 * 64, D)):
        _, _, keep = ops.token_attn_fwd(h, None, bank, idx, w, *ws, HEADS, 1, 1.0, False)
        assert seen[-1] == keep[2].data_ptr() and seen[-1] % 16 == 0 and torch.equal(keep[2], bank)
    assert seen[-1] == bank.data_ptr()          # (an aligned one is read where it is)


# ---- decoding ----------------------------------------------------------------------------------------------------
class _FakeLibrary:
    """Stands in for the native library: keeps the descriptors it is called with."""

    def __init__(self):
        self.seen = []

    def moc_decode_step_arena_bytes(self, s):
        return 16

    def moc_decode_step(self, s):
        self.seen.append(bytes(s._obj))
        return 0


@pytest.fixture
def decoder(monkeypatch):
    """A decoder on CPU tensors over the fake library, and what that was called with."""
    from types import SimpleNamespace
    from memory_b200 import MemoryDecoder, _lib as L, functional as F
    fake, status = _FakeLibrary(), torch.zeros(1, dtype=torch.int32)
    for name, fn in (("lib", lambda: fake), ("stream_ptr", lambda dev: 1), ("require_cuda", lambda *t: None),
                     ("status_word", lambda dev: status), ("device_index", lambda dev: 0)):
        monkeypatch.setattr(L, name, fn)
    monkeypatch.setattr(F, "_side_stream", lambda dev, main: 2)
    cache = SimpleNamespace(kv_bank=torch.zeros(9 * 64, 2 * D, dtype=torch.bfloat16), tokens_per_chapter=64)
    bf = torch.zeros(D, D, dtype=torch.bfloat16)
    return MemoryDecoder(cache, torch.zeros(9, D), torch.zeros(9), bf, bf.clone(), num_heads=HEADS, top_k=2), fake


def _decode_states():
    return torch.zeros(2, 1, D, dtype=torch.bfloat16), torch.zeros(2, 16, D, dtype=torch.bfloat16)


@pytest.mark.parametrize("change, where", [
    (dict(routed_scale=7.5), ("router", "routed_scale", 7.5)),
    (dict(num_shared=0), ("router", "num_shared", 0)),
    (dict(top_k=3), ("router", "top_k", 3)),
    (dict(scale=0.5), ("attn", "scale", 0.5)),
    (dict(num_heads=1, num_kv_heads=1), ("attn", "num_heads", 1)),
    (dict(tokens_per_chapter=32), ("attn", "tokens_per_chapter", 32)),
])
def test_a_decoder_changed_between_steps_decodes_with_the_change(decoder, change, where):
    from memory_b200 import _lib as L
    dec, fake = decoder
    dec.step(*_decode_states())
    dec.step(*_decode_states())
    for name, value in change.items():
        setattr(dec.cache if name == "tokens_per_chapter" else dec, name, value)
    dec.step(*_decode_states())
    first, _, last = (L.DecodeStepDesc.from_buffer_copy(b) for b in fake.seen)
    part, field, value = where
    assert getattr(getattr(last, part), field) == value != getattr(getattr(first, part), field)
    assert last.attn.n_chapters == last.router.num_shared + last.router.top_k


@pytest.mark.parametrize("name, tensor, error", [
    ("wq_c", torch.zeros(D, D), TypeError), ("wo_c", torch.zeros(D, D), TypeError),
    ("wq_c", torch.zeros(D, 64, dtype=torch.bfloat16), ValueError),
    ("wo_c", torch.zeros(D, 64, dtype=torch.bfloat16), ValueError),
    ("router_bias", torch.zeros(8), ValueError), ("router_weight", torch.zeros(9, 64), ValueError),
])
def test_a_decoder_refuses_weights_swapped_in_between_steps(decoder, name, tensor, error):
    dec, fake = decoder
    dec.step(*_decode_states())
    setattr(dec, name, tensor)
    with pytest.raises(error):
        dec.step(*_decode_states())
    assert len(fake.seen) == 1


def test_a_decoder_passes_dense_copies_of_strided_weights(decoder):
    from memory_b200 import _lib as L
    dec, fake = decoder
    wide = torch.zeros(D, 2 * D, dtype=torch.bfloat16)
    dec.wq_c = wide[:, :D]
    dec.step(*_decode_states())
    assert L.DecodeStepDesc.from_buffer_copy(fake.seen[0]).wq != wide.data_ptr()


@pytest.mark.gpu
@pytest.mark.parametrize("width", [64, 200])
def test_decoding_with_routing_states_of_another_width(width):
    import memory_b200 as M
    from memory_b200 import _lib as L, ops
    g = torch.Generator().manual_seed(11)
    rnd = lambda *s, scale=1.0: (torch.randn(*s, generator=g) * scale).cuda()      # noqa: E731
    cache = M.ProjectedBankCache(rnd(9 * 64, D), rnd(D, D, scale=0.1), rnd(D, D, scale=0.1), 64)
    dec = M.MemoryDecoder(cache, rnd(9, width), rnd(9), rnd(D, D, scale=0.1), rnd(D, D, scale=0.1), num_heads=HEADS, top_k=3)
    hidden, states = rnd(20, 1, D).bfloat16(), rnd(20, 16, width).bfloat16()
    out, info = dec.step(hidden, states)
    idx, _, cidx, cw, _ = M.route(states, dec.router_weight, dec.router_bias, 3, 1, 2.5, False)
    q = ops.gemm(hidden.view(20, D), dec.wq_c)
    o = ops.decode_attn(q.view(20, 1, D), cache.kv_bank, cidx, cw, HEADS, HEADS, 64, dec.scale)
    want = ops.gemm(o.view(20, D), dec.wo_c).view(20, 1, D)
    L.check_device_status(out.device)
    assert torch.equal(info["indices"], idx) and torch.equal(out, want)            # the same operators, issued singly


def test_the_descriptor_of_a_decoding_step_has_both_widths(decoder):
    from memory_b200 import _lib as L
    dec, fake = decoder
    dec.router_weight = torch.zeros(9, 64)
    dec.step(_decode_states()[0], torch.zeros(2, 16, 64, dtype=torch.bfloat16))
    s = L.DecodeStepDesc.from_buffer_copy(fake.seen[0])
    assert (s.router.hidden_dim, s.hidden_dim) == (64, D)


# ---- sparse attention --------------------------------------------------------------------------------------------
def _off_by(t, n):
    """The same numbers, contiguous, starting ``n`` elements into a buffer."""
    buf = torch.empty(t.numel() + n, dtype=t.dtype, device=t.device)
    return buf[n:].copy_(t.reshape(-1)).view(t.shape)


def test_unaligned_tensors_stay_with_the_kernels_that_take_them():
    from memory_b200 import ops
    q, k = torch.zeros(1, 5, 2, 64, dtype=torch.bfloat16), torch.zeros(1, 128, 2, 64, dtype=torch.bfloat16)
    assert ops.sparse_attn_tc_supported(q, k, 64, k, q)
    for bad in ((_off_by(q, 1), k, k), (q, _off_by(k, 4), k), (q, k, _off_by(k, 7))):
        assert not ops.sparse_attn_tc_supported(bad[0], bad[1], 64, bad[2])


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["q", "k", "v", "do"])
def test_unaligned_tensors_give_the_same_attention(which):
    import memory_b200 as M
    from memory_b200 import _lib as L
    g = torch.Generator().manual_seed(4)
    x = {n: torch.randn(1, r, h, 64, generator=g).bfloat16().cuda() for n, r, h in
         (("q", 33, 4), ("k", 5 * 64, 2), ("v", 5 * 64, 2), ("do", 33, 4))}
    bi = torch.rand(33 * 2, 5, generator=g).topk(2, dim=1).indices.view(1, 33, 2, 2).int().cuda()

    def run(x):
        leaves = [x[n].detach().requires_grad_(True) for n in ("q", "k", "v")]
        o = M.memory_cross_attn(*leaves, bi, 64)
        o.backward(x["do"])
        return [o.detach()] + [t.grad for t in leaves]
    want, got = run(x), run(dict(x, **{which: _off_by(x[which], 3)}))
    L.check_device_status(torch.device("cuda:0"))
    for a, b in zip(got, want):          # bf16 results of two kernels: probabilities rounded to bf16 in one, not in the other
        assert float((a.float() - b.float()).norm() / b.float().norm()) < 1e-2
