"""The router of one or two sequences in one launch: the same bits as the kernels that take three sequences, at the edges of what the
launch takes (widths, chapters, positions) and just beyond, and a decoding step whose queries go along."""
import pytest
import torch

pytestmark = pytest.mark.gpu
FIELDS = ("pooled", "logits", "probs", "idx", "weights", "comb_idx", "comb_w", "row_stats")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("seq,d,chapters,k,shared", [(1, 64, 5, 4, 1), (33, 256, 65, 4, 0), (1024, 768, 4097, 64, 1), (1025, 768, 300, 8, 2),
                                                     (128, 1024, 2049, 300, 1), (31, 1024, 9216, 16, 1), (7, 120, 9217, 16, 3), (40, 264, 5121, 1, 1)])
def test_same_bits_as_three_sequences(seq, d, chapters, k, shared, dtype):
    from memory_b200 import _lib as L, ops
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(seq + d)
    h = torch.randn(3, seq, d, generator=g, device=dev).to(dtype)
    w = torch.randn(chapters, d, generator=g, device=dev)
    b = torch.randn(chapters, generator=g, device=dev)
    want = ops.router_fwd(h, w, b, k, shared, 2.5, False)
    for n in (1, 2):
        got = ops.router_fwd(h[:n].contiguous(), w, b, k, shared, 2.5, False)
        for f in FIELDS:
            assert torch.equal(got[f], want[f][:n]), (n, f)
    L.check_device_status(dev)


@pytest.mark.parametrize("n_q", [1, 2])
@pytest.mark.parametrize("d", [64, 768, 1024])
def test_decoding_step(d, n_q):
    import memory_b200 as M
    from memory_b200 import _lib as L
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(d)
    rand = lambda *s: torch.randn(*s, generator=g, device=dev)
    heads, c = d // 64, 40
    cache = M.ProjectedBankCache(rand(c * 64, d), rand(d, d) * 0.05, rand(d, d) * 0.05, 64, 1)
    dec = M.MemoryDecoder(cache, rand(c, d), None, rand(d, d) * 0.05, rand(d, d) * 0.05, num_heads=heads, top_k=8)
    h, states = rand(3, n_q, d).bfloat16(), rand(3, 50, d).bfloat16()
    want, wi = dec.step(h, states)
    for n in (1, 2):
        out, info = dec.step(h[:n].contiguous(), states[:n].contiguous())
        assert torch.equal(info["indices"], wi["indices"][:n]) and torch.equal(info["weights"], wi["weights"][:n])
        # (the attention's clusters split the keys by the number of sequences: fp32 sums in another order, one bf16 rounding)
        assert (out.float() - want[:n].float()).abs().max() <= 2 ** -7 * want.float().abs().max()
    L.check_device_status(dev)
