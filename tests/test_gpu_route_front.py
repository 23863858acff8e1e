"""A decoding step of one or two rows routes in one launch: the same bits as the kernels that take three sequences, at the edges of
what the launch takes (widths, chapters, positions) and just beyond, and when it is captured."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _decoder(d, c, k, shared, states_d=None, bias=False):
    import memory_b200 as M
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(d + c)
    rand = lambda *s: torch.randn(*s, generator=g, device=dev)
    cache = M.ProjectedBankCache(rand(c * 8, d), rand(d, d) * 0.05, rand(d, d) * 0.05, 8, shared)
    dec = M.MemoryDecoder(cache, rand(c, states_d or d), rand(c) if bias else None, rand(d, d) * 0.05, rand(d, d) * 0.05,
                          num_heads=d // 64, top_k=k, num_shared_chapters=shared)
    return dec, rand


def _check(out, info, want, wi, n):
    for key in ("indices", "weights", "combined_indices", "combined_weights"):
        assert torch.equal(info[key], wi[key][:n]), key
    # (the attention's clusters split the keys by the number of sequences: fp32 sums in another order, roundings to bf16)
    assert (out.float() - want[:n].float()).abs().max() <= 2 ** -6 * want.float().abs().max()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("seq,d,states_d,chapters,k,shared", [(1, 64, 64, 5, 4, 1), (33, 256, 256, 65, 4, 0), (1024, 768, 768, 4097, 64, 1), (1025, 768, 768, 300, 8, 2),
                                                              (128, 1024, 1024, 2049, 300, 1), (31, 64, 1024, 9216, 16, 1), (7, 64, 120, 9217, 16, 3),
                                                              (40, 128, 264, 5121, 1, 1), (9, 1088, 1088, 40, 8, 1), (9, 64, 1032, 40, 8, 1)])
def test_same_bits_as_three_sequences(seq, d, states_d, chapters, k, shared, dtype):
    from memory_b200 import _lib as L
    dec, rand = _decoder(d, chapters, k, shared, states_d, bias=True)
    h, states = rand(3, 1, d).bfloat16(), rand(3, seq, states_d).to(dtype)
    want, wi = dec.step(h, states)
    for n in (1, 2):
        _check(*dec.step(h[:n].contiguous(), states[:n].contiguous()), want, wi, n)
    L.check_device_status(torch.device("cuda:0"))


@pytest.mark.parametrize("n_q", [1, 2])
def test_two_tokens_and_captured_steps(n_q):
    dec, rand = _decoder(128, 40, 8, 1)
    h, states = rand(3, n_q, 128).bfloat16(), rand(3, 50, 128).bfloat16()
    want, wi = dec.step(h, states)
    one, s1 = h[:1].contiguous(), states[:1].contiguous()
    _check(*dec.step(one, s1), want, wi, 1)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out, info = dec.step(one, s1)
    graph.replay()
    _check(out, info, want, wi, 1)


def test_the_launches_of_a_step_are_those_it_made():
    """One or two rows: router and queries, attention, output projection.  Captured steps, more rows and states that start off a
    16-byte boundary take pooling (of long windows in two kernels), logits, selection and queries apart; fp32 states are cast first."""
    from memory_b200 import ops
    dec, rand = _decoder(128, 40, 8, 1)
    h, states = rand(3, 1, 128).bfloat16(), rand(3, 1100, 128).bfloat16()

    def launches(rows, window, dtype=torch.bfloat16, off=0):
        r = torch.empty(rows * window * 128 + off, dtype=torch.bfloat16, device=h.device)[off:].view(rows, window, 128)
        r.copy_(states[:rows, :window])
        x = h[:rows].to(dtype).contiguous()
        before = ops.LAUNCHES
        dec.step(x, r)
        return ops.LAUNCHES - before

    assert launches(1, 50) == launches(2, 50) == 3
    assert launches(1, 50, torch.float32) == 4
    assert launches(3, 50) == 6 and launches(3, 50, torch.float32) == 7
    assert launches(1, 50, off=1) == launches(1, 1100) == 7
    with torch.cuda.graph(torch.cuda.CUDAGraph()):
        captured = launches(1, 50)
    assert captured == 6
