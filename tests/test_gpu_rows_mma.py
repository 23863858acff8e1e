"""Projections of some rows: remainders of the 16-column, 32-row tiles and of the K steps, both sides of the rules that choose between
the warps a column, the matrix instructions and the tensor-core tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("out", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("m,n,k", [(24, 1024, 768), (24, 1023, 768), (33, 1000, 8), (64, 771, 24), (63, 2048, 1024), (256, 768, 520),
                                   (256, 769, 512), (250, 768, 768), (257, 512, 768), (100, 1700, 1000), (31, 800, 1032),
                                   (8, 3072, 768), (9, 3071, 768), (1, 65536, 64), (3, 24001, 72), (16, 6145, 128), (65, 360, 520), (256, 64, 1024)])
def test_projection(m, n, k, out):
    from memory_b200 import _lib as L, ops
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(m + n + k)
    a, b = (torch.randn(r, k, generator=g, device=dev).bfloat16() for r in (m, n))
    got = ops.gemm(a, b, out_dtype=out)
    want = a.double() @ b.double().t()
    L.check_device_status(dev)
    # fp32 sums of k products of random signs; half an ulp of bf16 where the result is rounded
    bound = 2e-6 * k ** 0.5 * want.abs().max() + (2 ** -8 * want.abs() if out == torch.bfloat16 else 0)
    assert ((got.double() - want).abs() <= bound).all()
