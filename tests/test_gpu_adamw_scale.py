"""A gradient scale that is no number (a norm that overflowed, a loss that is NaN) spoils what has a gradient, no more."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [math.inf, math.nan, 0.0])
def test_chapters_without_a_gradient_ignore_its_scale(scale):
    from memory_b200 import _lib as L, ops
    t, d, chapters = 4, 40, 9
    g = torch.Generator().manual_seed(6)
    start = [torch.rand(chapters * t, d, generator=g).cuda() for _ in range(3)]
    uniq = torch.tensor([2, 5], dtype=torch.int32, device="cuda")
    rows = torch.randn(2 * t, d, generator=g).cuda()

    def step(n, scale):
        state = [x.clone() for x in start]
        ops.bank_adamw_step(*state, uniq, torch.tensor([n], dtype=torch.int32, device="cuda"), rows, t, lr=0.1, step=3,
                            grad_scale=scale)
        return [x.view(chapters, t, d) for x in state]
    got, want = step(2, scale), step(0, 1.0)
    L.check_device_status(uniq.device)
    for a, b in zip(got, want):
        rest = [c for c in range(chapters) if c not in (2, 5)]
        assert torch.equal(a[rest], b[rest])
        assert scale == 0.0 or not a[[2, 5]].isfinite().all()
