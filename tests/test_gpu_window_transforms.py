"""The routing window slides in one kernel that torch does not see; where torch has to see it, it concatenates as ever."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _window(prompt):
    import memory_b200 as M
    w = M.RoutingWindow(6, "hybrid")
    w.prefill(prompt)
    return w


def _inputs():
    g = torch.Generator().manual_seed(8)
    return [torch.randn(2, n, 16, generator=g).cuda() for n in (9, 2, 2)]


def test_a_traced_step_follows_its_input():
    prompt, first, second = _inputs()
    traced = torch.jit.trace(lambda p, h: _window(p).step(h), (prompt, first))
    assert torch.equal(traced(prompt, second), torch.cat([prompt[:, -4:], second], dim=1))


def test_forward_mode_gradients_pass_through():
    from torch.autograd import forward_ad as fw
    prompt, h, tangent = _inputs()
    with torch.no_grad(), fw.dual_level():
        out = fw.unpack_dual(_window(prompt).step(fw.make_dual(h, tangent)))
    assert torch.equal(out.primal, torch.cat([prompt[:, -4:], h], dim=1))
    assert torch.equal(out.tangent[:, 4:], tangent) and not out.tangent[:, :4].any()


def test_vmap_over_the_new_states():
    prompt, first, second = _inputs()
    with torch.no_grad():
        out = torch.func.vmap(lambda h: _window(prompt).step(h))(torch.stack([first, second]))
    assert torch.equal(out, torch.stack([torch.cat([prompt[:, -4:], h], dim=1) for h in (first, second)]))
