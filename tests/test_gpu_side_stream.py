"""A pass that is refused after it forked its second stream leaves that stream joined: the buffers it gives back may still be
written there, and the allocator orders their next use behind the caller's stream alone."""
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rnd(*s, dtype=torch.bfloat16):
    return torch.randn(*s, generator=torch.Generator().manual_seed(1)).to(dtype).cuda()


def _layer(d, heads, seq):
    from memory_b200 import functional as F
    p = [_rnd(9 * 64, d, dtype=torch.float32), _rnd(9, d, dtype=torch.float32), None] + [_rnd(d, d) for _ in range(4)]
    h = _rnd(2, seq, d).requires_grad_(True)
    return F.memory_layer(h, h, *p, num_heads=heads, num_kv_heads=None, tokens_per_chapter=64, top_k=2)[0]


def _layer_forward():
    return lambda: _layer(64, 2, 64)                              # head_dim 32: refused behind the router


def _layer_backward():
    out = _layer(128, 2, 40)                                      # 40 queries: refused behind a weight gradient
    return lambda: out.sum().backward()


def _attention_backward():
    from memory_b200 import functional as F
    out = F.cross_attention(_rnd(2, 40, 128).requires_grad_(True), _rnd(2, 64, 128), *[_rnd(128, 128) for _ in range(4)], 2)
    return lambda: out.sum().backward()


def _decode():
    from types import SimpleNamespace
    import memory_b200 as M
    cache = SimpleNamespace(kv_bank=_rnd(9 * 64, 128), tokens_per_chapter=64)
    dec = M.MemoryDecoder(cache, _rnd(9, 16, dtype=torch.float32), None, _rnd(64, 12), _rnd(12, 64), num_heads=1, top_k=2)
    hidden, states = _rnd(20, 1, 12, dtype=torch.float32), _rnd(20, 16, 16)
    return lambda: dec.step(hidden, states)                       # 12 columns: refused behind their conversion


@pytest.mark.parametrize("prepare", [_layer_forward, _layer_backward, _attention_backward, _decode])
def test_a_refused_pass_leaves_the_second_stream_joined(prepare):
    from memory_b200 import _lib as L, functional as F
    dev = torch.device("cuda:0")
    with pytest.raises((ValueError, RuntimeError)):
        prepare()()                                               # (kernels are loaded on their first launch, which waits)
    run = prepare()
    torch.cuda.synchronize()
    side = torch.cuda.ExternalStream(F._side_stream(0, L.stream_ptr(dev)))
    with torch.cuda.stream(side):
        torch.cuda._sleep(1_500_000_000)                          # most of a second
    with pytest.raises((ValueError, RuntimeError)):
        run()
    done = torch.cuda.Event()
    done.record()
    time.sleep(0.05)
    assert not done.query()
    torch.cuda.synchronize()
    L.check_device_status(dev)


def test_passes_from_threads_that_come_and_go():
    """Each thread has events of its own and gives them back; streams and results stay as they are."""
    import threading
    want, got = _layer(128, 2, 64).detach(), []

    def work(stream):
        with torch.cuda.stream(stream):
            got.append(_layer(128, 2, 64).detach())
    for _ in range(3):
        threads = [threading.Thread(target=work, args=(torch.cuda.Stream(),)) for _ in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    torch.cuda.synchronize()
    assert len(got) == 12 and all(torch.equal(g, want) for g in got)
    assert torch.equal(_layer(128, 2, 64).detach(), want)
