"""A bounded wait that runs out inside an LWE key switch: reported once, by the next call, graph launch or check; the
context is usable afterwards. The wait is a kernel's on a barrier that nothing completes, with a short limit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = 0xFFFFFFFF00000001
TIMEOUT = 4


def raises_timeout(call):
    from fhetoothpaste_b200 import TpError
    with pytest.raises(TpError) as e:
        call()
    assert e.value.status == TIMEOUT


def test_reported_once(native):
    import torch
    from fhetoothpaste_b200 import BlindRotationContext, GpuBlindRotator, GpuLWEtoLWEConverter, _native
    rng = np.random.default_rng(1)
    N, n, batch = 256, 8, 3
    conv = GpuLWEtoLWEConverter(N, n, 1 << 16, 4, rng.integers(0, P, N * 4 * (n + 1), dtype=np.uint64))
    ctx = BlindRotationContext(0, N, n, 1 << 16, 4)
    rot = GpuBlindRotator(ctx, rng.integers(0, P, ctx.key_words(), dtype=np.uint64))
    x = torch.from_numpy(rng.integers(0, P, (batch, N + 1), dtype=np.uint64).view(np.int64)).cuda()
    lwe = torch.from_numpy(rng.integers(0, 2 * N, (batch, n + 1), dtype=np.uint64).view(np.int64)).cuda()
    acc = torch.from_numpy(rng.integers(0, P, 2 * N, dtype=np.uint64).view(np.int64)).cuda()
    rl = torch.zeros((batch, 2 * N), dtype=torch.int64, device="cuda")
    out, want, boot = (torch.zeros((batch, n + 1), dtype=torch.int64, device="cuda") for _ in range(3))

    def switch(dst):
        dst.zero_()
        torch.cuda.synchronize()
        conv.convert_batch(batch, dst.data_ptr(), x.data_ptr())
        torch.cuda.synchronize()

    def run_out():
        _native.check(native.tp_debug_lwe_timeout(conv._h, None))
        torch.cuda.synchronize()
    switch(want)
    graph = rot.capture_bootstrap(conv, batch, rl.data_ptr(), lwe.data_ptr(), acc.data_ptr(), 0, boot.data_ptr())
    graph.launch()
    rot.check()
    first = boot.clone()
    run_out()
    raises_timeout(lambda: switch(out))
    switch(out)
    assert torch.equal(out, want)
    run_out()
    raises_timeout(graph.launch)
    graph.launch()
    rot.check()
    run_out()
    raises_timeout(rot.check)
    graph.launch()
    rot.check()
    assert torch.equal(boot, first)
    graph.close()


def test_scalar_contexts_have_no_wait(native):
    from fhetoothpaste_b200 import GpuLWEtoLWEConverter
    conv = GpuLWEtoLWEConverter(8, 2, 1 << 20, 3, np.zeros(8 * 3 * 3, np.uint64))  # digits above 16 bits
    assert native.tp_debug_lwe_timeout(conv._h, None) == 6
