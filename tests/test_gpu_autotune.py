"""The autotuner times the form that is chosen by batch size beside the named ones, for sets without a
double-precision kernel too, and keeps it where it is the fastest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = 0xFFFFFFFF00000001


def rotator(variant, N, beta, digits, n):
    from fhetoothpaste_b200 import BlindRotationContext, GpuBlindRotator
    ctx = BlindRotationContext(variant, N, n, 1 << beta, digits)
    return GpuBlindRotator(ctx, np.random.default_rng(N).integers(0, P, ctx.key_words(), dtype=np.uint64))


def runner(rot, N, n, batch):
    import torch
    rng = np.random.default_rng(batch)
    lwe, acc = (torch.from_numpy(x.view(np.int64)).cuda() for x in
                (rng.integers(0, 2 * N, (batch, n + 1), dtype=np.uint64), rng.integers(0, P, (batch, 2 * N), dtype=np.uint64)))
    out = torch.zeros_like(acc)

    def run():
        rot.blind_rotate_batch(out.data_ptr(), lwe.data_ptr(), n + 1, acc.data_ptr(), 2 * N, batch, True,
                               torch.cuda.current_stream().cuda_stream)
        return out
    return run


# batches whose rest behind full waves runs in a wider form: two launches while the form is open
@pytest.mark.parametrize("variant,N,beta,digits,n,batch", [(2, 2048, 16, 4, 16, 512), (1, 8192, 12, 3, 8, 100)])
def test_remainders_survive(native, variant, N, beta, digits, n, batch):
    rot = rotator(variant, N, beta, digits, n)
    run = runner(rot, N, n, batch)

    def launches():
        before = native.tp_kernel_launches()
        run()
        rot.check()
        return native.tp_kernel_launches() - before
    want = run().clone()
    assert launches() == 2
    rot.autotune(batch)
    assert launches() == 2
    rot.set_split(1)
    rot.autotune(batch)  # also from a form set by name
    assert launches() == 2
    assert np.array_equal(run().cpu().numpy(), want.cpu().numpy())


def test_one_rotation_of_a_large_ring(native):
    """One rotation of N = 8192 on eight blocks takes a third of its time on the default two."""
    import torch
    N, n = 8192, 16
    rot = rotator(1, N, 12, 3, n)
    run = runner(rot, N, n, 1)

    def ms():
        times = []
        for _ in range(7):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            run()
            e1.record()
            torch.cuda.synchronize()
            times.append(e0.elapsed_time(e1))
        return sorted(times)[3]
    before = ms()
    rot.autotune(1)
    assert ms() < 1.5 * before
