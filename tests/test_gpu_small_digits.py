"""The integer pass 0 of the digit transforms at the ends of the digits' range, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = 0xFFFFFFFF00000001


def words(rng, beta, *shape):
    """Words whose base-2^beta digits, from the top, are at and next to the ends and the middle of their range."""
    ends = np.array([0, 1, (1 << beta) - 1, 1 << (beta - 1), (1 << (beta - 1)) - 1, 1 << (beta - 2), 3 << (beta - 2)], np.uint64)
    x = np.zeros(shape, np.uint64)
    for shift in range(64 - beta, -1, -beta):
        x |= rng.choice(ends, shape) << np.uint64(shift)
    return x % np.uint64(P)


@pytest.mark.parametrize("N,beta,digits", [(128, 16, 4), (256, 15, 4), (1024, 16, 4), (2048, 16, 2), (4096, 14, 4), (2048, 17, 3),
                                           (8192, 16, 4)])
def test_rlwe_switch(native, oracle, N, beta, digits):
    from fhetoothpaste_b200 import GpuRLWEtoRLWEConverter
    rng = np.random.default_rng(N + beta)
    key = rng.integers(0, P, digits * 2 * N, dtype=np.uint64)
    x, base = words(rng, beta, 3, 2 * N), rng.integers(0, P, (3, 2 * N), dtype=np.uint64)
    out = base.copy()
    GpuRLWEtoRLWEConverter(N, 1 << beta, digits, key).Convert(out, x)
    for b in range(3):
        np.testing.assert_array_equal(out[b], oracle.rlwe_ks(N, beta, digits, key, x[b], out=base[b]))


@pytest.mark.parametrize("split", [1, 2, 4])
@pytest.mark.parametrize("variant,N,beta,digits", [(2, 2048, 16, 4), (2, 1024, 15, 4), (1, 512, 16, 3), (0, 256, 15, 4), (0, 256, 14, 4),
                                                   (0, 512, 16, 4)])
def test_rotation(native, oracle, variant, N, beta, digits, split):
    from fhetoothpaste_b200 import BlindRotationContext, GpuBlindRotator
    rng = np.random.default_rng(N + beta)
    n = 4
    ctx = BlindRotationContext(variant, N, n, 1 << beta, digits)
    key = rng.integers(0, P, ctx.key_words(), dtype=np.uint64)
    rot = GpuBlindRotator(ctx, key)
    rot.set_split(split)
    lwes = rng.integers(0, 2 * N, (3, n + 1), dtype=np.uint64)
    lwes[:, n] = 0
    accs = words(rng, beta, 3, 2 * N)
    got = rot.blind_rotate_batch_host(lwes, accs, out_coef=True)
    np.testing.assert_array_equal(got, oracle.blind_rotate_many(variant, N, n, beta, digits, key, lwes, accs, True, 3))


# two to four digits with and without integer first levels; more items than resident blocks; unaligned and in place
@pytest.mark.parametrize("N,beta,digits", [(1024, 16, 4), (1024, 20, 3), (2048, 16, 4), (2048, 8, 2), (4096, 12, 3), (4096, 20, 3)])
def test_staged_switch_equals_the_general_kernel(native, N, beta, digits):
    import torch
    from fhetoothpaste_b200 import GpuRLWEtoRLWEConverter
    rng = np.random.default_rng(N + digits)
    key = rng.integers(0, P, digits * 2 * N, dtype=np.uint64)
    conv, ref = (GpuRLWEtoRLWEConverter(N, 1 << beta, digits, key) for _ in range(2))
    ref.set_tile(4)  # a tile set by name runs the general kernel
    batch = 148 * (4096 // N) + 3
    x = torch.from_numpy(rng.integers(0, P, (batch, 2 * N), dtype=np.uint64).view(np.int64)).cuda()
    base = torch.from_numpy(rng.integers(0, P, (batch, 2 * N), dtype=np.uint64).view(np.int64)).cuda()
    for items in (1, batch):
        want, got = base.clone(), base.clone()
        ref.convert_batch(items, want.data_ptr(), x.data_ptr())
        conv.convert_batch(items, got.data_ptr(), x.data_ptr())
        torch.cuda.synchronize()
        assert torch.equal(got, want)
    odd = torch.zeros(batch * 2 * N + 1, dtype=torch.int64, device="cuda")
    odd[1:] = base.flatten()
    conv.convert_batch(batch, odd.data_ptr() + 8, x.data_ptr())
    same, named = x.clone(), x.clone()
    conv.convert_batch(batch, same.data_ptr(), same.data_ptr())
    ref.convert_batch(batch, named.data_ptr(), named.data_ptr())
    torch.cuda.synchronize()
    assert torch.equal(odd[1:].view(batch, 2 * N), want) and torch.equal(same, named)
