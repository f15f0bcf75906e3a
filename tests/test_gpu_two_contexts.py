"""Contexts of one ring and different LWE dimensions share kernels: a later, smaller one leaves the first usable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = 0xFFFFFFFF00000001


# one set per kernel family: double precision (N = 1024, 4096), modular (512, BMMP 2048), a cluster ring
@pytest.mark.parametrize("variant,N,beta,digits", [(1, 1024, 12, 3), (0, 4096, 14, 2), (1, 512, 12, 3), (2, 2048, 16, 3), (0, 8192, 16, 2)])
def test_smaller_context_created_later(native, oracle, variant, N, beta, digits):
    from fhetoothpaste_b200 import BlindRotationContext, GpuBlindRotator
    rng = np.random.default_rng(N)
    n, batch = 600, 80
    ctx = BlindRotationContext(variant, N, n, 1 << beta, digits)
    key = rng.integers(0, P, ctx.key_words(), dtype=np.uint64)
    rot = GpuBlindRotator(ctx, key)
    small = BlindRotationContext(variant, N, 2, 1 << beta, digits)
    GpuBlindRotator(small, rng.integers(0, P, small.key_words(), dtype=np.uint64))
    lwes = np.zeros((batch, n + 1), np.uint64)  # iterations at 0 are skipped: the oracle's time
    lwes[:, rng.integers(0, n, 4)] = rng.integers(1, 2 * N, (batch, 4), dtype=np.uint64)
    acc = rng.integers(0, P, 2 * N, dtype=np.uint64)
    got = [rot.blind_rotate_batch_host(lwes[:b], acc, out_coef=True) for b in (1, 20, batch)]
    for setter, value in ((rot.set_tile, 8), (rot.set_tile, 4), (rot.set_split, 2), (rot.set_split, 4)):
        try:
            setter(value)
        except Exception:  # not built for the set
            continue
        np.testing.assert_array_equal(rot.blind_rotate_batch_host(lwes[:3], acc, out_coef=True), got[-1][:3])
    want = oracle.blind_rotate_many(variant, N, n, beta, digits, key, lwes[:1], acc[None, :], True, 1)
    for words in got:
        np.testing.assert_array_equal(words[0], want[0])
        np.testing.assert_array_equal(words, got[-1][:len(words)])
