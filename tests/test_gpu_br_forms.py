"""Rotation launch forms chosen by batch size against the form named by hand: the same words."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = 0xFFFFFFFF00000001


def rotator(variant, N, beta, digits, n, seed):
    from fhetoothpaste_b200 import BlindRotationContext, GpuBlindRotator
    ctx = BlindRotationContext(variant, N, n, 1 << beta, digits)
    key = np.random.default_rng(seed).integers(0, P, ctx.key_words(), dtype=np.uint64)
    return GpuBlindRotator(ctx, key), key


def inputs(N, n, batch, seed):
    rng = np.random.default_rng(seed)
    lwes = rng.integers(0, 2 * N, (batch, n + 1), dtype=np.uint64)
    lwes[0, :2] = (0, N)
    return lwes, rng.integers(0, P, (batch, 2 * N), dtype=np.uint64)


@pytest.mark.parametrize("variant,N,beta,digits,batches", [
    (0, 8192, 14, 4, (1, 16, 75)), (1, 8192, 12, 3, (1, 15, 17, 33)), (1, 8192, 20, 3, (2, 16)),
    (2, 8192, 16, 4, (1, 16, 75)), (0, 16384, 16, 4, (1, 16)), (1, 16384, 8, 2, (1, 16)), (2, 16384, 14, 4, (1, 9))])
def test_large_rings_on_wider_clusters(native, oracle, variant, N, beta, digits, batches):
    n = 4
    rot, key = rotator(variant, N, beta, digits, n, N + variant)
    lwes, accs = inputs(N, n, max(batches), 3)
    got = [rot.blind_rotate_batch_host(lwes[:b], accs[:b], out_coef=bool(b & 1)) for b in batches]
    rot.set_mac_form(rot.mac_form)  # a launch form set by name: the default clusters
    for b, words in zip(batches, got):
        np.testing.assert_array_equal(words, rot.blind_rotate_batch_host(lwes[:b], accs[:b], out_coef=bool(b & 1)))
    want = oracle.blind_rotate(variant, N, n, beta, digits, key, lwes[0], accs[0], batches[0] & 1)
    np.testing.assert_array_equal(got[0][0], want)
