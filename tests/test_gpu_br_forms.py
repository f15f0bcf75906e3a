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


@pytest.mark.parametrize("variant,N,beta,digits,batches", [
    (2, 2048, 16, 4, (1, 33, 40, 75, 149, 222, 300)), (2, 1024, 12, 3, (2, 74, 297, 370)), (1, 512, 12, 3, (3, 60, 75, 303)),
    (1, 2048, 20, 3, (5, 150)), (1, 2048, 12, 3, (150, 300)), (0, 1024, 16, 4, (297, 310)), (2, 4096, 12, 3, (1, 150))])
def test_remainders_and_small_batches(native, oracle, variant, N, beta, digits, batches):
    """Full waves and the rest in a wider form, evaluation-domain results and strided accumulators among them."""
    import torch
    n = 4
    rot, key = rotator(variant, N, beta, digits, n, N + variant)
    lwes, accs = inputs(N, n, max(batches), 4)
    lwe, acc = (torch.from_numpy(x.view(np.int64)).cuda() for x in (lwes, accs))

    def run(b, stride, coef):
        out = torch.zeros((b, 2 * N), dtype=torch.int64, device="cuda")
        rot.blind_rotate_batch(out.data_ptr(), lwe.data_ptr(), n + 1, acc.data_ptr(), stride, b, coef)
        rot.check()
        return out.cpu().numpy().view(np.uint64)

    forms = [(b, 0 if b & 1 else 2 * N, b % 3 != 0) for b in batches]
    got = [run(*f) for f in forms]
    rot.set_split(1)  # a launch form set by name: one modular block per rotation
    for f, words in zip(forms, got):
        np.testing.assert_array_equal(words, run(*f))
    b, stride, coef = forms[-1]
    want = oracle.blind_rotate(variant, N, n, beta, digits, key, lwes[b - 1], accs[(b - 1) if stride else 0], int(coef))
    np.testing.assert_array_equal(got[-1][b - 1], want)
