"""The LWE key switch at the ends of what a context accepts, against the C oracle: contractions past 64 splits of the
exact length, more words than the grid has tiles for, several passes over the batch, and the largest 32-bit sums."""
import numpy as np
import pytest

from test_gpu_lwe_mma import P, expected, run

pytestmark = pytest.mark.gpu


# n_in l just past 64 x 258 x 128 = 2,113,536 with one and two digit planes; words past 65535 tiles of 32
@pytest.mark.parametrize("n_in,n_out,beta,digits,batch", [(264200, 1, 8, 8, 3), (528400, 2, 16, 4, 2), (1, 65535 * 32, 8, 1, 2)])
def test_ends_of_the_range(native, oracle, n_in, n_out, beta, digits, batch):
    rng = np.random.default_rng(n_in)
    width = n_in + 1
    key = rng.integers(0, P, n_in * digits * (n_out + 1), dtype=np.uint64)
    import torch
    from fhetoothpaste_b200 import GpuLWEtoLWEConverter
    conv = GpuLWEtoLWEConverter(n_in, n_out, 1 << beta, digits, key)
    x = rng.integers(0, P, (batch, width), dtype=np.uint64)
    out = rng.integers(0, P, (batch, n_out + 1), dtype=np.uint64)
    got = torch.from_numpy(out.view(np.int64)).cuda()
    conv.convert_batch(batch, got.data_ptr(), torch.from_numpy(x.view(np.int64)).cuda().data_ptr())
    torch.cuda.synchronize()
    b = batch - 1
    np.testing.assert_array_equal(got[b].cpu().numpy().view(np.uint64).astype(object),
                                  expected(oracle, n_in, n_out, beta, digits, key, x[b], out[b]))


def test_several_passes(native, oracle):
    """More than 256 MB of digit planes: 16384 ciphertexts a pass at n_in l = 8192 in two planes."""
    rng = np.random.default_rng(6)
    n_in, n_out, beta, digits, batch = 2048, 3, 16, 4, 2 * 16384 + 5
    before = native.tp_kernel_launches()
    key, x, out, got = run(n_in, n_out, beta, digits, batch, rng)
    assert native.tp_kernel_launches() - before == 2 + 3 * 3  # the key's constants and bytes; three passes
    for b in (0, 16383, 16384, 32767, 32768, batch - 1):
        np.testing.assert_array_equal(got[b].astype(object), expected(oracle, n_in, n_out, beta, digits, key, x[b], out[b]))


@pytest.mark.parametrize("beta,digits", [(16, 4), (8, 8)])
def test_largest_sums(native, oracle, beta, digits):
    """258 steps of K in one split (so many tiles that the plan leaves K whole: test_lwe_mma_plan_cpu), digits of which
    all bytes but the last digit's are 255 and key bytes of 255 but one each: sums within 10% of 255^2 K < 2^31."""
    import torch
    from fhetoothpaste_b200 import GpuLWEtoLWEConverter
    n_in, n_out, batch = 258 * 128 // digits, 37 * 32 - 1, 4 * 128
    word = 0xFFFFFFFE_FFFFFFFF
    assert word < P
    key = np.full(n_in * digits * (n_out + 1), word, np.uint64)
    conv = GpuLWEtoLWEConverter(n_in, n_out, 1 << beta, digits, key)
    # the digits are those of x + corr, corr = sum_j 2^(beta j + beta - 1): take x + corr = word
    corr = sum(1 << (beta * j + beta - 1) for j in range(64 // beta)) % P
    x = np.full((batch, n_in + 1), (word - corr) % P, np.uint64)
    out = np.zeros((batch, n_out + 1), np.uint64)
    got = torch.from_numpy(out.view(np.int64)).cuda()
    conv.convert_batch(batch, got.data_ptr(), torch.from_numpy(x.view(np.int64)).cuda().data_ptr())
    torch.cuda.synchronize()
    want = expected(oracle, n_in, n_out, beta, digits, key, x[0], out[0]).astype(np.uint64)
    assert np.array_equal(got.cpu().numpy().view(np.uint64), np.broadcast_to(want, out.shape))
