"""The double-precision key-switch kernel (packing, trace; N = 1024, 2048) against the oracle and the modular kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = 0xFFFFFFFF00000001
EXTREMES = [0, 1, P - 1, P - 2, P // 2, P // 2 + 1, 1 << 63, (1 << 32) - 1]


def packer(N, beta, digits, rng, key=None):
    from fhetoothpaste_b200 import GpuLWEtoRLWEPacker
    words = (N.bit_length() - 1) * digits * 2 * N
    key = rng.integers(0, P, words, dtype=np.uint64) if key is None else key
    return GpuLWEtoRLWEPacker(N, 1 << beta, digits, key), key


def lwes(rng, rows, N):
    x = rng.integers(0, P, (rows, N + 1), dtype=np.uint64)
    x[0, :len(EXTREMES)] = EXTREMES
    return x


# three and four limbs, two to four digits; 300 packs of two: more merges than resident blocks
@pytest.mark.parametrize("N,beta,digits", [(2048, 16, 4), (1024, 16, 4), (2048, 8, 4), (1024, 12, 3), (2048, 16, 2)])
def test_equals_modular_kernel(native, N, beta, digits):
    rng = np.random.default_rng(N + beta)
    fft, key = packer(N, beta, digits, rng)
    mod, _ = packer(N, beta, digits, rng, key)
    mod.set_tile(8)
    for packs, length in ((300, 2), (3, 16)):
        x = lwes(rng, packs * length, N)
        np.testing.assert_array_equal(fft.Pack(x, length), mod.Pack(x, length))
    for length in (2, 5):  # empty siblings
        x = lwes(rng, 2 * length, N)
        np.testing.assert_array_equal(fft.PackConsecutively(x, length), mod.PackConsecutively(x, length))


@pytest.mark.parametrize("N,beta,digits", [(1024, 16, 4), (2048, 12, 3)])
def test_equals_oracle(native, oracle, N, beta, digits):
    rng = np.random.default_rng(N)
    pk, key = packer(N, beta, digits, rng)
    x = lwes(rng, 4, N)
    before = native.tp_kernel_launches()
    got = pk.Pack(x, 4)[0]
    # the first level sets its leaves up itself: two merge levels and the traces, no set-up launch
    assert native.tp_kernel_launches() - before == 2 + (N.bit_length() - 1 - 2)
    np.testing.assert_array_equal(got, oracle.pack(N, beta, digits, key, x, len(x)))


def test_key_beyond_the_bound_runs_modular(native, oracle):
    """All limbs at their largest with three limbs fails the bound (the largest base that takes three)."""
    rng = np.random.default_rng(4)
    N, beta, digits = 2048, 14, 3
    worst = 2642246 // 2 - 1
    poly = oracle.ntt_forward(np.full(N, sum(worst * 2642246 ** i for i in range(3)) % P, np.uint64))
    pk, key = packer(N, beta, digits, rng, np.tile(poly, 11 * digits * 2))
    x = lwes(rng, 2, N)
    before = native.tp_kernel_launches()
    got = pk.Pack(x, 2)[0]
    assert native.tp_kernel_launches() - before == 12  # the set-up launch of the modular form, 11 levels
    np.testing.assert_array_equal(got, oracle.pack(N, beta, digits, key, x, len(x)))
