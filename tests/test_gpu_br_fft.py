"""The double-precision rotation kernels (N = 1024, 2048, 4096) against the C oracle and the modular kernels.

Every word has to be equal: the kernel runs only where its error bound proves that each
product coefficient rounds to the exact integer.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = 0xFFFFFFFF00000001
# (variant, N, log2 base, digits): three and four limbs, two to four digits, the largest digits of each limb count
SETS = [(1, 2048, 12, 3), (0, 2048, 14, 4), (1, 2048, 16, 4), (1, 2048, 8, 4), (0, 2048, 12, 3), (1, 1024, 12, 3),
        (0, 1024, 16, 4), (1, 1024, 16, 2), (0, 1024, 8, 2), (1, 4096, 12, 3), (0, 4096, 14, 4), (1, 4096, 8, 2)]
EXTREMES = [0, 1, P - 1, P - 2, P // 2, P // 2 + 1, 1 << 63, (1 << 63) - 1, (1 << 32) - 1]


def rotator(variant, N, beta, digits, n, rng, key=None):
    from fhetoothpaste_b200 import BlindRotationContext, GpuBlindRotator
    ctx = BlindRotationContext(variant, N, n, 1 << beta, digits)
    key = rng.integers(0, P, ctx.key_words(), dtype=np.uint64) if key is None else key
    return GpuBlindRotator(ctx, key), key


def inputs(rng, N, n, batch):
    lwes = rng.integers(0, 2 * N, (batch, n + 1), dtype=np.uint64)
    lwes[0, :3] = (0, N, 2 * N - 1)         # a skipped iteration and the sign boundaries
    lwes[0, n] = N                           # b past the half turn
    accs = rng.integers(0, P, (batch, 2 * N), dtype=np.uint64)
    accs[-1, :len(EXTREMES)] = EXTREMES      # digits at the ends of their range
    accs[-1, N:N + len(EXTREMES)] = EXTREMES
    return lwes, accs


@pytest.mark.parametrize("batch,coef", [(1, True), (15, False), (20, True), (75, False)])
@pytest.mark.parametrize("variant,N,beta,digits", SETS)
def test_equals_oracle(native, oracle, variant, N, beta, digits, batch, coef):
    rng = np.random.default_rng(N + 10 * beta + digits)
    n = 4
    rot, key = rotator(variant, N, beta, digits, n, rng)
    lwes, accs = inputs(rng, N, n, batch)
    before = native.tp_kernel_launches()
    got = rot.blind_rotate_batch_host(lwes, accs, out_coef=coef)
    # clusters of eight, four and (odd batch) pairs or one block each, halves on two blocks at N =
    # 4096; evaluation-domain results
    # are transformed in a second launch
    assert native.tp_kernel_launches() - before == (1 if coef else 2)
    want = oracle.blind_rotate_many(variant, N, n, beta, digits, key, lwes, accs, coef, 4)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("variant,N,beta,digits", SETS[:2] + SETS[5:7] + SETS[9:11])
@pytest.mark.parametrize("batch", [2 * 148 * 2 + 3, 60, 15])
def test_equals_modular_kernel_over_forms(native, variant, N, beta, digits, batch):
    """Strides, a shared accumulator, results in place, more rotations than resident blocks."""
    import torch
    rng = np.random.default_rng(7)
    n = 3
    rot, _ = rotator(variant, N, beta, digits, n, rng)
    lwes, accs = inputs(rng, N, n, batch)
    wide = np.zeros((batch, n + 6), np.uint64)
    wide[:, :n + 1] = lwes
    dev = [torch.from_numpy(x.view(np.int64)).cuda() for x in (wide, accs)]
    out = torch.zeros((batch, 2 * N), dtype=torch.int64, device="cuda")

    def run(stride, coef, in_place):
        dst = dev[1].clone() if in_place else out
        src = dst if in_place else dev[1]
        rot.blind_rotate_batch(dst.data_ptr(), dev[0].data_ptr(), n + 6, src.data_ptr(), stride, batch, coef)
        rot.check()
        return dst.cpu().numpy().copy()

    forms = [(2 * N, True, False), (2 * N, False, True), (0, True, False)]
    fft = [run(*f) for f in forms]
    rot.set_mac_form(rot.mac_form)  # a launch form set by name runs the modular kernels
    for f, got in zip(forms, fft):
        np.testing.assert_array_equal(got, run(*f))


@pytest.mark.parametrize("variant,N,beta,digits", SETS[:2])
def test_key_beyond_the_bound_runs_modular(native, oracle, variant, N, beta, digits):
    """Key coefficients whose limbs are all at their largest fail the error bound: same words, the other kernel."""
    rng = np.random.default_rng(3)
    n, batch = 3, 9
    base = 2642246 if digits == 3 else 1 << 16
    worst = base // 2 - 1
    value = sum(worst * base ** i for i in range(3 if digits == 3 else 4)) % P
    poly = oracle.ntt_forward(np.full(N, value, np.uint64))
    rot, key = rotator(variant, N, beta, digits, n, rng, np.tile(poly, n * (2 if variant else 1) * 4 * digits))
    lwes, accs = inputs(rng, N, n, batch)
    before = native.tp_kernel_launches()
    got = rot.blind_rotate_batch_host(lwes, accs, out_coef=False)
    launched = native.tp_kernel_launches() - before
    assert launched == (1 if digits == 3 else 2)  # four limbs keep room for such keys
    np.testing.assert_array_equal(got, oracle.blind_rotate_many(variant, N, n, beta, digits, key, lwes, accs, False, 4))


def test_out_of_range_words_are_reported(native):
    rng = np.random.default_rng(5)
    rot, _ = rotator(1, 1024, 12, 3, 3, rng)
    lwes, accs = inputs(rng, 1024, 3, 2)
    want = rot.blind_rotate_batch_host(lwes, accs)
    lwes[1, 2] += np.uint64(4096)
    from fhetoothpaste_b200 import TpError
    with pytest.raises(TpError):
        rot.blind_rotate_batch_host(lwes, accs)
    np.testing.assert_array_equal(rot.blind_rotate_batch_host(lwes % np.uint64(2048), accs), want)
