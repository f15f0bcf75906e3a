"""Parameter sets at the edge of three limbs: keys of ordinary length run the double-precision kernel (with four),
and a key that no limb count serves leaves no transforms behind."""
import numpy as np
import pytest

from test_gpu_br_fft import inputs, rotator
from test_gpu_recorded_keys import worst_poly

pytestmark = pytest.mark.gpu

P = 0xFFFFFFFF00000001


# the error bound holds with three limbs up to 1.076 and 1.067 of the mean squared norm; the largest of this many
# random limb polynomials lies near 1.11
@pytest.mark.parametrize("variant,N,beta,digits", [(0, 1024, 13, 4), (1, 1024, 14, 2)])
def test_edge_sets_run_double_precision(native, oracle, variant, N, beta, digits):
    rng = np.random.default_rng(N + beta)
    n = 300
    rot, key = rotator(variant, N, beta, digits, n, rng)
    lwes, accs = inputs(rng, N, n, 2)
    before = native.tp_kernel_launches()
    got = rot.blind_rotate_batch_host(lwes, accs, out_coef=False)
    assert native.tp_kernel_launches() - before == 2  # the modular kernel makes evaluations in one
    np.testing.assert_array_equal(got, oracle.blind_rotate_many(variant, N, n, beta, digits, key, lwes, accs, False, 2))


def test_unused_transforms_are_given_back(native, oracle):
    import torch
    from fhetoothpaste_b200 import _native
    rng = np.random.default_rng(8)
    N, n, digits = 2048, 100, 3
    rot, key = rotator(1, N, 12, digits, n, rng)
    lwes, accs = inputs(rng, N, n, 3)
    first = rot.blind_rotate_batch_host(lwes, accs)

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]
    held = free()
    bad = np.tile(worst_poly(oracle, N, 3), key.size // N)
    _native.check(native.tp_br_upload_key(rot.handle, _native.ptr(bad), bad.size))
    assert free() - held > 2.5 * key.nbytes  # three limbs, each as large as the key
    np.testing.assert_array_equal(rot.blind_rotate_batch_host(lwes, accs),
                                  oracle.blind_rotate_many(1, N, n, 12, digits, bad, lwes, accs, False, 3))
    _native.check(native.tp_br_upload_key(rot.handle, _native.ptr(key), key.size))
    np.testing.assert_array_equal(rot.blind_rotate_batch_host(lwes, accs), first)
