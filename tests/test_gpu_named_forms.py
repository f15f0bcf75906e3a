"""Launch settings by name: a new context's own values leave the choice by batch size open, others name a modular
kernel, and setting them back restores the choice. The modular kernels in their default form against the golden vectors."""
import numpy as np
import pytest

from brcases import case_inputs
from kscases import ks_inputs, ks_key
from test_gpu_br import ALL_CASES, rotator as golden_rotator
from test_gpu_br_fft import SETS, inputs, rotator

pytestmark = pytest.mark.gpu

P = 0xFFFFFFFF00000001


def launches(native, run):
    before = native.tp_kernel_launches()
    run()
    return native.tp_kernel_launches() - before


def test_default_values_leave_the_choice_open(native):
    rng = np.random.default_rng(2)
    N, n = 1024, 3
    rot, _ = rotator(1, N, 12, 3, n, rng)
    lwes, accs = inputs(rng, N, n, 5)

    def count():  # the double-precision kernel and the results' transform, or the modular kernel alone
        return launches(native, lambda: rot.blind_rotate_batch_host(lwes, accs, out_coef=False))
    assert count() == 2 and rot.tile == 4
    for name, own, other in (("tile", 4, 8), ("split", 1, 2), ("mac_form", rot.mac_form, 1 - rot.mac_form), ("radix", 2, 4)):
        named = getattr(rot, f"set_{name}")
        named(own)
        assert count() == 2, name
        named(other)
        assert count() == 1 and getattr(rot, name) == other, name
        named(own)
        assert count() == 2, name
    native.tp_debug_modular(rot.handle, 1)
    rot.set_split(1)
    assert count() == 1
    native.tp_debug_modular(rot.handle, 0)
    assert count() == 2


def test_default_split_keeps_remainders(native):
    rng = np.random.default_rng(3)
    N, n = 2048, 4
    rot, _ = rotator(2, N, 16, 4, n, rng)
    lwes, accs = inputs(rng, N, n, 222)
    rot.set_split(1)
    assert launches(native, lambda: rot.blind_rotate_batch_host(lwes, accs)) == 2  # 148 and 74


def test_key_switch_tile(native):
    from fhetoothpaste_b200 import GpuLWEtoRLWEPacker
    rng = np.random.default_rng(4)
    N, beta, digits, logn = 1024, 16, 4, 10
    pk = GpuLWEtoRLWEPacker(N, 1 << beta, digits, rng.integers(0, P, logn * digits * 2 * N, dtype=np.uint64))
    x = rng.integers(0, P, (4, N + 1), dtype=np.uint64)
    want = pk.Pack(x, 4)
    for tile, extra in ((4, 0), (8, 1), (4, 0)):  # the modular form sets its leaves up in a launch of its own
        pk.set_tile(tile)
        assert launches(native, lambda: np.testing.assert_array_equal(pk.Pack(x, 4), want)) == logn + extra


@pytest.mark.parametrize("name", ALL_CASES)
def test_modular_rotations_match_reference(native, oracle, golden, name):
    case, rot = golden_rotator(oracle, golden, name)
    native.tp_debug_modular(rot.handle, 1)
    lwes, accs, coefs = case_inputs(name, case)
    for oc in (0, 1):
        idx = [i for i, c in enumerate(coefs) if c == oc]
        np.testing.assert_array_equal(rot.blind_rotate_batch_host(lwes[idx], accs[idx], out_coef=bool(oc)),
                                      golden[1][f"br_{name}"][idx])


# strides, a shared accumulator, results in place, evaluation-domain results, batches past a wave
@pytest.mark.parametrize("variant,N,beta,digits,batch", [(*s, b) for s in SETS for b in (20, 310)] + [(*SETS[0], 40)] +
                         [(v, N, 14, 3, b) for v, N in ((0, 8192), (1, 8192), (2, 8192), (1, 16384)) for b in (1, 17)])
def test_open_forms_equal_modular_kernels(native, variant, N, beta, digits, batch):
    import torch
    rng = np.random.default_rng(N + batch)
    n = 3
    rot, _ = rotator(variant, N, beta, digits, n + variant // 2, rng)
    n += variant // 2
    lwes, accs = inputs(rng, N, n, batch)
    wide = np.zeros((batch, n + 5), np.uint64)
    wide[:, :n + 1] = lwes
    d_lwe, d_acc = (torch.from_numpy(x.view(np.int64)).cuda() for x in (wide, accs))

    def run(stride, coef, in_place):
        dst = d_acc.clone() if in_place else torch.zeros_like(d_acc)
        rot.blind_rotate_batch(dst.data_ptr(), d_lwe.data_ptr(), n + 5, (dst if in_place else d_acc).data_ptr(), stride,
                               batch, coef)
        rot.check()
        return dst
    forms = [(2 * N, True, False), (2 * N, False, True), (0, True, False)]
    got = [run(*f) for f in forms]
    native.tp_debug_modular(rot.handle, 1)
    for f, words in zip(forms, got):
        assert torch.equal(words, run(*f))


@pytest.mark.parametrize("name", ["rlwe_ks_n2048", "auto5_n2048", "pack2048_n2048"])
def test_modular_key_switches_match_reference(native, oracle, golden, name):
    from fhetoothpaste_b200 import GpuAutomorphismEvaluator, GpuLWEtoRLWEPacker, GpuRLWEtoRLWEConverter
    c, expect = golden[0]["ks"][name], golden[1][f"ks_{name}"]
    N, base, dg, key, x = c["N"], 1 << c["basis_log2"], c["digits"], ks_key(oracle, name, c), ks_inputs(c)
    out = np.zeros((2, 2 * N), np.uint64)
    if name.startswith("pack"):
        op = GpuLWEtoRLWEPacker(N, base, dg, key)
        native.tp_debug_ks_modular(op._h, 1)
        out = op.Pack(x, c["len"])
    elif name.startswith("auto"):
        op = GpuAutomorphismEvaluator(N, base, dg, c["index"], key)
        native.tp_debug_ks_modular(op._h, 1)
        op.Eval(out, x)
    else:
        op = GpuRLWEtoRLWEConverter(N, base, dg, key)
        native.tp_debug_ks_modular(op._h, 1)
        op.Convert(out, x)
    np.testing.assert_array_equal(out[:len(expect)], expect)


@pytest.mark.parametrize("N,beta,digits", [(1024, 20, 3), (2048, 16, 4), (2048, 8, 2), (4096, 12, 3)])
def test_staged_switch_equals_the_general_kernel(native, N, beta, digits):
    import torch
    from fhetoothpaste_b200 import GpuRLWEtoRLWEConverter
    rng = np.random.default_rng(N + digits)
    conv = GpuRLWEtoRLWEConverter(N, 1 << beta, digits, rng.integers(0, P, digits * 2 * N, dtype=np.uint64))
    batch = 148 * (4096 // N) + 3
    x, base = (torch.from_numpy(rng.integers(0, P, (batch, 2 * N), dtype=np.uint64).view(np.int64)).cuda() for _ in range(2))
    res = []
    for modular in (0, 1):
        native.tp_debug_ks_modular(conv._h, modular)
        out, same = base.clone(), x.clone()
        conv.convert_batch(batch, out.data_ptr(), x.data_ptr())
        conv.convert_batch(batch, same.data_ptr(), same.data_ptr())
        torch.cuda.synchronize()
        res.append((out, same))
    assert all(torch.equal(a, b) for a, b in zip(*res))
