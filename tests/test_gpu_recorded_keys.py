"""Recorded launches (the library's graphs and a caller's own capture) follow the key that is uploaded later,
also one whose double-precision products are not proven exact: then the modular kernels recorded beside run."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = 0xFFFFFFFF00000001


def worst_poly(oracle, N, limbs):
    """Evaluations of the polynomial whose limbs are all at their largest (three times the mean squared norm)."""
    base = 2642246 if limbs == 3 else 1 << 16
    return oracle.ntt_forward(np.full(N, sum((base // 2 - 1) * base ** i for i in range(limbs)) % P, np.uint64))


def graph_nodes(graph) -> int:
    n = ctypes.c_size_t()
    cudart = ctypes.CDLL("libcudart.so.12")
    assert cudart.cudaGraphGetNodes(ctypes.c_void_p(graph.raw_cuda_graph()), None, ctypes.byref(n)) == 0
    return n.value


# clusters of eight and four blocks, a pair or one block each, a remainder of its own, halves on two blocks; the limb
# counts are those whose bound the second key fails
@pytest.mark.parametrize("variant,N,beta,digits,limbs,batch,launches", [
    (1, 2048, 12, 3, 3, 1, 1), (1, 2048, 12, 3, 3, 20, 1), (1, 2048, 12, 3, 3, 75, 1), (1, 2048, 12, 3, 3, 160, 2),
    (1, 1024, 13, 3, 3, 75, 1), (1, 4096, 16, 4, 4, 16, 1)])
def test_rotations(native, oracle, variant, N, beta, digits, limbs, batch, launches):
    import torch
    from fhetoothpaste_b200 import BlindRotationContext, GpuBlindRotator, _native
    rng = np.random.default_rng(N + batch)
    n = 3
    ctx = BlindRotationContext(variant, N, n, 1 << beta, digits)
    keys = [rng.integers(0, P, ctx.key_words(), dtype=np.uint64),
            np.tile(worst_poly(oracle, N, limbs), ctx.key_words() // N),
            rng.integers(0, P, ctx.key_words(), dtype=np.uint64)]
    rot = GpuBlindRotator(ctx, keys[0])
    lwes = rng.integers(0, 2 * N, (batch, n + 1), dtype=np.uint64)
    accs = rng.integers(0, P, (batch, 2 * N), dtype=np.uint64)
    d_lwe, d_acc = (torch.from_numpy(x.view(np.int64)).cuda() for x in (lwes, accs))
    coef, evals = torch.zeros_like(d_acc), d_acc.clone()
    torch.cuda.synchronize()
    own = rot.capture_batch(coef.data_ptr(), d_lwe.data_ptr(), n + 1, d_acc.data_ptr(), 2 * N, batch, out_coef=True)
    theirs = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(theirs):  # in place, evaluations
        rot.blind_rotate_batch(evals.data_ptr(), d_lwe.data_ptr(), n + 1, evals.data_ptr(), 2 * N, batch, False,
                               torch.cuda.current_stream().cuda_stream)
    assert graph_nodes(theirs) == 3 * launches  # each with its modular form behind it, and the results' transform
    theirs.instantiate()
    for key in keys:
        _native.check(native.tp_br_upload_key(rot.handle, _native.ptr(key), key.size))
        coef.zero_()
        evals.copy_(d_acc)
        torch.cuda.synchronize()
        before = native.tp_kernel_launches()
        own.launch()
        assert native.tp_kernel_launches() - before == launches
        theirs.replay()
        torch.cuda.synchronize()
        rot.check()
        for b in sorted({0, batch // 2, batch - 1}):
            for got, form in ((coef, 1), (evals, 0)):
                want = oracle.blind_rotate(variant, N, n, beta, digits, key, lwes[b], accs[b], form)
                np.testing.assert_array_equal(got[b].cpu().numpy().view(np.uint64), want)
    own.close()
    rot.close()


@pytest.mark.parametrize("N,beta,digits,limbs,packs,length", [(2048, 14, 3, 3, 1, 4), (1024, 15, 3, 3, 3, 2)])
def test_packings(native, oracle, N, beta, digits, limbs, packs, length):
    """Merges and traces of a captured packing, allocation-free as a capture needs it."""
    import torch
    from fhetoothpaste_b200 import GpuLWEtoRLWEPacker, _native
    rng = np.random.default_rng(N)
    logn = N.bit_length() - 1
    keys = [rng.integers(0, P, logn * digits * 2 * N, dtype=np.uint64),
            np.tile(worst_poly(oracle, N, limbs), logn * digits * 2),
            rng.integers(0, P, logn * digits * 2 * N, dtype=np.uint64)]
    pk = GpuLWEtoRLWEPacker(N, 1 << beta, digits, keys[0])
    x = rng.integers(0, P, (packs * length, N + 1), dtype=np.uint64)
    d_x = torch.from_numpy(x.view(np.int64)).cuda()
    out = torch.zeros((packs, 2 * N), dtype=torch.int64, device="cuda")

    def pack(stream):
        _native.check(native.tp_pack_batch_noalloc(pk._h, packs, length, out.data_ptr(), d_x.data_ptr(), stream))

    pack(None)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        pack(torch.cuda.current_stream().cuda_stream)
    # set-up, each merge and trace with its modular kernel behind it, the copy of the results
    assert graph_nodes(graph) == 2 + 2 * logn
    graph.instantiate()
    for key in keys:
        _native.check(native.tp_ks_upload_key(pk._h, _native.ptr(key), key.size))
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        got = out.cpu().numpy().view(np.uint64)
        for p in range(packs):
            want = oracle.pack(N, beta, digits, key, x[p * length:(p + 1) * length], length)
            np.testing.assert_array_equal(got[p], want)
