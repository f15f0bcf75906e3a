"""The tensor-core LWE key switch against the C oracle at the edges of its tiles, planes and splits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = 0xFFFFFFFF00000001


def run(n_in, n_out, beta, digits, batch, rng, key=None):
    import torch
    from fhetoothpaste_b200 import GpuLWEtoLWEConverter
    key = rng.integers(0, P, n_in * digits * (n_out + 1), dtype=np.uint64) if key is None else key
    conv = GpuLWEtoLWEConverter(n_in, n_out, 1 << beta, digits, key)
    x = rng.integers(0, P, (batch, n_in + 1), dtype=np.uint64)
    x[0, :4] = (0, P - 1, P // 2, P // 2 + 1)
    out = rng.integers(0, P, (batch, n_out + 1), dtype=np.uint64)
    got = torch.from_numpy(out.view(np.int64)).cuda()
    conv.convert_batch(batch, got.data_ptr(), torch.from_numpy(x.view(np.int64)).cuda().data_ptr())
    return key, x, out, got.cpu().numpy().view(np.uint64)


def expected(oracle, n_in, n_out, beta, digits, key, x, out):
    """The switch subtracts into out[:n_out] and sets out[n_out]; the oracle's output is a fresh one."""
    fresh = oracle.lwe_ks(P, n_in, n_out, beta, digits, key, x).astype(object)
    fresh[:n_out] += out[:n_out].astype(object)
    return fresh % P


# n_in l below, at and past a K step; words below, at and past a tile; one and two planes; rows around a tile
@pytest.mark.parametrize("n_in,n_out,beta,digits,batch", [
    (31, 31, 16, 4, 1), (32, 32, 16, 4, 128), (33, 30, 8, 8, 129), (100, 65, 12, 3, 5), (256, 1, 1, 7, 3),
    (1024, 500, 16, 4, 127), (2048, 630, 16, 4, 300), (16500, 3, 14, 4, 2),
])
def test_equals_oracle(native, oracle, n_in, n_out, beta, digits, batch):
    rng = np.random.default_rng(n_in + batch)
    before = native.tp_kernel_launches()
    key, x, out, got = run(n_in, n_out, beta, digits, batch, rng)
    assert native.tp_kernel_launches() - before == 5  # key: constants, bytes; digits, product, update
    for b in sorted({0, 1, batch // 2, batch - 1} & set(range(batch))):
        np.testing.assert_array_equal(got[b].astype(object), expected(oracle, n_in, n_out, beta, digits, key, x[b], out[b]))


@pytest.mark.parametrize("beta,digits", [(16, 4), (8, 8)])
def test_largest_sums(native, oracle, beta, digits):
    """All key bytes and all digit bytes at 255: the largest 32-bit sums of one split."""
    rng = np.random.default_rng(1)
    n_in, n_out = 33024 // digits, 2
    key = np.full(n_in * digits * (n_out + 1), P - 1, np.uint64)
    key[::2] = 0xFFFFFFFE_FFFFFFFF
    _, x, out, got = run(n_in, n_out, beta, digits, 2, rng, key)
    np.testing.assert_array_equal(got[1].astype(object), expected(oracle, n_in, n_out, beta, digits, key, x[1], out[1]))


def test_capture_by_the_caller(native):
    """A call captured into a caller's graph replays on new inputs (the scalar kernel: no workspace of its own)."""
    import torch
    from fhetoothpaste_b200 import GpuLWEtoLWEConverter
    rng = np.random.default_rng(2)
    n_in, n_out, batch = 64, 40, 7
    conv = GpuLWEtoLWEConverter(n_in, n_out, 1 << 16, 4, rng.integers(0, P, n_in * 4 * (n_out + 1), dtype=np.uint64))
    xs = [torch.from_numpy(rng.integers(0, P, (batch, n_in + 1), dtype=np.uint64).view(np.int64)).cuda() for _ in range(2)]
    buf, out = xs[0].clone(), torch.zeros((batch, n_out + 1), dtype=torch.int64, device="cuda")
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        conv.convert_batch(batch, out.data_ptr(), buf.data_ptr(), torch.cuda.current_stream().cuda_stream)
    for x in xs:
        buf.copy_(x)
        out.zero_()
        graph.replay()
        want = torch.zeros_like(out)
        torch.cuda.synchronize()
        conv.convert_batch(batch, want.data_ptr(), x.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert torch.equal(out, want)
