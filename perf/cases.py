"""The work that users of this framework have it do, as timed cases.

Sizes come from the benchmark's configurations (blind rotation at N = 1024, 2048 and
4096, BMMP at N = 2048, packing, key switching, whole bootstraps, scheme switching)
and from the ring range that every context accepts (N = 128 .. 65536). A case is a
dict of plain values; `kind` picks the entry point.
"""
import numpy as np
import torch

import fhetoothpaste_b200 as tp

P = tp.GOLDILOCKS
BINARY, TERNARY, BMMP = tp.TP_BR_CGGI_BINARY, tp.TP_BR_CGGI_TERNARY, tp.TP_BR_BMMP_BINARY
GROUP_KEYS = {BINARY: 1, TERNARY: 2, BMMP: 3}  # RGSWs per iteration


def _rotate(name, variant, N, n, beta, digits, batch, **more):
    return dict(name=name, kind="rotate", variant=variant, N=N, n=n, beta=beta, digits=digits, batch=batch,
                coef=False, shared=False, **more)


def listed():
    return [
        # one bootstrap called from a C++-like host program: host buffers in and out, one rotation
        dict(name="host_one_1024", kind="rotate_host", variant=BINARY, N=1024, n=500, beta=16, digits=4, batch=1),
        # one rotation on device buffers: the latency of a single gate
        _rotate("one_2048", TERNARY, 2048, 630, 12, 3, 1),
        # the throughput form: thousands of independent ciphertexts, each with its own test polynomial
        _rotate("batch_2048", TERNARY, 2048, 630, 12, 3, 4096),
        # unrolled (BMMP) rotations, between one wave and the largest batches
        _rotate("bmmp_2048", BMMP, 2048, 768, 16, 4, 512),
        # the largest serving set, a launch of an odd size
        _rotate("serving_4096", TERNARY, 4096, 900, 12, 3, 101),
        # large-precision rings rotate on a cluster of CTAs
        _rotate("ring_8192", TERNARY, 8192, 64, 12, 3, 100),
        # whole bootstraps (rotation, extraction, LWE key switch, modulus switch) replayed as one graph
        dict(name="bootstrap_1024", kind="bootstrap", variant=BINARY, N=1024, n=500, beta=16, digits=4, batch=1024),
        # RLWE key switching of a batch of ciphertexts
        dict(name="rlwe_switch", kind="rlwe_ks", N=2048, beta=16, digits=4, batch=1024),
        # n-LWE -> RLWE packing: many packings of a full ring each
        dict(name="pack_2048", kind="pack", N=2048, beta=16, digits=4, packs=16, length=2048),
        # LWE dimension switch of a batch after a rotation
        dict(name="lwe_switch", kind="lwe_ks", n_in=2048, n_out=630, beta=16, digits=4, batch=4096),
        # polynomials to the evaluation domain and back: plaintext products, keys
        dict(name="transforms", kind="ntt", N=1024, batch=37),
        # LWE -> RGSW scheme switching (rotation, trace, key switch)
        dict(name="lwe_to_rgsw", kind="to_rgsw", N=2048, n=100, beta=14, digits=4, batch=256),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["rotate", "rotate", "rotate", "rotate", "rotate_host", "bootstrap", "rlwe_ks", "pack",
                       "lwe_ks", "ntt", "to_rgsw"])
    beta, digits = rng.choice([(12, 3), (16, 4), (14, 4), (8, 4), (16, 2), (20, 3)])
    if kind in ("rotate", "rotate_host"):
        variant = rng.choice([BINARY, TERNARY, TERNARY, BMMP])
        N = rng.choice([512, 1024, 1024, 2048, 2048, 2048, 4096, 8192])
        n = 2 * _log(rng, 32, 450 if N < 8192 else 64)
        batch = _log(rng, 1, 2048 * 2048 // N) if kind == "rotate" else _log(rng, 1, 24)
        c = dict(kind=kind, variant=variant, N=N, n=n, beta=beta, digits=digits, batch=batch)
        if kind == "rotate":
            c.update(coef=rng.random() < 0.5, shared=rng.random() < 0.3)
        return c
    if kind == "bootstrap":
        return dict(kind=kind, variant=rng.choice([BINARY, TERNARY]), N=rng.choice([1024, 2048]),
                    n=_log(rng, 100, 630), beta=beta, digits=digits, batch=_log(rng, 1, 1024))
    if kind == "rlwe_ks":
        return dict(kind=kind, N=rng.choice([1024, 2048, 4096, 8192]), beta=beta, digits=digits,
                    batch=_log(rng, 1, 4096))
    if kind == "pack":
        N = rng.choice([1024, 2048, 4096])
        return dict(kind=kind, N=N, beta=beta, digits=digits, packs=_log(rng, 1, 16), length=2 ** rng.randint(1, 10))
    if kind == "lwe_ks":
        return dict(kind=kind, n_in=rng.choice([1024, 2048]), n_out=_log(rng, 400, 900), beta=beta, digits=digits,
                    batch=_log(rng, 1, 4096))
    if kind == "ntt":
        return dict(kind=kind, N=2 ** rng.randint(7, 14), batch=_log(rng, 1, 2000))
    return dict(kind=kind, N=rng.choice([1024, 2048]), n=_log(rng, 32, 300), beta=14, digits=4,
                batch=_log(rng, 1, 256))


# ---- inputs ---------------------------------------------------------------------------

class _Source:
    """Seeded words on the GPU. Key and ciphertext words are (pseudo)random residues, as encryption makes them."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def residues(self, *shape):
        hi = torch.randint(0, 0xFFFFFFFF, shape, device="cuda", generator=self.g)  # below 2^32 - 1: the word is below p
        lo = torch.randint(0, 1 << 32, shape, device="cuda", generator=self.g)
        return (hi << 32) | lo

    def below(self, bound, *shape):
        return torch.randint(0, bound, shape, device="cuda", generator=self.g)

    def key(self, words):
        return self.residues(words).cpu().numpy().view(np.uint64)

    def test_polynomials(self, rows, N):
        """[0 | LUT] rows: 16 random table entries at scale p / 16, each over N / 16 coefficients."""
        out = torch.zeros((rows, 2 * N), dtype=torch.int64, device="cuda")
        lut = self.below(8, rows, 16) * (P // 16)
        out[:, N:] = lut.repeat_interleave(N // 16, dim=1)
        return out


def _br_key_words(c):
    groups = c["n"] // 2 if c["variant"] == BMMP else c["n"]
    return groups * GROUP_KEYS[c["variant"]] * 4 * c["N"] * c["digits"]


def _rotator(c, src):
    ctx = tp.BlindRotationContext(c["variant"], c["N"], c["n"], 1 << c["beta"], c["digits"])
    return tp.GpuBlindRotator(ctx, src.key(_br_key_words(c)))


def prepare(case, seed):
    c, src = case, _Source(seed)
    s = dict(c)
    kind = c["kind"]
    if kind in ("rotate", "rotate_host", "bootstrap"):
        s["rot"] = _rotator(c, src)
        s["lwe"] = src.below(2 * c["N"], c["batch"], c["n"] + 1)
        s["acc"] = src.test_polynomials(1 if c.get("shared") else c["batch"], c["N"])
        s["out"] = torch.empty((c["batch"], 2 * c["N"]), dtype=torch.int64, device="cuda")
    if kind == "rotate_host":
        s["lwe"], s["acc"] = (s[k].cpu().numpy().view(np.uint64) for k in ("lwe", "acc"))
        s["out"] = np.empty((c["batch"], 2 * c["N"]), np.uint64)
    elif kind == "bootstrap":
        s["ks"] = tp.GpuLWEtoLWEConverter(c["N"], c["n"], 1 << 16, 4, src.key(c["N"] * 4 * (c["n"] + 1)))
        s["fresh"] = torch.empty((c["batch"], c["n"] + 1), dtype=torch.int64, device="cuda")
        s["graph"] = s["rot"].capture_bootstrap(s["ks"], c["batch"], s["out"].data_ptr(), s["lwe"].data_ptr(),
                                                s["acc"].data_ptr(), 2 * c["N"], s["fresh"].data_ptr())
    elif kind == "rlwe_ks":
        s["ks"] = tp.GpuRLWEtoRLWEConverter(c["N"], 1 << c["beta"], c["digits"], src.key(c["digits"] * 2 * c["N"]))
        s["in"] = src.residues(c["batch"], 2 * c["N"])
        s["out"] = torch.empty_like(s["in"])
    elif kind == "pack":
        s["ks"] = tp.GpuLWEtoRLWEPacker(c["N"], 1 << c["beta"], c["digits"],
                                        src.key((c["N"].bit_length() - 1) * c["digits"] * 2 * c["N"]))
        s["in"] = src.residues(c["packs"] * c["length"], c["N"] + 1)
        s["out"] = torch.empty((c["packs"], 2 * c["N"]), dtype=torch.int64, device="cuda")
    elif kind == "lwe_ks":
        s["ks"] = tp.GpuLWEtoLWEConverter(c["n_in"], c["n_out"], 1 << c["beta"], c["digits"],
                                          src.key(c["n_in"] * c["digits"] * (c["n_out"] + 1)))
        s["in"] = src.residues(c["batch"], c["n_in"] + 1)
        s["out"] = torch.empty((c["batch"], c["n_out"] + 1), dtype=torch.int64, device="cuda")
    elif kind == "ntt":
        s["in"] = src.residues(c["batch"], c["N"])
        s["fwd"] = torch.empty_like(s["in"])
        s["bwd"] = torch.empty_like(s["in"])
    elif kind == "to_rgsw":
        N, d = c["N"], c["digits"]
        keys = [src.key(w) for w in (c["n"] * 4 * N * d, (N.bit_length() - 1) * d * 2 * N, d * 2 * N)]
        s["conv"] = tp.GpuLWEtoRGSWConverter((BINARY, N, c["n"], 1 << c["beta"], d), (1 << c["beta"], d),
                                             (1 << c["beta"], d), 4, 1 << 14, *keys)
        s["lwe"] = src.below(2 * N, c["batch"], c["n"] + 1)
        s["out"] = torch.empty((c["batch"], s["conv"].output_words), dtype=torch.int64, device="cuda")
    return s


# ---- one pass -------------------------------------------------------------------------

def run(s):
    kind, st = s["kind"], torch.cuda.current_stream().cuda_stream
    if kind == "rotate":
        s["rot"].blind_rotate_batch(s["out"].data_ptr(), s["lwe"].data_ptr(), s["n"] + 1, s["acc"].data_ptr(),
                                    0 if s["shared"] else 2 * s["N"], s["batch"], s["coef"], st)
    elif kind == "rotate_host":
        for b in range(s["batch"]):
            s["rot"].BlindRotate(s["out"][b], s["lwe"][b], s["acc"][b], True)
    elif kind == "bootstrap":
        s["graph"].launch(st)
        return s["fresh"], s["out"]
    elif kind in ("rlwe_ks", "lwe_ks"):
        s["out"].zero_()  # Convert subtracts into its output
        s["ks"].convert_batch(s["batch"], s["out"].data_ptr(), s["in"].data_ptr(), st)
    elif kind == "pack":
        s["ks"].pack_batch(s["packs"], s["length"], s["out"].data_ptr(), s["in"].data_ptr(), st)
    elif kind == "ntt":
        tp.ntt_forward(s["N"], s["batch"], s["fwd"].data_ptr(), s["in"].data_ptr(), st)
        tp.ntt_backward(s["N"], s["batch"], s["bwd"].data_ptr(), s["fwd"].data_ptr(), st)
        return s["fwd"], s["bwd"]
    elif kind == "to_rgsw":
        s["conv"].convert_batch(s["batch"], s["out"].data_ptr(), s["lwe"].data_ptr(), st)
    return s["out"]


# ---- what a pass cannot do without ----------------------------------------------------

def work(case):
    """Bytes of keys, inputs and outputs once each; flops as two per modular product (transforms N/2 log2 N each)."""
    c, kind = case, case["kind"]
    d = c.get("digits", 0)
    N = c.get("N", 0)
    ntt = N // 2 * (N.bit_length() - 1)
    if kind in ("rotate", "rotate_host", "bootstrap"):
        g, groups = GROUP_KEYS[c["variant"]], c["n"] // 2 if c["variant"] == BMMP else c["n"]
        words = _br_key_words(c) + c["batch"] * (c["n"] + 1 + 4 * N)
        mul = groups * c["batch"] * ((2 + 2 * d) * ntt + 4 * d * g * N + 2 * g * N)
        if kind == "bootstrap":
            words += 4 * N * (c["n"] + 1) + c["batch"] * (c["n"] + 1)
            mul += c["batch"] * 4 * N * (c["n"] + 1)
    elif kind == "rlwe_ks":
        words = 2 * d * N + 4 * c["batch"] * N
        mul = c["batch"] * d * (ntt + 2 * N)
    elif kind == "pack":
        logn, loglen = N.bit_length() - 1, c["length"].bit_length() - 1
        words = logn * d * 2 * N + c["packs"] * (c["length"] * (N + 1) + 2 * N)
        mul = c["packs"] * (c["length"] - 1 + logn - loglen) * ((d + 3) * ntt + 2 * d * N)
    elif kind == "lwe_ks":
        words = c["n_in"] * d * (c["n_out"] + 1) + c["batch"] * (c["n_in"] + c["n_out"] + 2)
        mul = c["batch"] * c["n_in"] * d * (c["n_out"] + 1)
    elif kind == "ntt":
        words, mul = 3 * c["batch"] * N, 2 * c["batch"] * ntt
    else:
        logn = N.bit_length() - 1
        words = c["n"] * 4 * N * d + (logn + 1) * d * 2 * N + c["batch"] * (c["n"] + 1 + 16 * N)
        mul = c["batch"] * (c["n"] * ((2 + 2 * d) * ntt + 4 * d * N) + 4 * (logn + 1) * ((d + 3) * ntt + 2 * d * N))
    return {"bytes": 8 * words, "flops": 2 * mul}


# ---- the same results in plain numpy --------------------------------------------------

_U = np.uint64
_M32 = _U(0xFFFFFFFF)


def _add(a, b):
    s = a + b
    s = s + np.where(s < a, _M32, _U(0))
    return np.where(s >= _U(P), s - _U(P), s)


def _sub(a, b):
    return np.where(a >= b, a - b, a + (_U(P) - b))


def _mul(a, b):
    a0, a1, b0, b1 = a & _M32, a >> _U(32), b & _M32, b >> _U(32)
    m0 = a0 * b0
    m1 = a1 * b0 + (m0 >> _U(32))
    m2 = a0 * b1 + (m1 & _M32)
    hi = a1 * b1 + (m1 >> _U(32)) + (m2 >> _U(32))
    lo = (m2 << _U(32)) | (m0 & _M32)
    h1, h0 = hi >> _U(32), hi & _M32
    t = lo - h1
    t = np.where(lo < h1, t - _M32, t)
    r = t + h0 * _M32
    r = np.where(r < t, r + _M32, r)
    return np.where(r >= _U(P), r - _U(P), r)


class _Ring:
    """Negacyclic transforms over Goldilocks, slot k at psi^(2 brv(k) + 1), psi = 7^((p-1)/2N)."""

    def __init__(self, N):
        self.N, self.log = N, N.bit_length() - 1
        psi = pow(7, (P - 1) // (2 * N), P)
        self.pow = np.array([pow(psi, k, P) for k in range(2 * N)], _U)
        self.brv = np.array([int(format(k, "0%db" % self.log)[::-1], 2) for k in range(N)])
        self.tw, self.twi = self.pow[self.brv], self.pow[(2 * N - self.brv) % (2 * N)]

    def forward(self, x):
        x, rows, m, t = x.copy(), x.shape[0], 1, self.N
        while m < self.N:
            t //= 2
            v = x.reshape(rows, m, 2, t)
            u, w = v[:, :, 0].copy(), _mul(v[:, :, 1], self.tw[m:2 * m, None])
            v[:, :, 0], v[:, :, 1] = _add(u, w), _sub(u, w)
            m *= 2
        return x

    def backward(self, x):
        x, rows, m, t = x.copy(), x.shape[0], self.N // 2, 1
        while m:
            v = x.reshape(rows, m, 2, t)
            u, w = v[:, :, 0].copy(), v[:, :, 1].copy()
            v[:, :, 0], v[:, :, 1] = _add(u, w), _mul(_sub(u, w), self.twi[m:2 * m, None])
            m //= 2
            t *= 2
        return _mul(x, _U(pow(self.N, P - 2, P)))

    def mono(self, a):
        """X^a in every slot."""
        return self.pow[(2 * self.brv + 1) * a % (2 * self.N)]


def _digits(x, beta, digits, signed):
    """Gadget digits of canonical words, most significant first, as residues."""
    top = -(-64 // beta)
    if not signed:
        return [(x >> _U(beta * (top - 1 - d))) & _U((1 << beta) - 1) for d in range(digits)]
    last = 64 - beta * top  # the last shift, at most 0
    least = 1 << (last + beta - 1)
    y = _add(x, np.full_like(x, (sum(1 << (64 - beta * k - 1 + beta) for k in range(1, top)) + least) % P))
    out = []
    for d in range(digits):
        sh, half, mask = (0, least, 2 * least - 1) if d == top - 1 else (64 - beta * (d + 1), 1 << (beta - 1), (1 << beta) - 1)
        out.append(_sub((y >> _U(sh)) & _U(mask), np.full_like(x, half)))
    return out


def _rotate_exact(c, key, lwe, acc, coef):
    """CGGI and BMMP blind rotation of one ciphertext."""
    N, d, g = c["N"], c["digits"], GROUP_KEYS[c["variant"]]
    R = _Ring(N)
    key = key.reshape(-1, g, 2 * d, 2, N)
    one = np.ones(N, _U)
    x = _mul(R.forward(acc.reshape(2, N)), R.mono(int(lwe[-1])))
    for i, k in enumerate(key):
        if c["variant"] == BMMP:
            m0, m1 = (R.mono(-int(a) % (2 * N)) for a in lwe[2 * i:2 * i + 2])
            w0, w1 = _sub(m0, one), _sub(m1, one)
            weights, src = (w0, w1, _mul(w0, w1)), x
        else:
            down, up = (_sub(R.mono(s * int(lwe[i]) % (2 * N)), one) for s in (-1, 1))
            weights, src = ((one,), _mul(x, down)) if c["variant"] == BINARY else ((down, up), x)
        y = R.backward(src)
        rows = R.forward(np.concatenate([np.stack(_digits(h, c["beta"], d, c["variant"] != BINARY)) for h in y]))
        for q in range(g):
            e = np.zeros_like(x)
            for r in range(2 * d):
                e = _add(e, _mul(rows[r][None], k[q, r]))
            x = _add(x, _mul(e, weights[q][None]))
    return R.backward(x) if coef else x


def _words(t):
    return t.cpu().numpy().view(_U)


def exact(case, seed):
    """Every output is whole numbers; those that plain numpy gives within seconds are given here."""
    c, src, kind = case, _Source(seed), case["kind"]
    if kind in ("rotate", "rotate_host"):
        steps = c["n"] // 2 if c["variant"] == BMMP else c["n"]
        if steps * c["batch"] * c["N"] * (2 * c["digits"] + 2) > 10_000_000:
            return None
        key, lwe = src.key(_br_key_words(c)), _words(src.below(2 * c["N"], c["batch"], c["n"] + 1))
        acc = _words(src.test_polynomials(1 if c.get("shared") else c["batch"], c["N"]))
        return np.stack([_rotate_exact(c, key, lwe[b], acc[b % len(acc)], c.get("coef", True)).reshape(-1)
                         for b in range(c["batch"])]).view(np.int64 if kind == "rotate" else _U)
    if kind == "ntt" and c["batch"] * c["N"] <= 1 << 18:
        x = _words(src.residues(c["batch"], c["N"]))
        return _Ring(c["N"]).forward(x).view(np.int64), x.view(np.int64)
    if kind == "rlwe_ks" and c["batch"] * c["N"] * c["digits"] <= 1 << 18:
        N, d = c["N"], c["digits"]
        key, x = src.key(d * 2 * N).reshape(d, 2, N), _words(src.residues(c["batch"], 2 * N))
        out, R = np.zeros_like(x).reshape(-1, 2, N), _Ring(N)
        for r, dig in enumerate(_digits(x[:, :N], c["beta"], d, True)):
            out = _sub(out, _mul(R.forward(dig)[:, None], key[r][None]))
        out[:, 1] = _add(out[:, 1], x[:, N:])
        return out.reshape(x.shape).view(np.int64)
    return None
