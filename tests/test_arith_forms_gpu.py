"""The arithmetics of the transform passes (the reference's butterflies, relaxed
integers, FP64) chosen by modulus width and batch size: every op bit-exact
against the oracle, for moduli on both sides of each limit in one batch, for
single limbs, pairs of limbs and an odd last group, on uniform, extreme and
sparse inputs (zeros and small values need the exact lazy quotient)."""
import numpy as np
import pytest

from helpers import dev, dev_empty, host, ptr

pytestmark = pytest.mark.gpu


def limit_moduli(oracle, n):
    """Smallest and largest NTT primes around the limits 2^50 and 2^59, a small and the widest ones."""
    picks = [(30, 1, 2), (40, 1, 2), (50, 1, 1), (51, 0, 1), (59, 1, 1), (60, 0, 1), (62, 1, 1)]
    out = []
    for bits, num, den in picks:
        q = oracle.find_ntt_prime_near(n, bits, num, den)
        out.append((q, oracle.find_primitive_root(n, q)))
    return out


def inputs(rng, n, bounds):
    """Per limb, by turns: uniform, all bound - 1, one nonzero coefficient, small values."""
    x = np.zeros((len(bounds), n), np.uint64)
    for i, b in enumerate(bounds):
        kind = i // 7 % 4
        if kind == 0:
            x[i] = rng.integers(0, b, n, dtype=np.uint64)
        elif kind == 1:
            x[i] = b - 1
        elif kind == 2:
            x[i, rng.integers(n)] = int(rng.integers(1, b, dtype=np.uint64))
        else:
            x[i] = rng.integers(0, 3, n, dtype=np.uint64)
    return x


# single limbs, a pair below and above the size from which limbs share a
# thread, an odd last group; one pass (N <= 2^13 by plan) and two
@pytest.mark.parametrize("n,polys", [(16, 1), (64, 2), (256, 5), (512, 1), (1024, 2), (4096, 92), (8192, 1), (16384, 23),
                                     (32768, 2), (65536, 6), (131072, 1)])
def test_forms_match_oracle(cuda, oracle, n, polys):
    mods = limit_moduli(oracle, n)
    L, count = len(mods), len(mods) * polys
    ntts = cuda.NTT.create_many([(n, q, psi) for q, psi in mods])
    tabs = [oracle.tables(n, q, psi) for q, psi in mods]
    rng = np.random.default_rng(n + polys)
    qs = [mods[i % L][0] for i in range(count)]
    x4, x2 = inputs(rng, n, [4 * q for q in qs]), inputs(rng, n, [2 * q for q in qs])
    m4, m2 = inputs(rng, n, [4 * q for q in qs]), inputs(rng, n, [2 * q for q in qs])
    sc = [(2 * q) // 3 for q, _ in mods]
    d4, d2, e4, e2, o = dev(x4), dev(x2), dev(m4), dev(m2), dev_empty(count * n)
    fwd = lambda i, v, f=1: oracle.forward(v, qs[i], tabs[i % L][0], 1, f)
    inv = lambda i, v, f=1: oracle.inverse(v, qs[i], tabs[i % L][1], tabs[i % L][2], 2, f)
    red = lambda i, v: oracle.reduce(v, qs[i], 4, 2)
    ops = {
        "forward 4": (lambda: cuda.forward_batch(ntts, ptr(o), ptr(d4), count, 4, 4), lambda i: fwd(i, x4[i], 4)),
        "forward 1": (lambda: cuda.forward_batch(ntts, ptr(o), ptr(d4), count, 4, 1), lambda i: fwd(i, x4[i])),
        "inverse 1": (lambda: cuda.inverse_batch(ntts, ptr(o), ptr(d2), count, 2, 1), lambda i: inv(i, x2[i])),
        "inverse 4->1": (lambda: cuda.inverse_batch(ntts, ptr(o), ptr(d4), count, 4, 1),
                         lambda i: inv(i, red(i, x4[i]))),
        "inverse 2": (lambda: cuda.inverse_batch(ntts, ptr(o), ptr(d2), count, 2, 2), lambda i: inv(i, x2[i], 2)),
        "forward mul": (lambda: cuda.forward_mul_batch(ntts, ptr(o), ptr(d4), ptr(e4), count),
                        lambda i: oracle.mul(fwd(i, x4[i], 4), m4[i], qs[i], 4)),
        "mul inverse": (lambda: cuda.mul_inverse_batch(ntts, ptr(o), ptr(d4), ptr(e4), count, 1),
                        lambda i: inv(i, oracle.mul(x4[i], m4[i], qs[i], 4))),
        "chain mul 1": (lambda: cuda.chain_mul_batch(ntts, ptr(o), ptr(d4), ptr(e2), count, 4, 1),
                        lambda i: fwd(i, oracle.mul(inv(i, red(i, x4[i]), 2), m2[i], qs[i], 2))),
        "chain fma 4": (lambda: cuda.chain_fma_batch(ntts, ptr(o), ptr(d2), sc, ptr(e2), count, 2, 4),
                        lambda i: fwd(i, oracle.fma(inv(i, x2[i], 2), sc[i % L], m2[i], qs[i], 2), 4)),
        "product 1": (lambda: cuda.product_batch(ntts, ptr(o), ptr(d4), ptr(e4), count, 4, 1),
                      lambda i: inv(i, oracle.mul(fwd(i, x4[i], 4), m4[i], qs[i], 4))),
        "product 2": (lambda: cuda.product_batch(ntts, ptr(o), ptr(d4), ptr(e4), count, 4, 2),
                      lambda i: inv(i, oracle.mul(fwd(i, x4[i], 4), m4[i], qs[i], 4), 2)),
    }
    for name, (run, expect) in ops.items():
        run()
        got = host(o).reshape(count, n)
        for i in range(count):
            np.testing.assert_array_equal(got[i], expect(i), err_msg=f"{name}: limb {i}, q of {qs[i].bit_length()} bits")


# The last group of limbs holds some of the moduli only: few limbs (up to 64), more,
# and enough for two limbs per thread, with and without partners for most.
@pytest.mark.parametrize("n,counts", [(4096, (66, 71, 606, 1008)), (16384, (8, 13, 33, 64, 65, 160)), (65536, (8, 13, 39)),
                                      (131072, (9,))])
def test_partial_last_group(cuda, oracle, n, counts):
    mods = limit_moduli(oracle, n)
    L, top = len(mods), max(counts)
    ntts = cuda.NTT.create_many([(n, q, psi) for q, psi in mods])
    tabs = [oracle.tables(n, q, psi) for q, psi in mods]
    rng = np.random.default_rng(n)
    qs = [mods[i % L][0] for i in range(top)]
    x, m = inputs(rng, n, [2 * q for q in qs]), inputs(rng, n, [2 * q for q in qs])
    sc = [(2 * q) // 3 for q, _ in mods]
    d, e, o = dev(x), dev(m), dev_empty(top * n)
    fwd = lambda i, v, f=1: oracle.forward(v, qs[i], tabs[i % L][0], 1, f)
    inv = lambda i, v, f=1: oracle.inverse(v, qs[i], tabs[i % L][1], tabs[i % L][2], 2, f)
    ops = {
        "forward 1": (lambda c: cuda.forward_batch(ntts, ptr(o), ptr(d), c, 2, 1), lambda i: fwd(i, x[i])),
        "forward 4": (lambda c: cuda.forward_batch(ntts, ptr(o), ptr(d), c, 2, 4), lambda i: fwd(i, x[i], 4)),
        "inverse 1": (lambda c: cuda.inverse_batch(ntts, ptr(o), ptr(d), c, 2, 1), lambda i: inv(i, x[i])),
        "chain fma 1": (lambda c: cuda.chain_fma_batch(ntts, ptr(o), ptr(d), sc, ptr(e), c, 2, 1),
                        lambda i: fwd(i, oracle.fma(inv(i, x[i], 2), sc[i % L], m[i], qs[i], 2))),
        "chain fma 4": (lambda c: cuda.chain_fma_batch(ntts, ptr(o), ptr(d), sc, 0, c, 2, 4),
                        lambda i: fwd(i, oracle.fma(inv(i, x[i], 2), sc[i % L], None, qs[i], 2), 4)),
        "product 1": (lambda c: cuda.product_batch(ntts, ptr(o), ptr(d), ptr(e), c, 4, 1),
                      lambda i: inv(i, oracle.mul(fwd(i, x[i], 4), m[i], qs[i], 4))),
    }
    for name, (run, expect) in ops.items():
        want = np.stack([expect(i) for i in range(top)])
        for c in counts:
            o.fill_(-1)
            run(c)
            got = host(o).reshape(top, n)
            np.testing.assert_array_equal(got[:c], want[:c], err_msg=f"{name}, {c} limbs")
            assert (got[c:] == np.uint64(2 ** 64 - 1)).all(), f"{name}, {c} limbs: written past the last"


@pytest.mark.parametrize("bits", [50, 59])
def test_in_place_and_unaligned(cuda, oracle, bits):
    """In place, and at 8- and 16-byte aligned addresses (the wide accesses fall back)."""
    n, polys = 16384, 24
    q = oracle.find_ntt_prime_near(n, bits, 1, 1)
    psi = oracle.find_primitive_root(n, q)
    t = cuda.NTT(n, q, psi)
    fwd, inv, ninv = oracle.tables(n, q, psi)
    x = inputs(np.random.default_rng(bits), n, [q] * polys)
    exp = np.stack([oracle.forward(v, q, fwd, 1, 1) for v in x])
    for words in (0, 1, 2):
        buf = dev(np.concatenate([np.zeros(words, np.uint64), x.reshape(-1)]))
        p = ptr(buf) + 8 * words
        cuda.forward_batch([t], p, p, polys, 1, 1)
        np.testing.assert_array_equal(host(buf)[words:].reshape(polys, n), exp, err_msg=f"forward at +{words}")
        cuda.inverse_batch([t], p, p, polys, 1, 1)
        np.testing.assert_array_equal(host(buf)[words:].reshape(polys, n), x, err_msg=f"inverse at +{words}")


@pytest.mark.parametrize("factor", [1, 2, 4])
def test_tensor_forms(cuda, oracle, factor):
    """The tensor product on moduli around the FP64 limit (any modulus, prime or not), uniform and extreme inputs."""
    n, qs = 1026, [17, (1 << 30) - 35, (1 << 50) - 27, (1 << 50) + 55, (1 << 61) + 15]
    rng = np.random.default_rng(factor)
    count = 4 * 7 * len(qs)
    bounds = [factor * qs[i % len(qs)] for i in range(count)]
    x = [inputs(rng, n, bounds) for _ in range(4)]
    d = [dev(v) for v in x]
    r = [dev_empty(count * n) for _ in range(3)]
    cuda.tensor_product(*[ptr(t) for t in (*r, *d)], n, count, qs, factor)
    got = [host(t).reshape(count, n) for t in r]
    for i in range(count):
        q = qs[i % len(qs)]
        c0, c1, d0, d1 = (v[i] for v in x)
        mul = lambda a, b: oracle.mul(a, b, q, factor)
        exp = (mul(c0, d0), oracle.add(mul(c0, d1), mul(c1, d0), q), mul(c1, d1))
        for k in range(3):
            np.testing.assert_array_equal(got[k][i], exp[k], err_msg=f"limb {i} output {k} q={q}")


@pytest.mark.parametrize("n,count", [(2, 1), (514, 3), (4096, 40), (2048, 1024), (32768, 9)])
def test_tensor_without_fp64_moduli(cuda, oracle, n, count):
    qs = [(1 << 50) + 55, (1 << 61) + 15]
    rng = np.random.default_rng(n)
    x = [np.stack([rng.integers(0, 2 * qs[i % 2], n, dtype=np.uint64) for i in range(count)]) for _ in range(4)]
    d = [dev(v) for v in x]
    r = [dev_empty(count * n) for _ in range(3)]
    cuda.tensor_product(*[ptr(t) for t in (*r, *d)], n, count, qs, 2)
    got = [host(t).reshape(count, n) for t in r]
    for i in sorted({0, 1, count // 2, count - 1} & set(range(count))):
        q = qs[i % 2]
        mul = lambda a, b: oracle.mul(a[i], b[i], q, 2)
        c0, c1, d0, d1 = x
        for k, exp in enumerate((mul(c0, d0), oracle.add(mul(c0, d1), mul(c1, d0), q), mul(c1, d1))):
            np.testing.assert_array_equal(got[k][i], exp, err_msg=f"limb {i} output {k}")


def sparse_inputs(rng, n, q):
    """Zeros, a constant, polynomials in X^2 and X^4, a zero upper half, multiples of q, small values."""
    x = np.zeros((8, n), np.uint64)
    x[1, 0] = q - 1
    x[2, ::2] = rng.integers(0, q, n // 2, dtype=np.uint64)
    x[3, ::4] = rng.integers(0, 4 * q, n // 4, dtype=np.uint64)
    x[4, : n // 2] = rng.integers(0, q, n // 2, dtype=np.uint64)
    x[5] = q * rng.integers(0, 4, n).astype(np.uint64)
    x[6] = rng.integers(0, 3, n, dtype=np.uint64)
    x[7] = np.where(rng.integers(0, 2, n) == 0, 0, rng.integers(0, 4 * q, n, dtype=np.uint64))
    return x


# enough residues for the FP64 form of a lazy forward
@pytest.mark.parametrize("n,copies", [(64, 768), (4096, 13), (16384, 4), (65536, 1)])
@pytest.mark.parametrize("bits,num,den", [(20, 1, 2), (30, 1, 2), (45, 1, 2), (50, 1, 1)])
def test_lazy_forward_of_sparse_inputs(cuda, oracle, n, copies, bits, num, den):
    q = oracle.find_ntt_prime_near(n, bits, num, den)
    psi = oracle.find_primitive_root(n, q)
    t = cuda.NTT(n, q, psi)
    fwd, inv, ninv = oracle.tables(n, q, psi)
    rng = np.random.default_rng(n + bits)
    x = sparse_inputs(rng, n, q)
    x2, m = x % np.uint64(2 * q), rng.integers(0, 2 * q, n, dtype=np.uint64)
    count = len(x) * copies
    d, d2, e, o = dev(np.tile(x, (copies, 1))), dev(np.tile(x2, (copies, 1))), dev(np.tile(m, count)), dev_empty(count * n)
    cuda.forward_batch([t], ptr(o), ptr(d), count, 4, 4)
    want = np.stack([oracle.forward(v, q, fwd, 4, 4) for v in x])
    np.testing.assert_array_equal(host(o).reshape(copies, len(x), n), np.broadcast_to(want, (copies, len(x), n)))
    cuda.chain_mul_batch([t], ptr(o), ptr(d2), ptr(e), count, 2, 4)
    want = np.stack([oracle.forward(oracle.mul(oracle.inverse(v, q, inv, ninv, 2, 2), m, q, 2), q, fwd, 1, 4) for v in x2])
    np.testing.assert_array_equal(host(o).reshape(copies, len(x), n), np.broadcast_to(want, (copies, len(x), n)))
