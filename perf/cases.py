"""Performance cases: the calls that a user of the library times.

Each case is one pass through the public entry points of `axhel_b200.capi` on
device-resident residues, with the shapes of the repository's own
configurations (one limb of N = 4096; RNS polynomials of N = 2^12..2^17 and 1
to 48 limbs; the batch of 768 limbs of N = 2^16; the tensor product of 64
ciphertext pairs; uneven batches; served requests), primes of 30-60 bits.

`exact` recomputes every output from the reference's formulas (Harvey
butterflies with lazy ranges, Barrett / conditional-subtract element-wise
operations) in plain torch integer arithmetic.
"""
import functools
import math

import numpy as np
import torch

from axhel_b200 import capi, params

CHAIN_MUL, CHAIN_FMA = "chain_mul", "chain_fma"


def listed():
    return [
        # One ciphertext limb handled alone, as SEAL's evaluator does per call:
        # two forward transforms, the dyadic product, a scalar addition and the
        # inverse.  Bound by launches.
        dict(name="single_limb_n4096", kind="single", logn=12, bits=50),
        # A fresh ciphertext of a small parameter set (2 polynomials, 5 primes)
        # to evaluation form, lazy output as SEAL's ntt_negacyclic_harvey_lazy.
        dict(name="forward_lazy_n8192_10", kind="forward", logn=13, L=5, polys=2, lo=40, hi=44, in_f=1, out_f=4),
        # Three polynomials of 9 primes back to coefficient form before a
        # modulus switch: an odd limb count, normalized output.
        dict(name="inverse_n16384_27", kind="inverse", logn=14, L=9, polys=3, lo=48, hi=50, in_f=2, out_f=1),
        # Key-switching digits to evaluation form with canonical output.
        dict(name="forward_n32768_225", kind="forward", logn=15, L=15, polys=15, lo=40, hi=59, in_f=1, out_f=1),
        # The headline: 16 ciphertexts x 2 polynomials x 24 primes, lazy
        # forward and normalized inverse with the 4q -> 2q reduction fused.
        dict(name="roundtrip_n65536_768", kind="roundtrip", logn=16, L=24, polys=32, lo=50, hi=59),
        # A served request's work called directly: INTT -> MulMod -> NTT.
        dict(name="chain_mul_n32768_40", kind=CHAIN_MUL, logn=15, L=40, polys=1, lo=40, hi=59, in_f=2, out_f=4),
        # The same with a scalar and an addend at the largest degree, a ragged
        # number of limbs, canonical output.
        dict(name="chain_fma_n131072_23", kind=CHAIN_FMA, logn=17, L=23, polys=1, lo=40, hi=59, in_f=4, out_f=1),
        # multiply_plain of a ciphertext batch: NTT -> MulMod -> INTT.
        dict(name="product_n65536_96", kind="product", logn=16, L=24, polys=4, lo=50, hi=59, out_f=1),
        # Many ciphertexts of different parameter sets in one batch object,
        # per-phase launches.
        dict(name="uneven_batch_64", kind="uneven", polys=64, mix=1, form="phased"),
        # A ciphertext multiplication: 64 pairs x 16 primes, one fused launch.
        dict(name="tensor_n32768_1024", kind="tensor", logn=15, L=16, pairs=64, lo=40, hi=55, factor=1),
        # Element-wise calls on a long vector of odd length at 16-byte and
        # 8-byte alignment.
        dict(name="eltwise_4194303", kind="eltwise", n=4194303, bits=59, factor=4, offset=1),
        # A burst of device-resident requests through the serving loop.
        dict(name="serve_burst_12", kind="serve", requests=12, mix=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "forward", "forward", "inverse", "inverse", "roundtrip", "roundtrip", CHAIN_MUL,
                       CHAIN_FMA, "product", "halves", "uneven", "tensor", "eltwise", "serve"])
    if kind == "single":
        return dict(kind=kind, logn=rng.randint(12, 17), bits=rng.randint(30, 60))
    if kind == "uneven":
        return dict(kind=kind, polys=rng.randint(4, 40), mix=rng.randint(3, 1 << 20),
                    form=rng.choice(["phased", "phased", "one launch"]))
    if kind == "serve":
        return dict(kind=kind, requests=rng.randint(1, 12), mix=rng.randint(3, 1 << 20))
    if kind == "eltwise":
        return dict(kind=kind, n=_log_int(rng, 2048, 1 << 24), bits=rng.randint(30, 60),
                    factor=rng.choice([1, 2, 4]), offset=rng.randint(0, 1))
    lo = rng.randint(30, 58)
    hi = rng.randint(max(lo, 40), 60)
    logn = rng.randint(12, 17)
    # at most 2^25 residues (half the headline batch), 2^23 for the chains
    most = (1 << (23 if kind in (CHAIN_MUL, CHAIN_FMA, "product", "halves") else 25)) >> logn
    limbs = _log_int(rng, 1, min(most, 2048))
    L = rng.randint(1, min(48, limbs, 2 * (hi - lo + 1)))
    c = dict(kind=kind, logn=logn, L=L, polys=max(1, limbs // L), lo=lo, hi=hi)
    if kind == "tensor":
        c["pairs"] = c.pop("polys")
        c["factor"] = rng.choice([1, 2, 4])
    elif kind in ("forward", "inverse"):
        c.update(in_f=rng.choice([1, 4] if kind == "forward" else [2, 4]),
                 out_f=rng.choice([1, 4] if kind == "forward" else [1, 2]))
    elif kind in (CHAIN_MUL, CHAIN_FMA):
        c.update(in_f=rng.choice([2, 4]), out_f=rng.choice([1, 4]))
    elif kind in ("product", "halves"):
        c.update(out_f=rng.choice([1, 2]))
    return c


# ------------------------------------------------------------------ inputs

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _stream():
    return torch.cuda.current_stream().cuda_stream


@functools.lru_cache(maxsize=None)
def _moduli(n, L, lo, hi):
    return tuple(params.rns_moduli(n, L, lo, hi))


@functools.lru_cache(maxsize=None)
def _modulus(n, bits, pos):
    q = params.ntt_prime_near(n, bits, pos, 4)
    return q, params.primitive_root(n, q)


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(seed)


def _rows(gen, bounds, n):
    """One row of n residues per bound, uniform in [0, bound); few distinct bounds."""
    x = torch.randint(0, (1 << 63) - 1, (len(bounds), n), dtype=torch.int64, device=_device(), generator=gen)
    return x.remainder_(torch.tensor(bounds, dtype=torch.int64, device=_device()).unsqueeze(1))


def _limb_jobs(case):
    """The jobs of an uneven batch or a burst of requests: (kind, n, moduli, in_f, out_f, scalars)."""
    rng = np.random.default_rng(case["mix"])
    jobs = []
    if case["kind"] == "uneven":
        for j in range(case["polys"]):
            n, L = 1 << int(rng.integers(12, 18)), int(rng.integers(1, 49))
            kind = ("forward", "inverse", CHAIN_MUL)[j % 3]
            mods = [_modulus(n, int(rng.integers(30, 61)), int(rng.integers(1, 4))) for _ in range(L)]
            out_f = int(rng.choice([1, 2] if kind == "inverse" else [1, 4]))
            jobs.append((kind, n, mods, int(rng.choice([1, 2, 4])), out_f, None))
    else:
        for j in range(case["requests"]):
            n, L = 1 << int(rng.integers(13, 18)), int(rng.integers(2, 41))
            mods = [_modulus(n, 40 + i % 20, 1 + i // 20) for i in range(L)]
            kind = CHAIN_FMA if j % 2 else CHAIN_MUL
            scalars = [int(rng.integers(0, 2 * q)) for q, _ in mods] if j % 2 else None
            jobs.append((kind, n, mods, 2, 4, scalars))
    return jobs


def _inputs(case, seed):
    """The case's operands (tensors by name) and its moduli, made from the seed alone."""
    gen = _generator(seed)
    kind = case["kind"]
    if kind in ("uneven", "serve"):
        jobs = _limb_jobs(case)
        ops = []
        for k, n, mods, in_f, _, _ in jobs:
            x = _rows(gen, [in_f * q for q, _ in mods], n)
            ops.append((x, _rows(gen, [2 * q for q, _ in mods], n) if k in (CHAIN_MUL, CHAIN_FMA) else None))
        return dict(jobs=jobs, ops=ops)
    if kind == "eltwise":
        q = _modulus(4096, case["bits"], 2)[0]
        f, n, off = case["factor"], case["n"], case["offset"]
        a, b = (_rows(gen, [f * q], n + off)[0] for _ in range(2))
        return dict(q=q, a=a[off:], b=b[off:], scalar=f * q - 3)
    n = 1 << case["logn"]
    if kind == "single":
        mods = (_modulus(n, case["bits"], 1),)
        x = _rows(gen, [mods[0][0]] * 2, n)
        return dict(mods=mods, x=x, scalar=mods[0][0] // 3)
    mods = _moduli(n, case["L"], case["lo"], case["hi"])
    if kind == "tensor":
        bounds = [case["factor"] * q for q, _ in mods] * case["pairs"]
        return dict(mods=mods, ops=[_rows(gen, bounds, n) for _ in range(4)])
    f = {"roundtrip": 1, "product": 4, "halves": 4}.get(kind) or case["in_f"]
    x = _rows(gen, [f * q for q, _ in mods] * case["polys"], n)
    d = dict(mods=mods, x=x)
    if kind in (CHAIN_MUL, CHAIN_FMA):
        d["v"] = _rows(gen, [2 * q for q, _ in mods] * case["polys"], n)
        d["scalars"] = [(2 * q) // 3 for q, _ in mods]
    elif kind in ("product", "halves"):
        d["v"] = _rows(gen, [4 * q for q, _ in mods] * case["polys"], n)
    return d


def _ntts(n, mods):
    return capi.NTT.create_many([(n, q, psi) for q, psi in mods])


JOB = {"forward": capi.JOB_FORWARD, "inverse": capi.JOB_INVERSE, CHAIN_MUL: capi.JOB_CHAIN_MUL,
       CHAIN_FMA: capi.JOB_CHAIN_FMA}


def prepare(case, seed):
    st = dict(_inputs(case, seed), case=case)
    kind = case["kind"]
    if kind in ("uneven", "serve"):
        st["ntts"] = [_ntts(n, mods) for _, n, mods, _, _, _ in st["jobs"]]
        st["outs"] = [torch.empty_like(x) for x, _ in st["ops"]]
        if kind == "uneven":
            st["batch"] = capi.Batch([
                dict(kind=JOB[k], ntts=t, count=len(mods), result=y.data_ptr(), operand=x.data_ptr(),
                     vector=v.data_ptr() if v is not None else 0, in_f=in_f, out_f=out_f)
                for (k, n, mods, in_f, out_f, _), (x, v), t, y in zip(st["jobs"], st["ops"], st["ntts"], st["outs"])])
        else:
            st["server"] = capi.Server(budget_bytes=8 << 30, max_inflight=8, max_batch_requests=1)
            torch.cuda.synchronize()  # the server's streams read the operands
    elif kind == "eltwise":
        off = case["offset"]
        st["outs"] = [torch.empty(case["n"] + off, dtype=torch.int64, device=_device())[off:] for _ in range(4)]
    elif kind == "tensor":
        st["outs"] = [torch.empty_like(st["ops"][0]) for _ in range(3)]
    else:
        st["ntts"] = _ntts(1 << case["logn"], st["mods"])
        k = 2 if kind in ("single", "roundtrip", "halves") else 1
        st["outs"] = [torch.empty_like(st["x"]) for _ in range(k)]
    return st


# --------------------------------------------------------------------- run

def run(state):
    """One pass; returns every output."""
    case, s = state["case"], _stream()
    kind, outs = case["kind"], state["outs"]
    if kind == "uneven":
        state["batch"].launch(s, phased=case["form"] == "phased")
        return outs
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(JOB[k], t, len(mods), x.data_ptr(), y.data_ptr(), vector=v.data_ptr(), scalars=sc,
                          in_f=in_f, out_f=out_f)
               for (k, n, mods, in_f, out_f, sc), (x, v), t, y in
               zip(state["jobs"], state["ops"], state["ntts"], outs)]
        for i in ids:
            status, _ = srv.wait(i)
            if status:
                raise RuntimeError(f"request failed: status {status}")
        return outs
    if kind == "eltwise":
        n, q, f, sc = case["n"], state["q"], case["factor"], state["scalar"]
        a, b = state["a"].data_ptr(), state["b"].data_ptr()
        capi.mul(outs[0].data_ptr(), a, b, n, q, f, s)
        capi.fma(outs[1].data_ptr(), a, sc, b, n, q, f, s)
        capi.reduce(outs[2].data_ptr(), a, n, q, q, 1, s)
        capi.add(outs[3].data_ptr(), outs[0].data_ptr(), outs[1].data_ptr(), n, q, s)
        return outs
    n = 1 << case["logn"]
    if kind == "tensor":
        capi.tensor_product(*[t.data_ptr() for t in (*outs, *state["ops"])], n, case["pairs"] * case["L"],
                            [q for q, _ in state["mods"]], case["factor"], s)
        return outs
    ntts, x, y = state["ntts"], state["x"], outs[0]
    count, xp, yp = x.shape[0], x.data_ptr(), y.data_ptr()
    if kind == "single":
        t, q = ntts[0], state["mods"][0][0]
        zp = outs[1].data_ptr()
        t.forward(yp, xp, 1, 1, s)
        t.forward(yp + 8 * n, xp + 8 * n, 1, 1, s)
        capi.mul(zp, yp, yp + 8 * n, n, q, 1, s)
        capi.add(zp, zp, state["scalar"], n, q, s, scalar=True)
        t.inverse(zp + 8 * n, zp, 1, 1, s)
        return outs
    if kind == "forward":
        capi.forward_batch(ntts, yp, xp, count, case["in_f"], case["out_f"], s)
    elif kind == "inverse":
        capi.inverse_batch(ntts, yp, xp, count, case["in_f"], case["out_f"], s)
    elif kind == "roundtrip":
        capi.forward_batch(ntts, yp, xp, count, 1, 4, s)
        capi.inverse_batch(ntts, outs[1].data_ptr(), yp, count, 4, 1, s)
    elif kind == CHAIN_MUL:
        capi.chain_mul_batch(ntts, yp, xp, state["v"].data_ptr(), count, case["in_f"], case["out_f"], s)
    elif kind == CHAIN_FMA:
        capi.chain_fma_batch(ntts, yp, xp, state["scalars"], state["v"].data_ptr(), count, case["in_f"],
                             case["out_f"], s)
    elif kind == "product":
        capi.product_batch(ntts, yp, xp, state["v"].data_ptr(), count, 4, case["out_f"], s)
    elif kind == "halves":
        capi.forward_mul_batch(ntts, yp, xp, state["v"].data_ptr(), count, s)
        capi.mul_inverse_batch(ntts, outs[1].data_ptr(), xp, state["v"].data_ptr(), count, case["out_f"], s)
    return outs


def work(case):
    """Bytes: every operand read once and every output written once, twiddles
    {w, quotient} of each modulus read once per direction.  flops: 64-bit
    integer operations, six per butterfly (three products, three additions)
    and about as many per element-wise product."""
    kind = case["kind"]
    if kind == "eltwise":
        return {"bytes": 8 * case["n"] * 6, "flops": 14 * case["n"]}
    if kind in ("uneven", "serve"):
        b = f = 0
        for k, n, mods, _, _, _ in _limb_jobs(case):
            chain = k in (CHAIN_MUL, CHAIN_FMA)
            b += len(mods) * n * ((24 + 32) if chain else (16 + 16))
            f += len(mods) * (3 * n * (n.bit_length() - 1) * (2 if chain else 1) + (6 * n if chain else 0))
        return {"bytes": b, "flops": f}
    n = 1 << case["logn"]
    if kind == "single":
        return {"bytes": 8 * n * 10 + 32 * n, "flops": 3 * (3 * n * case["logn"]) + 8 * n}
    if kind == "tensor":
        words = case["pairs"] * case["L"] * n
        return {"bytes": 56 * words, "flops": 24 * words}
    words = case["polys"] * case["L"] * n
    table = 16 * n * case["L"]
    one = 3 * words * case["logn"]
    if kind in ("forward", "inverse"):
        return {"bytes": 16 * words + table, "flops": one}
    if kind == "roundtrip":
        return {"bytes": 24 * words + 2 * table, "flops": 2 * one}
    if kind == "halves":
        return {"bytes": 32 * words + 2 * table, "flops": 2 * one + 12 * words}
    return {"bytes": 24 * words + 2 * table, "flops": 2 * one + 6 * words}


# ------------------------------------------------------------------- exact
# Unsigned 64-bit arithmetic on int64 tensors; every value is below 2^63.

_M32 = 0xFFFFFFFF


def _mulhi(a, b):
    a0, a1, b0, b1 = a & _M32, (a >> 32) & _M32, b & _M32, (b >> 32) & _M32
    mid = a1 * b0 + (((a0 * b0) >> 32) & _M32)
    mid2 = a0 * b1 + (mid & _M32)
    return a1 * b1 + ((mid >> 32) & _M32) + ((mid2 >> 32) & _M32)


def _shoup(v, w, wq, q):
    return v * w - _mulhi(v, wq) * q


def _csub(x, bound):
    return torch.where(x >= bound, x - bound, x)


def _mulmod(a, b, q):
    """a * b mod q for a, b < q < 2^60, two bits of b at a time."""
    r = torch.zeros_like(a)
    for i in range(58, -2, -2):
        r = (4 * r + a * ((b >> i) & 3)).remainder_(q)
    return r


def _column(v):
    """Python integers below 2^64 as an int64 column."""
    return torch.from_numpy(np.array(v, dtype=np.uint64).view(np.int64)).to(_device()).unsqueeze(-1)


def _powers(base, count, q):
    out = [1] * count
    for i in range(1, count):
        out[i] = out[i - 1] * base % q
    return out


@functools.lru_cache(maxsize=8)
def _tables(n, mods):
    """psi^bitrev(i) and psi^-bitrev(i) with their Shoup quotients: the forward
    stage of m blocks takes entries m .. 2m-1 of the first table, the inverse
    stage of m blocks those of the second.  (moduli, n) each."""
    bits = n.bit_length() - 1
    i = np.arange(n)
    rev = sum(((i >> b) & 1) << (bits - 1 - b) for b in range(bits))
    out = [np.empty((len(mods), n), np.uint64) for _ in range(4)]
    for i, (q, psi) in enumerate(mods):
        for k, base in enumerate((psi, pow(psi, -1, q))):
            p = _powers(base, n, q)
            out[2 * k][i] = np.array(p, dtype=np.uint64)[rev]
            out[2 * k + 1][i] = np.array([(v << 64) // q for v in p], dtype=np.uint64)[rev]
    return [torch.from_numpy(a.view(np.int64)).to(_device()) for a in out]


def _mod_index(rows, L):
    return torch.arange(rows, device=_device()) % L


def _forward(x, n, mods, lazy):
    """Cooley-Tukey, x in [0, 4q), as the reference's native forward transform."""
    w_all, wq_all, _, _ = _tables(n, mods)
    idx = _mod_index(x.shape[0], len(mods))
    q = _column([m for m, _ in mods])[idx].unsqueeze(-1)
    x = x.clone()
    m, t = 1, n // 2
    while m < n:
        v = x.view(x.shape[0], m, 2, t)
        w, wq = (a[idx, m:2 * m].unsqueeze(-1) for a in (w_all, wq_all))
        g, p = _csub(v[:, :, 0], 2 * q), _shoup(v[:, :, 1], w, wq, q)
        v[:, :, 0], v[:, :, 1] = g + p, g + 2 * q - p
        m, t = 2 * m, t // 2
    q = q.squeeze(-1)
    return x if lazy else _csub(_csub(x, 2 * q), q)


def _inverse(x, n, mods, lazy):
    """Gentleman-Sande, x in [0, 2q), N^-1 in the last stage."""
    _, _, w_all, wq_all = _tables(n, mods)
    idx = _mod_index(x.shape[0], len(mods))
    qs = [m for m, _ in mods]
    q = _column(qs)[idx].unsqueeze(-1)
    x = x.clone()
    m, t = n // 2, 1
    while m > 1:
        v = x.view(x.shape[0], m, 2, t)
        w, wq = (a[idx, m:2 * m].unsqueeze(-1) for a in (w_all, wq_all))
        a, b = v[:, :, 0].clone(), v[:, :, 1].clone()
        v[:, :, 0], v[:, :, 1] = _csub(a + b, 2 * q), _shoup(a + 2 * q - b, w, wq, q)
        m, t = m // 2, 2 * t
    ninv = [pow(n, -1, m) for m in qs]
    last = [pow(p, -(n // 2), m) * v % m for (m, p), v in zip(mods, ninv)]
    c = [_column(v)[idx] for v in (ninv, [(a << 64) // m for a, m in zip(ninv, qs)], last,
                                   [(a << 64) // m for a, m in zip(last, qs)])]
    q = q.squeeze(-1)
    a, b = _csub(x[:, :n // 2], 2 * q), x[:, n // 2:]
    x = torch.cat([_shoup(a + b, c[0], c[1], q), _shoup(a + 2 * q - b, c[2], c[3], q)], dim=1)
    return x if lazy else _csub(x, q)


def _apply(kind, x, v, n, mods, in_f, out_f, scalars=None):
    """One limb job; x (rows, n), row i under modulus i mod len(mods)."""
    mods = tuple(mods)
    if kind == "forward":
        return _forward(x, n, mods, out_f == 4)
    q = _column([m for m, _ in mods])[_mod_index(x.shape[0], len(mods))]
    if in_f == 4:
        x = _csub(x, 2 * q)
    if kind == "inverse":
        return _inverse(x, n, mods, out_f == 2)
    y = _csub(_inverse(x, n, mods, True), q)
    if kind == CHAIN_MUL:
        y = _mulmod(y, _csub(v, q), q)
    else:
        sc = _column([s - m if s >= m else s for s, (m, _) in zip(scalars, mods)])
        sc = sc[_mod_index(x.shape[0], len(mods))]
        y = _csub(_mulmod(y, sc.expand_as(y), q) + _csub(v, q), q)
    return _forward(y, n, mods, out_f == 4)


def exact(case, seed):
    kind = case["kind"]
    d = _inputs(case, seed)
    if kind in ("uneven", "serve"):
        if sum(n * len(mods) for _, n, mods, *_ in d["jobs"]) > 1 << 22:
            return None  # tables of so many moduli take longer than 20 seconds here
        return [_apply(k, x, v, n, mods, in_f, out_f, sc)
                for (k, n, mods, in_f, out_f, sc), (x, v) in zip(d["jobs"], d["ops"])]
    if kind == "eltwise":
        q, f, a, b = d["q"], case["factor"], d["a"], d["b"]
        ar, br = a % q, b % q
        sc = torch.full_like(a, d["scalar"] % q)
        m = _mulmod(ar, br, q)
        s = _csub(_mulmod(ar, sc, q) + br, q)
        return [m, s, ar, _csub(m + s, q)]
    n, mods = 1 << case["logn"], tuple(d["mods"])
    if kind == "tensor":
        L = case["L"]
        q = _column([m for m, _ in mods])[_mod_index(case["pairs"] * L, L)]
        c0, c1, d0, d1 = (t % q for t in d["ops"])
        mid = _csub(_mulmod(c0, d1, q) + _mulmod(c1, d0, q), q)
        return [_mulmod(c0, d0, q), mid, _mulmod(c1, d1, q)]
    x = d["x"]
    if kind == "single":
        q = mods[0][0]
        y = _forward(x, n, mods, False)
        z = (_mulmod(y[:1], y[1:], q) + d["scalar"]) % q
        return [y, torch.cat([z, _inverse(z, n, mods, False)])]
    if kind == "roundtrip":
        L = case["L"]
        y, z = torch.empty_like(x), torch.empty_like(x)
        step = max(1, (1 << 24) // (n * L)) * L  # bounded temporaries
        q = _column([m for m, _ in mods])
        for i in range(0, x.shape[0], step):
            y[i:i + step] = _forward(x[i:i + step], n, mods, True)
            r = _csub(y[i:i + step], 2 * q[_mod_index(y[i:i + step].shape[0], L)])
            z[i:i + step] = _inverse(r, n, mods, False)
        return [y, z]
    if kind in ("product", "halves"):
        q = _column([m for m, _ in mods])[_mod_index(x.shape[0], len(mods))]
        v = d["v"] % q
        fm = _mulmod(_forward(x, n, mods, False), v, q)
        if kind == "product":
            return [_inverse(fm, n, mods, case["out_f"] == 2)]
        return [fm, _inverse(_mulmod(x % q, v, q), n, mods, case["out_f"] == 2)]
    return [_apply(kind, x, d.get("v"), n, mods, case["in_f"], case["out_f"], d.get("scalars"))]
