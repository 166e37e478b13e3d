"""Which plan a call runs: the tuned one where no modulus has another form than
the reference's butterflies, and one set by hand exactly as it was set."""
import numpy as np
import pytest

from helpers import dev, dev_empty, host, ptr

pytestmark = pytest.mark.gpu


def passes_run(cuda, call):
    """(lg, lr, tg) of the forward and inverse pass kernels a call launches, by kind."""
    cuda.profile_enable(True)
    try:
        cuda.profile_report()
        call()
        rep = cuda.profile_report()
    finally:
        cuda.profile_enable(False)
    out = {"fwd": set(), "inv": set()}
    for name in rep:
        if name.startswith(("ntt_fwd_pass", "ntt_inv_pass")):
            f = dict(p.split("=") for p in name.split()[1:])
            out[name[4:7]].add((int(f["lg"]), int(f["lr"]), int(f["tg"])))
    return out


def make(cuda, oracle, n, bits, external):
    q = oracle.find_ntt_prime_near(n, bits, 1, 1)
    psi = oracle.find_primitive_root(n, q)
    tabs = oracle.tables(n, q, psi)
    return q, tabs, cuda.NTT(n, q, tables=tabs) if external else cuda.NTT(n, q, psi)


# moduli from 2^59 on and caller-provided tables have the reference's form only
@pytest.mark.parametrize("bits,external", [(60, False), (45, True)])
def test_exact_moduli_run_the_tuned_plan(cuda, oracle, bits, external):
    n, count = 65536, 64
    q, (fwd, inv, ninv), t = make(cuda, oracle, n, bits, external)
    x = np.random.default_rng(bits).integers(0, q, (count, n), dtype=np.uint64)
    d, o = dev(x), dev_empty(count * n)
    run = passes_run(cuda, lambda: cuda.forward_batch([t], ptr(o), ptr(d), count, 1, 1))
    assert run["fwd"] == set(cuda.plan_get(False, 16, count))
    np.testing.assert_array_equal(host(o, n), oracle.forward(x[0], q, fwd, 1, 1))
    run = passes_run(cuda, lambda: cuda.inverse_batch([t], ptr(o), ptr(d), count, 1, 1))
    plan = cuda.plan_get(True, 16, count)
    assert run["inv"] == set(plan)
    np.testing.assert_array_equal(host(o, n), oracle.inverse(x[0], q, inv, ninv, 1, 1))
    # the passes beside the fused one
    run = passes_run(cuda, lambda: cuda.chain_mul_batch([t], ptr(o), ptr(d), ptr(d), count, 1, 1))
    assert (run["inv"], run["fwd"]) == ({plan[0]}, {plan[0]})
    run = passes_run(cuda, lambda: cuda.product_batch([t], ptr(o), ptr(d), ptr(d), count, 1, 1))
    assert (run["inv"], run["fwd"]) == ({plan[1]}, {plan[1]})
    want = oracle.inverse(oracle.mul(oracle.forward(x[0], q, fwd, 1, 4), x[0], q, 4), q, inv, ninv, 2, 1)
    np.testing.assert_array_equal(host(o, n), want)


@pytest.mark.parametrize("phased", [False, True])
def test_batches_of_exact_moduli(cuda, oracle, phased):
    """Jobs whose moduli have the reference's form only beside one that has others:
    each as its direct call, launched by class (small jobs together, a large one
    alone) and as one launch."""
    jobs = [(n, bits, external, count, kind, out_f) for bits, external in [(60, False), (45, True), (45, False)]
            for n, count in [(4096, 3), (32768, 40)]
            for kind, out_f in [(cuda.JOB_FORWARD, 1), (cuda.JOB_INVERSE, 1), (cuda.JOB_CHAIN_MUL, 1),
                                (cuda.JOB_CHAIN_MUL, 4)]]
    rng = np.random.default_rng(60)
    specs, outs, wants, ctx = [], [], [], {}
    for n, bits, external, count, kind, out_f in jobs:
        if (n, bits, external) not in ctx:
            ctx[n, bits, external] = make(cuda, oracle, n, bits, external)
        q, _, t = ctx[n, bits, external]
        x, m = (dev(rng.integers(0, q, count * n, dtype=np.uint64)) for _ in range(2))
        o, w = dev_empty(count * n), dev_empty(count * n)
        specs.append(dict(kind=kind, ntts=[t], count=count, result=ptr(o), operand=ptr(x), vector=ptr(m), in_f=1,
                          out_f=out_f, keep=(x, m)))
        if kind == cuda.JOB_FORWARD:
            cuda.forward_batch([t], ptr(w), ptr(x), count, 1, out_f)
        elif kind == cuda.JOB_INVERSE:
            cuda.inverse_batch([t], ptr(w), ptr(x), count, 1, out_f)
        else:
            cuda.chain_mul_batch([t], ptr(w), ptr(x), ptr(m), count, 1, out_f)
        outs.append(o)
        wants.append(w)
    b = cuda.Batch(specs)
    b.launch(phased=phased)
    assert b.status() == 0
    for o, w, j in zip(outs, wants, jobs):
        np.testing.assert_array_equal(host(o), host(w), err_msg=str(j))
    b.close()


def test_small_jobs_of_wide_moduli_share_their_launches(cuda, oracle):
    """Small jobs without FP64 moduli, lazy and normalized outputs: one launch per
    phase, class and pass width, as for the reference's butterflies."""
    n, count = 4096, 3
    q, (fwd, inv, ninv), t = make(cuda, oracle, n, 55, False)
    rng = np.random.default_rng(55)
    x = [rng.integers(0, q, (count, n), dtype=np.uint64) for _ in range(4)]
    d, outs = [dev(v) for v in x], [dev_empty(count * n) for _ in x]
    b = cuda.Batch([dict(kind=cuda.JOB_FORWARD, ntts=[t], count=count, result=ptr(o), operand=ptr(i), in_f=1,
                         out_f=(1, 4)[j % 2]) for j, (i, o) in enumerate(zip(d, outs))])
    b.launch(phased=True)
    before = cuda.launch_count()
    b.launch(phased=True)
    assert cuda.launch_count() - before == 2
    for j, o in enumerate(outs):
        want = np.stack([oracle.forward(v, q, fwd, 1, (1, 4)[j % 2]) for v in x[j]])
        np.testing.assert_array_equal(host(o).reshape(count, n), want)
    b.close()


# 16 registers per thread (the reference's butterflies), and 8 with tiles wider
# than the relaxed modes' own
@pytest.mark.parametrize("bits", [45, 55])
@pytest.mark.parametrize("col,row", [((7, 4, 16), (7, 4, 16)), ((7, 3, 32), (7, 3, 16))])
def test_forced_plans_run_as_set(cuda, oracle, bits, col, row):
    n, count = 16384, 40
    q, (fwd, inv, ninv), t = make(cuda, oracle, n, bits, False)
    rng = np.random.default_rng(bits)
    x, m = (rng.integers(0, q, (count, n), dtype=np.uint64) for _ in range(2))
    d, e, o = dev(x), dev(m), dev_empty(count * n)
    want = {
        "forward": lambda a, b: oracle.forward(a, q, fwd, 1, 1),
        "inverse": lambda a, b: oracle.inverse(a, q, inv, ninv, 1, 1),
        "chain": lambda a, b: oracle.forward(oracle.mul(oracle.inverse(a, q, inv, ninv, 1, 2), b, q, 2), q, fwd, 1, 1),
        "product": lambda a, b: oracle.inverse(oracle.mul(oracle.forward(a, q, fwd, 1, 4), b, q, 4), q, inv, ninv, 2, 1),
    }
    call = {
        "forward": lambda: cuda.forward_batch([t], ptr(o), ptr(d), count, 1, 1),
        "inverse": lambda: cuda.inverse_batch([t], ptr(o), ptr(d), count, 1, 1),
        "chain": lambda: cuda.chain_mul_batch([t], ptr(o), ptr(d), ptr(e), count, 1, 1),
        "product": lambda: cuda.product_batch([t], ptr(o), ptr(d), ptr(e), count, 1, 1),
    }
    passes = {"forward": {"fwd": {col, row}, "inv": set()}, "inverse": {"fwd": set(), "inv": {row, col}},
              "chain": {"fwd": {row}, "inv": {row}}, "product": {"fwd": {col}, "inv": {col}}}
    try:
        cuda.plan_set(False, 14, [col, row])
        cuda.plan_set(True, 14, [row, col])
        for name in want:
            assert passes_run(cuda, call[name]) == passes[name], name
            got = host(o).reshape(count, n)
            for i in (0, count - 1):
                np.testing.assert_array_equal(got[i], want[name](x[i], m[i]), err_msg=f"{name}: limb {i}")
    finally:
        cuda.plan_set(False, 14, [])
        cuda.plan_set(True, 14, [])


def plans(logn):
    """Splits of a forward, outermost stages first, whose passes hold the relaxed
    modes (8 registers per thread, groups of 2^4 .. 2^12), with the narrowest,
    a middle and the widest tiles; three passes; and passes without those modes."""
    def widths(lg, most):
        top = min(most, 512 >> (lg - 3))
        return sorted({1, min(8, top), top})

    out = [[(logn, 3, 1)]] if 4 <= logn <= 12 else []
    for col in range(4, min(12, logn - 4) + 1):
        row = logn - col
        if not 4 <= row <= 12:
            continue
        cw, rw = widths(col, 1 << row), widths(row, 1 << col)
        out += [[(col, 3, cw[i % len(cw)]), (row, 3, rw[-1 - i % len(rw)])] for i in range(3)]
    if logn >= 12:
        a, b = logn // 3, (logn - logn // 3) // 2
        out += [[(a, 3, 8), (b, 3, 16), (logn - a - b, 3, 4)], [(b, 3, 16), (logn - a - b, 3, 1), (a, 3, 16)],
                [(logn // 2, 4, 8), (logn - logn // 2, 3, 8)], [(logn // 2, 3, 8), (logn - logn // 2, 5, 4)]]
    return out


# An odd number of limbs per modulus (pairs and a last one alone), from N = 2^9 on
# enough residues for two limbs per thread; moduli of every arithmetic, one with caller-provided tables.
@pytest.mark.parametrize("logn,polys", [(6, 5), (9, 949), (11, 239), (12, 119), (13, 61), (14, 31), (16, 9),
                                        (17, 7)])
def test_forms_under_every_plan(cuda, oracle, logn, polys):
    import torch

    n, bits = 1 << logn, [(45, 1, 2), (50, 1, 1), (58, 1, 2), (60, 1, 2), (44, 1, 2)]
    qs = [oracle.find_ntt_prime_near(n, *b) for b in bits]
    psis = [oracle.find_primitive_root(n, q) for q in qs]
    tabs = [oracle.tables(n, q, psi) for q, psi in zip(qs, psis)]
    ntts = cuda.NTT.create_many(list(zip([n] * 4, qs, psis))) + [cuda.NTT(n, qs[4], tables=tabs[4])]
    L, count = len(qs), len(qs) * polys
    rng = np.random.default_rng(logn)
    x4, m4, x2, m2 = (np.stack([rng.integers(0, f * qs[i % L], n, dtype=np.uint64) for i in range(count)])
                      for f in (4, 4, 2, 2))
    sc = [(2 * q) // 3 for q in qs]

    def limbs(f):
        return dev(np.concatenate([f(i, qs[i % L], *tabs[i % L]) for i in range(count)]))

    fwd = lambda v, q, t, f=1: oracle.forward(v, q, t, 1, f)
    inv = lambda v, q, t, ninv, f=1: oracle.inverse(v, q, t, ninv, 2, f)
    lazy = [fwd(x4[i], qs[i % L], tabs[i % L][0], 4) for i in range(count)]
    prod = [oracle.mul(lazy[i], m4[i], qs[i % L], 4) for i in range(count)]
    back = [inv(x2[i], qs[i % L], tabs[i % L][1], tabs[i % L][2], 2) for i in range(count)]
    d4, e4, d2, e2, o = dev(x4), dev(m4), dev(x2), dev(m2), dev_empty(count * n)
    P, c = ptr, count
    ops = {
        "forward 4": (limbs(lambda i, *_: lazy[i]), lambda: cuda.forward_batch(ntts, P(o), P(d4), c, 4, 4)),
        "forward 1": (limbs(lambda i, q, *_: oracle.reduce(lazy[i], q, 4, 1)),
                      lambda: cuda.forward_batch(ntts, P(o), P(d4), c, 4, 1)),
        "forward mul": (limbs(lambda i, *_: prod[i]), lambda: cuda.forward_mul_batch(ntts, P(o), P(d4), P(e4), c)),
        "inverse 2": (limbs(lambda i, *_: back[i]), lambda: cuda.inverse_batch(ntts, P(o), P(d2), c, 2, 2)),
        "inverse 1": (limbs(lambda i, q, *_: oracle.reduce(back[i], q, 2, 1)),
                      lambda: cuda.inverse_batch(ntts, P(o), P(d2), c, 2, 1)),
        "mul inverse": (limbs(lambda i, q, f, t, ninv: inv(oracle.mul(x4[i], m4[i], q, 4), q, t, ninv)),
                        lambda: cuda.mul_inverse_batch(ntts, P(o), P(d4), P(e4), c, 1)),
        "chain mul 1": (limbs(lambda i, q, t, *_: fwd(oracle.mul(back[i], m2[i], q, 2), q, t)),
                        lambda: cuda.chain_mul_batch(ntts, P(o), P(d2), P(e2), c, 2, 1)),
        "chain fma 4": (limbs(lambda i, q, t, *_: fwd(oracle.fma(back[i], sc[i % L], m2[i], q, 2), q, t, 4)),
                        lambda: cuda.chain_fma_batch(ntts, P(o), P(d2), sc, P(e2), c, 2, 4)),
        "product 1": (limbs(lambda i, q, f, t, ninv: inv(prod[i], q, t, ninv)),
                      lambda: cuda.product_batch(ntts, P(o), P(d4), P(e4), c, 4, 1)),
        "product 2": (limbs(lambda i, q, f, t, ninv: inv(prod[i], q, t, ninv, 2)),
                      lambda: cuda.product_batch(ntts, P(o), P(d4), P(e4), c, 4, 2)),
    }
    ran = dict.fromkeys(ops, 0)
    try:
        for plan in plans(logn):
            cuda.plan_set(False, logn, plan)
            try:
                cuda.plan_set(True, logn, plan[::-1])  # its tiles may not fit the inverse's strides
            except cuda.AxhelError:
                cuda.plan_set(True, logn, [])
            for name, (want, run) in ops.items():
                o.fill_(-1)
                try:
                    run()
                except cuda.AxhelError:
                    # a chain or product runs the inverse plan's passes both ways round
                    assert name[:7] in ("chain m", "chain f", "product"), name
                    continue
                ran[name] += 1
                assert torch.equal(o, want), f"{name} under {plan}"
    finally:
        cuda.plan_set(False, logn, [])
        cuda.plan_set(True, logn, [])
    assert min(ran.values()) >= 1, ran
