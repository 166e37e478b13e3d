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
    # the passes beside the fused one, and a batch's
    run = passes_run(cuda, lambda: cuda.chain_mul_batch([t], ptr(o), ptr(d), ptr(d), count, 1, 1))
    assert (run["inv"], run["fwd"]) == ({plan[0]}, {plan[0]})
    run = passes_run(cuda, lambda: cuda.product_batch([t], ptr(o), ptr(d), ptr(d), count, 1, 1))
    assert (run["inv"], run["fwd"]) == ({plan[1]}, {plan[1]})
    want = oracle.inverse(oracle.mul(oracle.forward(x[0], q, fwd, 1, 4), x[0], q, 4), q, inv, ninv, 2, 1)
    np.testing.assert_array_equal(host(o, n), want)


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
