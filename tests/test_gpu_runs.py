"""Runs of small steps (one CTA per string, the table in shared memory): started, ended and split at every step.

A prefix to K and a resume from K cut the runs of both ends there, and the wide steps between them; the whole string,
and one step alone, are the extremes.  Against the oracle."""
import os
import tempfile

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [128, 64])
@pytest.mark.parametrize("n", [16, 36])
def test_prefix_and_resume_at_every_step(n, prec):
    """complex128 to the parity bound; complex64 tables to 16 roundings of an entry (the steps that mix one), its
    log2 Pr to 1e-5."""
    import gsb
    import workloads
    from oracle import Oracle
    w = workloads.matching_instance(n, n, 11, 8, 20000)
    ns = len(w["steps"])
    path = os.path.join(tempfile.mkdtemp(), "plan.txt")
    open(path, "w").write(w["plan"])
    o = Oracle(path, prec)
    rng = np.random.default_rng(n)
    with gsb.Engine(path, precision=prec) as eng:
        for K in range(ns + 1):
            line = rng.integers(0, 2, ns)
            line[max(K, ns - 5):] = -1
            dump, ls, lp = eng.prefix(line, K)
            odump, ols, olp = o.prefix(line, K)
            tol = 1e-9 if prec == 128 else 16 * 2.0 ** -24
            assert np.abs(dump - odump).max() <= tol * np.linalg.norm(odump)
            assert abs(ls - ols) <= (1e-9 if prec == 128 else 1e-6)
            assert abs(lp - olp) <= (1e-9 if prec == 128 else 1e-5)
            if K == ns:
                continue
            bits, full, pre, cond = eng.resume(line, K, 5, 2, [dump], [ls])
            obits, ofull, opre, ocond = o.resume(line, K, 5, 2, [odump], [ols])
            assert list(bits) == list(obits)
            tol = 1e-9 if prec == 128 else max(1e-5, 6 * float(gsb.c64_sigma(ofull, ns)))
            assert abs(full - ofull) <= tol and abs(pre - opre) <= tol
            assert np.abs(np.log2(cond[K:] / ocond[K:])).max() <= 2 * tol
    o.close()


def test_runs_follow_new_matrices():
    """The step descriptors on the device are written again when the matrices change."""
    import gsb
    import workloads
    w = workloads.matching_instance(20, 20, 11, 8, 20000)
    w2 = workloads.build(w["n"], w["body"], workloads.circuits.matching_circuit(20, 20, seed=12)[2], w["order"])[0]
    strings = workloads.random_strings(len(w["steps"]), 7, seed=1)
    with gsb.Engine.from_text(w["plan"], precision=128) as a, gsb.Engine.from_text(w2, precision=128) as b:
        first = a.chain(strings)[0]
        a.set_matrices_from_text(w2)
        second = a.chain(strings)[0]
        assert (second == b.chain(strings)[0]).all() and (first != second).any()
