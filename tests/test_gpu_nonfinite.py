"""Non-finite tables: a result that is not a number stays one.  Only a branch of probability 0 is -inf.

A matrix with a NaN or an infinity, and a resume whose slices add up to zeros, on plans that are one run (n = 16) and on
plans with wide steps (n = 36, one pass per step): the oracle's NaNs in the same places."""
import os
import tempfile

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def with_row(plan, k, b, value):
    """The plan text with step k's row M[b] set to (value, 0) (value, 0)."""
    lines = plan.strip().split("\n")
    t = lines[k + 1].split()
    t[len(t) - 8 + 4 * b:len(t) - 4 + 4 * b] = [value, "0", value, "0"]
    lines[k + 1] = " ".join(t)
    return "\n".join(lines) + "\n"


@pytest.mark.parametrize("prec", [128, 64])
@pytest.mark.parametrize("n", [16, 36])
def test_nan_matrix(n, prec):
    import gsb
    import workloads
    from oracle import Oracle
    w = workloads.matching_instance(n, n, 11, 8, 20000)
    ns = len(w["steps"])
    strings = workloads.random_strings(ns, 6, seed=2)
    for k in range(0, ns, 5):
        strings[::2, k] = 1
        strings[1::2, k] = 0
        text = with_row(w["plan"], k, 1, "nan")
        path = os.path.join(tempfile.mkdtemp(), "plan.txt")
        open(path, "w").write(text)
        o = Oracle(path, prec)
        with gsb.Engine(path, precision=prec) as eng:
            eng.set_fusion(1)
            lp, cond = eng.chain(strings)
            plp = eng.prob(strings)
            bits, slp = eng.sample(2, 3)
            hb, hlp, hc = eng.hybrid(strings, 1)
            for i, s in enumerate(strings):
                r, c = o.chain1(s)
                assert np.isnan(lp[i]) == np.isnan(r) == bool(s[k])
                assert (np.isnan(cond[i]) == np.isnan(c)).all()
                assert np.isnan(plp[i]) and np.isnan(o.prob(s))     # both branch norms enter
                assert np.isnan(hlp[i]) == np.isnan(o.hybrid(s, 1, i)[1]) == bool(s[k])
                assert (np.isnan(hc[i]) == np.isnan(o.hybrid(s, 1, i)[2])).all() and (hb[i] == s).all()
            assert np.isnan(slp).all()
            for i in range(2):
                assert list(bits[i]) == list(o.sample(0, 3, i)[0])
            dump, ls, pre = eng.prefix(strings[0], k + 1)
            assert np.isnan(pre) and np.isnan(dump).all()
        o.close()


@pytest.mark.parametrize("prec", [128, 64])
@pytest.mark.parametrize("n", [16, 36])
def test_infinite_matrix(n, prec):
    """An infinite entry leaves infinities or NaNs, never an impossible string."""
    import gsb
    import workloads
    w = workloads.matching_instance(n, n, 11, 8, 20000)
    ns = len(w["steps"])
    strings = workloads.random_strings(ns, 3, seed=4)
    for k in range(0, ns, 5):
        strings[:, k] = 1
        with gsb.Engine.from_text(with_row(w["plan"], k, 1, "inf"), precision=prec) as eng:
            eng.set_fusion(1)
            for lp in (eng.chain(strings)[0], eng.prob(strings), eng.hybrid(strings, 1)[1]):
                assert (np.isnan(lp) | (lp == np.inf)).all()


@pytest.mark.parametrize("prec", [128, 64])
@pytest.mark.parametrize("n", [16, 36])
def test_resume_of_zeros(n, prec):
    """Slices that add up to a table of zeros: log2 Pr(prefix) is -inf, and nothing after it is a number."""
    import gsb
    import workloads
    from oracle import Oracle
    w = workloads.matching_instance(n, n, 11, 8, 20000)
    ns = len(w["steps"])
    path = os.path.join(tempfile.mkdtemp(), "plan.txt")
    open(path, "w").write(w["plan"])
    o = Oracle(path, prec)
    with gsb.Engine(path, precision=prec) as eng:
        for K in range(1, ns - 3, 4):
            line = np.random.default_rng(K).integers(0, 2, ns)
            line[-3:] = -1
            nothing = np.zeros_like(eng.prefix(line, K)[0])
            bits, full, pre, cond = eng.resume(line, K, 5, 0, [nothing], [0.0])
            obits, ofull, opre, ocond = o.resume(line, K, 5, 0, [nothing.astype(complex)], [0.0])
            assert pre == opre == -np.inf and np.isnan(full) and np.isnan(ofull)
            assert list(bits) == list(obits)
            assert np.isnan(cond[K:]).all() and np.isnan(ocond[K:]).all()
    o.close()
