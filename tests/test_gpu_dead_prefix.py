"""Prefixes of probability 0: the dump is a table of zeros, whatever the engine evaluated before, so that a slice that
cannot contribute adds nothing to a resume.

A step whose matrix row for bit 1 is zero ends every prefix that takes bit 1 there, in exact arithmetic."""
import os
import tempfile

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORACLE_FREE = 5   # sampled steps of the resumed lines at most


def without_bit_one(plan, k):
    """The plan text with step k's row M[1] set to zeros."""
    lines = plan.strip().split("\n")
    lines[k + 1] = " ".join(lines[k + 1].split()[:-4] + ["0", "0", "0", "0"])
    return "\n".join(lines) + "\n"


def instance(n, k, prec):
    """Plan text (step k never takes bit 1) of an instance that is one run (n = 16) or has wide steps (n = 36)."""
    import workloads
    from oracle import Oracle
    w = workloads.matching_instance(n, n, 11, 8, 20000)
    text = without_bit_one(w["plan"], k)
    path = os.path.join(tempfile.mkdtemp(), "plan.txt")
    open(path, "w").write(text)
    return text, len(w["steps"]), Oracle(path, prec)


@pytest.mark.parametrize("prec", [128, 64])
@pytest.mark.parametrize("n", [16, 36])
def test_dead_prefix_dumps_zeros(n, prec):
    """Dead at its last step (the oracle dumps the zeros that step wrote) or at an earlier one, after a live prefix."""
    import gsb
    rng = np.random.default_rng(n)
    for k in range(0, n, 3):
        text, ns, o = instance(n, k, prec)
        with gsb.Engine.from_text(text, precision=prec) as eng:
            for K in sorted({k + 1, min(k + 4, ns), ns}):
                line = rng.integers(0, 2, ns)
                line[k] = 0
                live, _, lp = eng.prefix(line, K)
                assert np.isfinite(lp) and np.abs(live).max() > 0
                line[k] = 1
                dump, ls, lp = eng.prefix(line, K)
                odump, ols, olp = o.prefix(line, K)
                assert lp == olp == -np.inf and abs(ls - ols) <= 1e-6
                assert dump.shape == live.shape and not dump.any()
                if K == k + 1:
                    assert not odump.any()
        o.close()


@pytest.mark.parametrize("prec", [128, 64])
@pytest.mark.parametrize("n", [16, 36])
def test_resume_with_a_dead_slice(n, prec):
    """A live and a dead slice, in both orders, against the oracle's sum of the same two."""
    import gsb
    for k in range(1, n - 6, 4):
        K = k + 1
        text, ns, o = instance(n, k, prec)
        line = np.random.default_rng(k).integers(0, 2, ns)
        line[max(K, ns - ORACLE_FREE):] = -1
        with gsb.Engine.from_text(text, precision=prec) as eng:
            got, want = [], []
            for bit in (0, 1):
                line[k] = bit
                got.append(eng.prefix(line, K)[:2])
                want.append(o.prefix(line, K)[:2])
            line[k] = 0
            for order in ([0, 1], [1, 0]):
                bits, full, pre, cond = eng.resume(line, K, 5, 2, [got[i][0] for i in order], [got[i][1] for i in order])
                obits, ofull, opre, ocond = o.resume(line, K, 5, 2, [want[i][0] for i in order], [want[i][1] for i in order])
                tol = 1e-9 if prec == 128 else max(1e-5, 6 * float(gsb.c64_sigma(ofull, ns)))
                assert list(bits) == list(obits)
                assert abs(full - ofull) <= tol and abs(pre - opre) <= tol
                assert np.abs(np.log2(cond[K:] / ocond[K:])).max() <= 2 * tol
        o.close()
