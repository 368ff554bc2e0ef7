"""'prob' runs one pass per step where every step conserves probability, and the normalised two-pass chain elsewhere: a plan
with scaled or mixed matrix rows, and one with a flipped term sign, against the oracle's two-pass chain."""
import os
import tempfile

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _changed(text, how, rng):
    """The plan with every third step's matrix or term signs changed."""
    rows = text.strip().split("\n")
    for k in range(1, len(rows), 3):
        r = rows[k].split()
        nk, nt = int(r[1]), int(r[5])
        if how == "rows":        # other row weights: no longer unitary
            r[-8:] = ["%.17g" % (float(x) * f) for x, f in zip(r[-8:], [1.3] * 4 + [0.6] * 4)]
        elif how == "mixed":     # columns no longer orthogonal
            r[-8:] = ["%.17g" % x for x in rng.normal(size=8)]
        elif nt >= 4:            # the sign of one x = 1 term: the coset map is no isometry any more
            terms = [6 + nk + 4 * i for i in range(nt)]
            i = [t for t in terms if r[t + 1] == "1"][-1]
            r[i + 3] = str(1 - int(r[i + 3]))
        rows[k] = " ".join(r)
    return "\n".join(rows) + "\n"


@pytest.mark.parametrize("prec", [128, 64])
@pytest.mark.parametrize("n", [18, 38])
@pytest.mark.parametrize("how", ["rows", "mixed", "signs", "none"])
def test_prob_is_the_normalised_chain(how, n, prec):
    import gsb
    import workloads
    from oracle import Oracle
    w = workloads.matching_instance(n, n, 5, 8, 20000)
    text = w["plan"] if how == "none" else _changed(w["plan"], how, np.random.default_rng(n))
    path = os.path.join(tempfile.mkdtemp(), "plan.txt")
    open(path, "w").write(text)
    strings = workloads.random_strings(len(w["steps"]), 5, seed=3)
    o = Oracle(path, prec)
    ref = np.array([o.prob(s) for s in strings])
    o.close()
    with gsb.Engine(path, precision=prec) as eng:
        lp = eng.prob(strings)
        assert np.abs(lp - ref).max() <= (1e-9 if prec == 128 else 1e-5 + 6 * gsb.c64_sigma(ref, len(w["steps"])).max())
        one = eng.chain(strings)[0]
        same = np.abs(one - ref).max() <= 1e-4
        assert same == (how == "none")          # the one-pass chain's number is another one on the changed plans
        # new matrices decide anew (the one-pass chain's number, from then on)
        if how in ("rows", "mixed"):
            eng.set_matrices_from_text(w["plan"])
            assert np.abs(eng.prob(strings) - eng.chain(strings)[0]).max() <= 1e-12
