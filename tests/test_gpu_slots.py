"""Calls that carry several strings or samples per launch (slots): every mode against the oracle, at string counts
around the slot counts (1, 2, 3, one more than a power of two) and at widths from a single small run (width 6) to
fused passes of two and three steps (width 18); zero-probability strings beside live ones; and the fused passes'
bounded wait running out in several slots at once."""
import os
import tempfile

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# complex128: the parity bound of the other tests (complex64: 6 standard deviations of its error model, c64_sigma)
TOL128 = 1e-9


@pytest.fixture(scope="module")
def instances():
    import workloads
    made = {}

    def get(n):
        if n not in made:
            w = workloads.matching_instance(n, n, 7, 8, 20000)
            w["path"] = os.path.join(tempfile.mkdtemp(), "plan.txt")
            open(w["path"], "w").write(w["plan"])
            made[n] = w
        return made[n]
    return get


@pytest.mark.parametrize("prec", [128, 64])
@pytest.mark.parametrize("n,count", [(18, 1), (18, 2), (18, 67), (29, 5), (33, 3), (38, 1), (38, 2), (38, 9), (44, 3)])
def test_counts_against_oracle(instances, n, count, prec):
    import gsb
    import workloads
    from oracle import Oracle
    w = instances(n)
    ns = len(w["steps"])
    strings = workloads.random_strings(ns, count, seed=n + count)
    free = strings.copy()
    free[:, ns // 3:ns // 2] = -1
    free[::2, -4:] = -1
    o = Oracle(w["path"], prec)

    def tol(lp):
        return TOL128 if prec == 128 else max(1e-6, 6 * float(gsb.c64_sigma(lp, ns)))
    with gsb.Engine(w["path"], precision=prec) as eng:
        for _ in range(2):                                   # the second call replays the graphs
            lp, cond = eng.chain(strings)
            plp = eng.prob(strings)
            bits, slp = eng.sample(count, 31, first=4)
            hb, hlp, hc = eng.hybrid(free, 77, first_line=3)
        for i in range(count):
            r, c = o.chain1(strings[i])
            assert abs(lp[i] - r) <= tol(r) and abs(plp[i] - r) <= tol(r)
            assert np.abs(np.log2(cond[i] / c)).max() <= 2 * tol(r)
            ob, r = o.sample(0, 31, 4 + i)
            assert list(bits[i]) == list(ob) and abs(slp[i] - r) <= tol(r)
            ob, r, c = o.hybrid(free[i], 77, 3 + i)
            assert list(hb[i]) == list(ob) and abs(hlp[i] - r) <= tol(r)
            assert np.abs(np.log2(hc[i] / c)).max() <= 2 * tol(r)
        eng.set_hybrid_prefix(ns // 3)
        hb2, hlp2, hc2 = eng.hybrid(free, 77, first_line=3)
        assert (hb2 == hb).all()
        for i in range(count):
            assert abs(hlp2[i] - hlp[i]) <= 2 * tol(hlp[i])
            assert np.abs(np.log2(hc2[i] / hc[i])).max() <= 2 * tol(hlp[i])
    o.close()


@pytest.mark.parametrize("prec", [128, 64])
@pytest.mark.parametrize("n", [16, 36])
def test_dead_strings_beside_live_ones(n, prec):
    """A bipartite graph state with one side measured in X: its bits are parities of the other side's, so a random
    string has probability 0 and a sampled one 2^-(n/2)."""
    import circuits
    import gsb
    import workloads
    from oracle import Oracle
    rng = np.random.default_rng(3)
    body = [("h", [q]) for q in range(n)]
    body += [("cz", [a, b]) for a in range(n // 2) for b in range(n // 2, n) if rng.random() < 0.5]
    body += [("h", [q]) for q in range(n // 2, n)]
    from graphform import graph_form
    A, _ = graph_form(circuits.tableau_of(n, body))
    order, _ = gsb.order_search(A, seed=8, ngreedy=4, iters=20000)
    text, st, R = workloads.build(n, body, [], order)
    path = os.path.join(tempfile.mkdtemp(), "plan.txt")
    open(path, "w").write(text)
    o = Oracle(path, prec)
    with gsb.Engine(path, precision=prec) as eng:
        bits, slp = eng.sample(6, 5)
        strings = workloads.random_strings(len(st), 13, seed=9)
        strings[1::4] = bits[:3]
        lp, _ = eng.chain(strings)
        plp = eng.prob(strings)
        # a zero is a difference of rounded numbers: at most (6e-8)^2 of a likely string's probability comes out
        ref = np.array([o.chain1(x)[0] for x in strings])
        live = ref > -n
        assert live[1::4].all() and not live.all()
        assert np.abs(lp[live] - ref[live]).max() <= 1e-5 and np.abs(plp[live] - ref[live]).max() <= 1e-5
        assert np.exp2(lp[~live]).max() <= 1e-12 and np.exp2(plp[~live]).max() <= 1e-12
        for i in range(6):
            ob, r = o.sample(0, 5, i)
            assert list(bits[i]) == list(ob) and abs(slp[i] - r) <= 1e-5
    o.close()


def test_bounded_wait_of_several_slots(instances):
    """Every slot's CTAs give up; the call reports it, and the engine works again with the hook off."""
    import gsb
    import workloads
    w = instances(38)
    strings = workloads.random_strings(len(w["steps"]), 5, seed=2)
    with gsb.Engine(w["path"], precision=128) as eng:
        eng.set_fusion(2)
        ref, _ = eng.chain(strings)
        eng.test_withhold_tile_loads(True)
        with pytest.raises(gsb.GsbError) as e:
            eng.chain(strings)
        assert e.value.code == 20 and "gave up waiting" in str(e.value)
        eng.test_withhold_tile_loads(False)
        assert (eng.chain(strings)[0] == ref).all()
