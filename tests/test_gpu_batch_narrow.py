"""Narrow instances of a batch: a warp per item with its tables at hand (up to width 8) or in memory, items dealt out to the warps
or taken after wider ones, more items than warps; against the executor's complex128 'chain'."""
import numpy as np
import pytest

from test_gpu_batch_passes import _run
from test_gpu_dead_prefix import without_bit_one

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def narrow():
    """One instance per width 1 .. 9, 11 and 12."""
    import workloads
    found = {}
    for n in range(4, 36):
        w = workloads.matching_instance(n, n, n, 8, 2000)
        found.setdefault(w["width"], w)
    assert {1, 7, 8, 9, 11, 12} <= set(found)
    return [found[r] for r in sorted(found) if r <= 12]


@pytest.mark.parametrize("prec", [128, 64])
@pytest.mark.parametrize("shape", [None, (64, 24, 4), (128, 9, 1), (512, 8, 1), (256, 0, 2)])
def test_every_width(narrow, shape, prec):
    ns = [len(w["steps"]) for w in narrow]
    for K in ([1] * len(ns), [n // 2 for n in ns], [n - 1 for n in ns]):
        _run(narrow, K, prec, 2, 3, shape)


@pytest.mark.parametrize("prec", [128, 64])
def test_more_items_than_warps(narrow, prec):
    """296 blocks of 8 warps are dealt their first items; the rest are taken from the queue."""
    ws = [w for w in narrow if w["width"] <= 9]
    _run(ws, [len(w["steps"]) // 2 for w in ws], prec, 2400 // len(ws) + 30, 1)


@pytest.mark.parametrize("prec", [128, 64])
def test_beside_a_wide_instance(narrow, prec):
    import workloads
    ws = narrow + [workloads.matching_instance(38, 38, 11, 8, 2000)]
    _run(ws, [len(w["steps"]) // 2 for w in ws], prec, 3, 2)


@pytest.mark.parametrize("prec", [128, 64])
def test_impossible_strings(narrow, prec):
    """A prefix, or a suffix, that takes the bit whose matrix row is zero is -inf; the strings beside it are not."""
    import gsb
    for w in narrow:
        ns = len(w["steps"])
        for k in (0, ns // 3, ns // 2, ns - 1):
            K = ns // 2
            b = gsb.Batch([without_bit_one(w["plan"], k)] * 2, precision=prec)
            pre, suf = np.zeros((2, K), np.int8), np.zeros((2, 2, ns - K), np.int8)
            if k < K:
                pre[1, k] = 1
            else:
                suf[:, 1, k - K] = 1
            b.set_strings([K, K], [pre, pre], [suf, suf])
            lp, _ = b.run()
            b.close()
            dead = np.zeros((2, 2), bool)
            dead[(1, slice(None)) if k < K else (slice(None), 1)] = True
            assert (np.isneginf(lp) == dead).all(), (ns, k, lp)


@pytest.mark.parametrize("prec", [128, 64])
def test_prefix_lengths_in_any_order(narrow, prec):
    """One batch, prefix lengths drawn anew for every instance: the passes that earlier lengths left behind and new ones."""
    import gsb
    import workloads
    ws = narrow + [workloads.matching_instance(n, n, 11, 8, 2000) for n in (33, 37)]
    ns = [len(w["steps"]) for w in ws]
    rng = np.random.default_rng(6)
    b = gsb.Batch([w["plan"] for w in ws], precision=prec)
    strings = [rng.integers(0, 2, (4, n), dtype=np.int8) for n in ns]
    ref = []
    for w, x in zip(ws, strings):
        with gsb.Engine.from_text(w["plan"], precision=128) as eng:
            ref.append(eng.chain(x)[0])
    for turn in range(12):
        K = [int(rng.integers(1, n)) for n in ns] if turn else [1] * len(ns)
        b.set_strings(K, [x[:, :k] for x, k in zip(strings, K)], [x[:, None, k:] for x, k in zip(strings, K)])
        lp, _ = b.run()
        for i, n in enumerate(ns):
            tol = 1e-9 if prec == 128 else 6 * gsb.c64_sigma(ref[i], n)
            assert (np.abs(lp[i][:, 0] - ref[i]) <= tol).all(), (turn, n, K[i])
    b.close()
