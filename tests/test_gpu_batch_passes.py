"""The batch kernel's fused passes and teams: prefixes cut at every parity, instances wide enough for a cluster beside
narrow ones, steps of generic shape (m = 1), every block size; against the executor's complex128 'chain'."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(ws, K, prec, npre, nsuf, shape=None, seed=3):
    import gsb
    rng = np.random.default_rng(seed)
    pre = [rng.integers(0, 2, (npre, k), dtype=np.int8) for k in K]
    suf = [rng.integers(0, 2, (npre, nsuf, len(w["steps"]) - k), dtype=np.int8) for w, k in zip(ws, K)]
    b = gsb.Batch([w["plan"] for w in ws], precision=prec)
    if shape:
        b.set_shape(*shape)
    b.set_strings(K, pre, suf)
    lp, _ = b.run()
    again, _ = b.run()
    assert np.array_equal(lp, again)
    b.close()
    for i, w in enumerate(ws):
        ns = len(w["steps"])
        strings = np.concatenate([np.repeat(pre[i][:, None], nsuf, 1), suf[i]], 2).reshape(-1, ns)
        with gsb.Engine.from_text(w["plan"], precision=128) as eng:
            ref = eng.chain(strings)[0].reshape(npre, nsuf)
        tol = 1e-9 if prec == 128 else 6 * gsb.c64_sigma(ref, ns)
        assert (np.abs(lp[i] - ref) <= tol).all(), (i, ns)


@pytest.mark.parametrize("prec", [128, 64])
@pytest.mark.parametrize("shape", [None, (64, 8, 4), (128, 12, 1), (256, 0, 2), (512, 14, 1)])
def test_widths_and_prefix_lengths(prec, shape):
    """n = 4 .. 36: the widest instances go to clusters (their items exceed an even share of this small batch)."""
    import workloads
    ws = [workloads.qubit_order_instance(n, n, 50 + n) for n in (4, 9, 16, 21, 26, 31, 36)]
    ns = [len(w["steps"]) for w in ws]
    for K in ([1] * 7, [n - 1 for n in ns], [n // 2 for n in ns], [n // 2 + 1 for n in ns]):
        _run(ws, K, prec, 2, 2, shape)


@pytest.mark.parametrize("prec", [128, 64])
def test_generic_shapes(prec):
    """A twin-vertex graph state has steps with one output class (m = 1) on wide tables."""
    import workloads
    w = workloads.twin_graph_instance(h=24, ntw=10, seed=4)
    assert any(s["m"] == 1 for s in w["steps"]) if "m" in w["steps"][0] else True
    ns = len(w["steps"])
    for K in (ns // 3, ns // 2, ns - 3):
        _run([w], [K], prec, 3, 2)


def test_new_prefix_lengths_replace_the_passes():
    """set_strings with other prefix lengths on the same batch, with the totals of bits unchanged."""
    import gsb
    import workloads
    ws = [workloads.qubit_order_instance(n, n, 7) for n in (18, 18)]
    rng = np.random.default_rng(1)
    bits = [rng.integers(0, 2, (4, 18), dtype=np.int8) for _ in ws]
    b = gsb.Batch([w["plan"] for w in ws], precision=128)
    got = []
    for K in ([5, 9], [9, 5], [5, 9]):
        b.set_strings(K, [x[:, :k] for x, k in zip(bits, K)], [x[:, None, k:] for x, k in zip(bits, K)])
        got.append(b.run()[0])
    assert np.abs(got[0] - got[1]).max() <= 1e-9 and np.array_equal(got[0], got[2])
