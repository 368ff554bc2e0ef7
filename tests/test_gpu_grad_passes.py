"""The adjoint sweep's passes of two steps: tables kept before every pass, every second one, or one for the whole sweep,
at widths from one entry per class to several classes per thread.

Z is linear in every step's M row, so sum_x M_k[b_k][x] dZ/dM_k[b_k][x] = Z for every string and step; Z itself is the
executor's.  A derivative with respect to one entry is the difference of two sweeps (linearity again, no step size)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count,every", [(5, 3, 4), (17, 33, 4), (33, 5, 4), (33, 2, 8), (33, 1, 64), (41, 3, 4), (41, 2, 13)])
def test_derivatives_against_linearity(n, count, every):
    import adjoint
    import gsb
    import torch
    import workloads
    w = workloads.rotation_instance(n, n, seed=9, order_seed=12, iters=4000)
    ns = len(w["steps"])
    bits = workloads.random_strings(ns, count, seed=n)
    M = adjoint.step_matrices(torch.tensor(w["theta0"]), w["M0"], w["step_vertices"]).numpy()
    sweep = gsb.GradSweep(w["plan"], every=every)
    z, dz = sweep.run(M, bits)
    with gsb.Engine.from_text(w["plan"], precision=128) as eng:
        eng.set_matrices(M)
        assert np.abs(np.log2(np.abs(z) ** 2) - n - eng.prob(bits)).max() <= 1e-9
    rows = M[np.arange(ns)[None, :], bits]                      # [count, ns, 2]
    # each of the ns steps rounds sums of up to 4 terms: far below 1e-10 of the sums' size |row| |dZ| + |Z|
    size = np.linalg.norm(rows, axis=2) * np.linalg.norm(dz, axis=2) + np.abs(z)[:, None]
    assert (np.abs((rows * dz).sum(2) - z[:, None]) <= 1e-10 * size).all()
    rng = np.random.default_rng(n)
    for k in rng.integers(0, ns, 4):
        x = int(rng.integers(2))
        M2 = M.copy()
        M2[k, :, x] += 1.0
        z2, _ = sweep.run(M2, bits)
        assert (np.abs(z2 - z - dz[:, k, x]) <= 1e-10 * (np.abs(z2) + np.abs(z) + np.abs(dz[:, k, x]))).all()
