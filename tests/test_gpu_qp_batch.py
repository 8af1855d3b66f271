"""Batched QPs at the edges of their lane layout (K lanes per problem on
the P side, with idle lanes where K does not divide 32; 64 problems per CTA on
the Q side) and on problems whose bounds bind, against the oracle's
solver.  The minimiser is unique, so both find the same point; 1e-9 is the
bound the QP tests of this suite use for K up to 12."""
import numpy as np
import pytest

from conftest import small_cohort

pytestmark = pytest.mark.gpu


def problems(K, n, cols, seed):
    """SPD blocks and gradients that push about half of the variables to a bound."""
    rng = np.random.default_rng(seed)
    X = np.empty((K, K, n * cols), order="F")
    for a in range(n * cols):
        B = rng.normal(size=(K, K + 2))
        X[:, :, a] = 50.0 * (B @ B.T) + np.eye(K)
    z = np.asfortranarray(rng.normal(scale=60.0, size=(K, n * cols)))
    return X, z, rng


@pytest.mark.parametrize("K", [1, 2, 3, 7, 8, 9, 10, 12])
@pytest.mark.parametrize("n", [1, 63, 65])
def test_bounds_bind_and_last_groups(hx, O, K, n):
    c = small_cohort(40, 8, K, seed=K)
    d = hx.GB300Admix(c["bed"], 40, 8, K, bytes_per_snp=c["bed"].shape[1], n_snp=c["bed"].shape[0])
    X, z, rng = problems(K, n, 1, 100 * K + n)
    q = np.asfortranarray(np.maximum(rng.dirichlet(np.full(K, 0.3), size=n).T, 1e-5))
    want, _ = O.qp_q(X, z, q)    # with one variable and one equality the oracle may cycle at d = 0
    assert np.abs(d.qp_q(X, z, q) - want).max() < 1e-9
    X, z, rng = problems(K, n, 4, 100 * K + n + 1)
    p = np.asfortranarray(np.maximum(rng.dirichlet(np.full(4, 0.3), size=(K, n)).reshape(K, 4 * n), 1e-5))
    want, fails = O.qp_p(X, z, p)
    assert fails == 0
    assert np.abs(d.qp_p(X, z, p) - want).max() < 1e-9
    d.close()
