"""QPs of cohorts with fewer blocks or individuals than variables: pivots at their floor,
bounds met one after another.  Such steps take the dense solver for all their problems,
the QP entry points the batched kernels; both perform the same operations on the same
sums, so the results are equal bit for bit (the minimiser itself is not unique)."""
import numpy as np
import pytest

from conftest import small_cohort

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("K,I,J", [(4, 5, 300), (8, 3, 40), (12, 23, 33), (5, 9, 65), (8, 300, 2), (12, 2999, 13),
                                   (5, 2500, 3), (6, 65, 1)])
def test_dense_and_batched_solvers_agree(hx, O, K, I, J, precision):
    c = small_cohort(I, J, K, seed=I + J, miss=0.02)
    rng = np.random.default_rng(I)
    q = rng.dirichlet(np.ones(K), size=I).T
    p = rng.dirichlet(np.ones(4), size=(K, J)).reshape(K, 4 * J)
    d = hx.GB300Admix(c["bed"], I, J, K, bytes_per_snp=c["bed"].shape[1], n_snp=c["bed"].shape[0], precision=precision)
    q, p = d.project_q(q), d.project_p(p)
    d.set_qp(q, p)
    d.update_q()
    qn = d.get_qp("x_next")[0]
    X, z = d.update_q_accum(q, p)
    assert np.array_equal(qn, d.project_q(q + d.qp_q(X, z, q)), equal_nan=True)
    d.update_p()
    X, z = d.update_p_accum(qn, p)
    assert np.array_equal(d.get_qp("x_next")[1], d.project_p(p + d.qp_p(X, z, p)), equal_nan=True)
    d.close()
