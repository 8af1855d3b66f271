"""Mixed log-likelihood where its chunks and its renormalised products can go wrong:
ragged sizes, small likelihoods (every pair is renormalised, so that products do not
underflow; a pair's own likelihood has to be a normal FP32 number), zeros and NaN.  A
pair's FP32 likelihood carries K + 8 roundings of 2^-24 at most (qp, two
factors, products), which bounds the sum's error by (K + 8) 2^-24 per pair; only
over many pairs do they average out to the mixed method's 1e-8."""
import numpy as np
import pytest

from conftest import small_cohort

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("I,J,K", [(1, 1, 2), (255, 9, 3), (257, 64, 8), (700, 1031, 5), (130, 71, 12)])
@pytest.mark.parametrize("floor", [1e-5, 1e-14, 0.0])
def test_small_and_zero_likelihoods(hx, O, I, J, K, floor):
    c = small_cohort(I, J, K, seed=I + 7 * J, miss=0.05)
    b = O.Bed(c["bed"], I, J)
    rng = np.random.default_rng(K)
    q = np.asfortranarray(rng.dirichlet(np.ones(K), size=I).T)
    p = rng.dirichlet(np.ones(4), size=(K, J))
    p[:, ::3, 2] = floor
    p = np.asfortranarray(p.reshape(K, 4 * J))
    d = hx.GB300Admix(c["bed"], I, J, K, bytes_per_snp=c["bed"].shape[1], n_snp=c["bed"].shape[0], precision="mixed")
    want = O.loglik(b, K, q, p)
    got = d.loglikelihood(q, p)
    assert got == want if np.isinf(want) else abs(got - want) <= (K + 8) * 2.0 ** -24 * I * J
    p[:, 5 % (4 * J)] = np.nan
    assert np.isnan(d.loglikelihood(q, p)) == np.isnan(O.loglik(b, K, q, p))
    d.close()
