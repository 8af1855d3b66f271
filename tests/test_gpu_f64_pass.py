"""Plain-method passes (exact digit sums on the tensor cores) against the CPU
oracle, where their tiles, windows and ranges can go wrong.

Tolerances: every term carries a few roundings of 2^-53 (qp, reciprocal,
weight) on both sides, and sums of positive terms cannot amplify them: 1e-13
per entry leaves a factor of 100 at the sizes here (the oracle's own FP64
accumulation over at most 2,000 terms is the larger part).  Weights beyond the digits' range
(qp below 1e-4) go another way and are held to the same bound.
"""
import numpy as np
import pytest

from conftest import small_cohort

pytestmark = pytest.mark.gpu


def entry_err(a, b):
    a, b = np.asarray(a), np.asarray(b)
    return (np.abs(a - b) / np.maximum(np.abs(b), 1e-300)).max()


def compare(hx, O, c, q, p, tol=1e-13):
    b = O.Bed(c["bed"], c["I"], c["J"])
    d = hx.GB300Admix(c["bed"], c["I"], c["J"], c["K"], bytes_per_snp=c["bed"].shape[1], n_snp=c["bed"].shape[0])
    for got, want in ((d.update_q_accum(q, p), O.accum_q(b, c["K"], q, p)),
                      (d.update_p_accum(q, p), O.accum_p(b, c["K"], q, p)),
                      (d.em_accum(q, p), O.em_accum(b, c["K"], q, p))):
        for g, w in zip(got, want):
            assert entry_err(g, w) < tol
    d.close()


@pytest.mark.parametrize("I,J,K", [(1, 1, 2), (127, 8, 1), (128, 33, 3), (129, 257, 5), (31, 1500, 6), (1501, 31, 8),
                                   (257, 129, 9), (200, 40, 10), (161, 65, 11), (97, 260, 12)])
def test_tiles_windows_and_column_groups(hx, O, I, J, K):
    c = small_cohort(I, J, K, seed=I + J + K, miss=0.08)
    rng = np.random.default_rng(I)
    q = np.asfortranarray(rng.dirichlet(np.ones(K), size=I).T)
    p = np.asfortranarray(rng.dirichlet(np.ones(4), size=(K, J)).reshape(K, 4 * J))
    compare(hx, O, c, np.maximum(q, 1e-5), np.maximum(p, 1e-5))


@pytest.mark.parametrize("floor", [1e-5, 1e-8, 1e-40])
def test_weights_beyond_the_digits(hx, O, floor):
    """Observed haplotypes at frequency `floor`: W = 1e10, 1e16, 1e80."""
    K, I, J = 4, 150, 70
    c = small_cohort(I, J, K, seed=11, miss=0.05)
    rng = np.random.default_rng(5)
    q = np.asfortranarray(rng.dirichlet(np.ones(K), size=I).T)
    p = rng.dirichlet(np.ones(4), size=(K, J)).reshape(K, J, 4)
    p[:, ::7, 1] = floor
    p[:, ::5, 2] = floor
    compare(hx, O, c, q, np.asfortranarray(p.reshape(K, 4 * J)))


def test_rare_ancestry_keeps_its_relative_precision(hx, O):
    K, I, J = 5, 260, 90
    c = small_cohort(I, J, K, seed=23, miss=0.02)
    rng = np.random.default_rng(6)
    q = rng.dirichlet(np.ones(K), size=I).T
    q[2] = 1e-5
    p = rng.dirichlet(np.ones(4), size=(K, J)).reshape(K, 4 * J)
    compare(hx, O, c, np.asfortranarray(q), np.asfortranarray(p))


def test_non_finite_and_zero_frequencies_reach_the_hessian(hx, O):
    K, I, J = 3, 140, 20
    c = small_cohort(I, J, K, seed=29, miss=0.0)
    rng = np.random.default_rng(7)
    q = np.asfortranarray(rng.dirichlet(np.ones(K), size=I).T)
    p = np.asfortranarray(rng.dirichlet(np.ones(4), size=(K, J)).reshape(K, 4 * J))
    d = hx.GB300Admix(c["bed"], I, J, K, bytes_per_snp=c["bed"].shape[1], n_snp=c["bed"].shape[0])
    for bad in (0.0, np.nan):
        x = p.copy(order="F")
        x[:, 13] = bad
        assert np.isnan(d.update_q_accum(q, x)[0]).all()
        assert np.isnan(d.update_p_accum(q, x)[0][:, :, 13]).all()
        d.set_qp(q, x)
        with pytest.raises(hx.HxError):
            d.update_q()
    # and nothing of it stays behind
    ok = d.update_q_accum(q, p)
    b = O.Bed(c["bed"], I, J)
    assert entry_err(ok[0], O.accum_q(b, K, q, p)[0]) < 1e-13
    d.close()


@pytest.mark.parametrize("I,J,K", [(1, 1, 1), (33, 9, 2), (128, 8, 4), (129, 127, 7), (500, 65, 12)])
def test_loglik_items_and_chunks(hx, O, I, J, K):
    """Log-likelihood from class words and from BED bytes; a zero frequency of
    an observed haplotype gives -inf, a NaN one NaN."""
    import torch
    c = small_cohort(I, J, K, seed=3 * I + J, miss=0.1)
    b = O.Bed(c["bed"], I, J)
    rng = np.random.default_rng(J)
    q = np.asfortranarray(rng.dirichlet(np.ones(K), size=I).T)
    p = np.asfortranarray(rng.dirichlet(np.ones(4), size=(K, J)).reshape(K, 4 * J))
    d = hx.GB300Admix(c["bed"], I, J, K, bytes_per_snp=c["bed"].shape[1], n_snp=c["bed"].shape[0])
    bed = torch.from_numpy(c["bed"]).cuda()
    ll = torch.empty((), dtype=torch.float64, device="cuda")

    def noalloc(p):
        dq, dp = torch.from_numpy(q.T.copy()).cuda(), torch.from_numpy(p.T.copy()).cuda()
        st = hx.load().hx_loglikelihood_noalloc(bed.data_ptr(), c["bed"].shape[1], I, J, K, dq.data_ptr(),
                                                dp.data_ptr(), 0, ll.data_ptr(), None)
        assert st == 0
        torch.cuda.synchronize()
        return float(ll)

    want = O.loglik(b, K, q, p)
    assert d.loglikelihood(q, p) == pytest.approx(want, rel=1e-13)
    assert noalloc(p) == pytest.approx(want, rel=1e-13)
    z = p.copy(order="F")
    z[:, :4] = 0.0
    want = O.loglik(b, K, q, z)
    for got in (d.loglikelihood(q, z), noalloc(z)):
        assert got == want or got == pytest.approx(want, rel=1e-13)
    z[:, :4] = np.nan
    want = O.loglik(b, K, q, z)
    for got in (d.loglikelihood(q, z), noalloc(z)):
        assert np.isnan(got) == np.isnan(want)
    d.close()
