"""Mixed EM gradient (Q side) and the no-allocation mixed log-likelihood at the
edges of their tiles: individuals around 128 per CTA, blocks around 64 (Q stage)
and 16 (no-allocation stage), every storage form of K.  Bounds: a term of the
gradient carries K + 8 FP32 roundings of 2^-24 (qp, factors, reciprocal), a stage
adds 256 positive terms one by one, and the normalisation to a row sum doubles the
relative error: 2 (K + 264) 2^-24 of values up to 1.  The log-likelihood: K + 8
roundings per pair."""
import numpy as np
import pytest
import torch

from conftest import small_cohort

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("I,J,K", [(1, 1, 1), (127, 8, 3), (128, 64, 8), (129, 65, 5), (300, 517, 9), (130, 130, 12)])
def test_em_q_and_noalloc(hx, O, I, J, K):
    c = small_cohort(I, J, K, seed=3 * I + J, miss=0.05)
    b = O.Bed(c["bed"], I, J)
    rng = np.random.default_rng(I + K)
    q = np.asfortranarray(rng.dirichlet(np.ones(K), size=I).T)
    p = np.asfortranarray(np.maximum(rng.dirichlet(np.ones(4), size=(K, J)), 1e-5).reshape(K, 4 * J))
    step = []
    for prec in ("fp64", "mixed"):
        d = hx.GB300Admix(c["bed"], I, J, K, bytes_per_snp=c["bed"].shape[1], n_snp=c["bed"].shape[0], precision=prec)
        d.set_qp(q, p)
        d.em_step()
        step.append(d.get_qp("x_next")[0])
        d.close()
    assert np.abs(step[1] - step[0]).max() <= 2 * (K + 264) * 2.0 ** -24

    bed = torch.from_numpy(c["bed"]).cuda()
    ll = torch.empty((), dtype=torch.float64, device="cuda")

    def noalloc(p):
        dq, dp = torch.from_numpy(q.T.copy()).cuda(), torch.from_numpy(p.T.copy()).cuda()
        st = hx.load().hx_loglikelihood_noalloc(bed.data_ptr(), c["bed"].shape[1], I, J, K, dq.data_ptr(),
                                                dp.data_ptr(), 1, ll.data_ptr(), None)
        assert st == 0
        torch.cuda.synchronize()
        return float(ll)

    assert abs(noalloc(p) - O.loglik(b, K, q, p)) <= (K + 8) * 2.0 ** -24 * I * J
    z = p.copy(order="F")
    z[:, :4] = 0.0
    want = O.loglik(b, K, q, z)
    assert noalloc(z) == want if np.isinf(want) else abs(noalloc(z) - want) <= (K + 8) * 2.0 ** -24 * I * J
    z[:, :4] = np.nan
    assert np.isnan(noalloc(z)) == np.isnan(O.loglik(b, K, q, z))
