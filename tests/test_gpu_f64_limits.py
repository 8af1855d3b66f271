"""Plain-method sums at the limits of their number formats: long sums of one
repeated term, inputs off the simplex, frequencies below the digits' range, and
entries made of small products only.  Values are compared entry by entry.

Tolerance 1e-13: a term carries some (2 K + 8) roundings of 2^-53 on both sides,
and sums of positive terms cannot amplify them; the oracle's own additions (at most
a few hundred terms here, or a closed form) add less than 1e-14."""
import numpy as np
import pytest

from conftest import small_cohort

pytestmark = pytest.mark.gpu


def entry_err(a, b):
    a, b = np.asarray(a), np.asarray(b)
    return (np.abs(a - b) / np.maximum(np.abs(b), 1e-300)).max()


def handle(hx, c):
    return hx.GB300Admix(c["bed"], c["I"], c["J"], c["K"], bytes_per_snp=c["bed"].shape[1], n_snp=c["bed"].shape[0])


def test_one_term_repeated_over_the_longest_chunk(hx):
    """65,536 individuals of one Q, all homozygous for one haplotype, in a cohort
    whose P pass takes them in one chunk: every digit of every order repeats, so
    the integer sums grow as fast as they can."""
    import torch
    I, J, K = 65536, 4736, 2
    qv, pv = np.array([0.102, 0.898]), np.array([0.023, 0.207])
    bed = torch.zeros((2 * J, I // 4), dtype=torch.uint8, device="cuda")     # haplotype 0, twice, everywhere
    q = np.asfortranarray(np.repeat(qv[:, None], I, axis=1))
    p = np.empty((K, J, 4))
    p[:, :, 0] = pv[:, None]
    p[:, :, 1:] = ((1.0 - pv) / 3.0)[:, None, None]
    d = hx.GB300Admix(bed.data_ptr(), I, J, K, bytes_per_snp=I // 4, n_snp=2 * J, bed_on_device=True)
    X, z = d.update_p_accum(q, np.asfortranarray(p.reshape(K, 4 * J)))
    d.close()
    qp = float(qv @ pv)
    assert entry_err(X[:, :, 0::4], (2.0 * I / qp / qp * np.outer(qv, qv))[:, :, None]) < 1e-13
    assert entry_err(z[:, 0::4], (2.0 * I / qp * qv)[:, None]) < 1e-13
    assert not X.reshape(K, K, J, 4)[..., 1:].any() and not z.reshape(K, J, 4)[..., 1:].any()


def accums(d, q, p):
    return d.update_q_accum(q, p) + d.update_p_accum(q, p) + d.em_accum(q, p)


def oracle_accums(O, c, q, p):
    b = O.Bed(c["bed"], c["I"], c["J"])
    return O.accum_q(b, c["K"], q, p) + O.accum_p(b, c["K"], q, p) + O.em_accum(b, c["K"], q, p)


def draws(c, seed, lo=1e-3):
    rng = np.random.default_rng(seed)
    q = np.maximum(rng.dirichlet(np.ones(c["K"]), size=c["I"]).T, lo)
    p = np.maximum(rng.dirichlet(np.ones(4), size=(c["K"], c["J"])).reshape(c["K"], -1), lo)
    return np.asfortranarray(q), np.asfortranarray(p)


@pytest.mark.parametrize("sq,sp", [(1e3, 1.0), (1e6, 1.0), (1e9, 1.0), (1.0, 1e4), (1e-6, 1.0), (1e-3, 1e-3)])
def test_inputs_off_the_simplex(hx, O, sq, sp):
    c = small_cohort(150, 70, 3, seed=31, miss=0.05)
    q, p = draws(c, 8)
    d = handle(hx, c)
    for g, w in zip(accums(d, sq * q, sp * p), oracle_accums(O, c, sq * q, sp * p)):
        assert entry_err(g, w) < 1e-13
    d.close()


def test_scales_that_differ_between_rows(hx, O):
    c = small_cohort(150, 70, 4, seed=32, miss=0.05)
    q, p = draws(c, 9)
    q = np.asfortranarray(q * 10.0 ** np.random.default_rng(1).integers(-9, 9, size=(1, c["I"])))
    d = handle(hx, c)
    for g, w in zip(accums(d, q, p), oracle_accums(O, c, q, p)):
        assert entry_err(g, w) < 1e-13
    d.close()


@pytest.mark.parametrize("floor", [1e-6, 1e-8, 1e-13])
def test_small_pseudocounts(hx, O, floor):
    """Individuals near the vertices and haplotypes private to one ancestry, down to
    the floor in all others; and the same bits from a second run."""
    c = small_cohort(120, 60, 4, seed=33, miss=0.05)
    q, p = vertices(c, floor)
    d = handle(hx, c)
    got = accums(d, q, p)
    for g, w in zip(got, oracle_accums(O, c, q, p)):
        assert entry_err(g, w) < 1e-13
    for g, w in zip(got, accums(d, q, p)):
        assert np.array_equal(g, w)
    d.close()


def vertices(c, floor):
    K, I, J = c["K"], c["I"], c["J"]
    rng = np.random.default_rng(17)
    q = np.full((K, I), floor)
    q[rng.integers(0, K, size=I), np.arange(I)] = 1.0 - (K - 1) * floor
    p = rng.dirichlet(np.ones(4), size=(K, J))
    p[1:, ::3, 1] = floor
    p[:2, ::4, 2] = floor
    p[2:, ::5, 3] = floor
    return np.asfortranarray(q), np.asfortranarray(np.maximum(p, floor).reshape(K, 4 * J))


@pytest.mark.parametrize("K,I,J", [(3, 30, 40), (5, 250, 40), (8, 60, 30), (9, 90, 30), (11, 80, 24), (12, 129, 33)])
def test_entries_of_small_products_only(hx, O, K, I, J):
    """Floored rows at the fit's own pseudocount: where all carriers of a haplotype
    are of one ancestry, an entry of two others sums products of two floors, 1e-10 of
    the row's largest."""
    c = small_cohort(I, J, K, seed=K + I, miss=0.03)
    q, p = vertices(c, 1e-5)
    d = handle(hx, c)
    for g, w in zip(accums(d, q, p), oracle_accums(O, c, q, p)):
        assert entry_err(g, w) < 1e-13
    d.close()


def test_zero_frequencies_leave_the_gradient(hx, O):
    """A haplotype of frequency zero that no genotype of its block allows: its terms
    are 0 in the gradient (and 0 / 0 in the Hessian only)."""
    c = small_cohort(90, 30, 3, seed=36, miss=0.0)
    c["bed"][:2 * 4] = 0                      # blocks 0 .. 3: haplotype 0 only
    q, p = draws(c, 12)
    p = p.reshape(3, 30, 4).copy()
    p[:, :4, 3] = 0.0
    p = np.asfortranarray(p.reshape(3, 120))
    d = handle(hx, c)
    zq = d.update_q_accum(q, p)[1]
    zp = d.update_p_accum(q, p)[1]
    d.close()
    b = O.Bed(c["bed"], 90, 30)
    p[p == 0.0] = 1e-300                      # 0 / p instead of 0 / 0
    assert entry_err(zq, O.accum_q(b, 3, q, p)[1]) < 1e-13
    assert entry_err(zp, O.accum_p(b, 3, q, p)[1]) < 1e-13


@pytest.mark.parametrize("side", ["q", "p", "em"])
def test_wait_budget(hx, O, side):
    """The plain passes' pipeline waits are bounded by hx_set_wait_budget: with one
    cycle the call returns HX_ETIMEOUT, and the handle works again afterwards."""
    from haplo_gb300 import _lib
    c = small_cohort(300, 900, 4, seed=37, miss=0.03)
    q, p = draws(c, 13)
    b = O.Bed(c["bed"], c["I"], c["J"])
    d = handle(hx, c)
    call = {"q": d.update_q_accum, "p": d.update_p_accum, "em": d.em_accum}[side]
    want = {"q": O.accum_q, "p": O.accum_p, "em": O.em_accum}[side](b, c["K"], q, p)
    for _ in range(2):
        d.set_wait_budget(1)
        with pytest.raises(hx.HxError) as e:
            call(q, p)
        assert e.value.status == _lib.HX_ETIMEOUT
        d.set_wait_budget(0)
        for g, w in zip(call(q, p), want):
            assert entry_err(g, w) < 1e-13
    d.close()
