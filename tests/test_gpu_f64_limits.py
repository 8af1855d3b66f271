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
