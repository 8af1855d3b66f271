"""Decode at the edges of its 16-individual x 8-block tiles and of the upload's
slices, from host and device memory (rows of any byte length, device pointers
of any alignment): census and double-missing counts, bit-exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def expected(bed, I, J):
    n = bed.shape[0] // 2 * 2
    codes = np.stack([(bed >> (2 * r)) & 3 for r in range(4)], -1).reshape(bed.shape[0], -1)[:n, :I]
    g = np.array([0, 3, 1, 2])[codes]
    census = np.zeros(16, dtype=np.uint64)
    for a in range(4):
        for b in range(4):
            census[4 * a + b] = np.count_nonzero((g[0:2 * J:2] == a) & (g[1:2 * J:2] == b))
    return census, ((codes[0::2] == 1) & (codes[1::2] == 1)).sum(0)


@pytest.mark.parametrize("I,J,extra", [(1, 1, 0), (15, 7, 1), (16, 8, 3), (17, 9, 40), (129, 64, 17), (1003, 40, 5),
                                       (65, 900, 0)])
@pytest.mark.parametrize("shift", [None, 0, 1, 3])
def test_census_and_double_missing(hx, I, J, extra, shift):
    import torch
    rng = np.random.default_rng(I + J)
    bed = rng.integers(0, 256, size=(2 * J + extra, (I + 3) // 4), dtype=np.uint8)
    if shift is None:
        d = hx.GB300Admix(bed, I, J, 3, bytes_per_snp=bed.shape[1], n_snp=bed.shape[0])
    else:   # device memory, the matrix at any byte of its allocation
        t = torch.zeros(bed.size + shift, dtype=torch.uint8, device="cuda")
        t[shift:] = torch.from_numpy(bed.ravel()).cuda()
        torch.cuda.synchronize()
        d = hx.GB300Admix(t.data_ptr() + shift, I, J, 3, bytes_per_snp=bed.shape[1], n_snp=bed.shape[0],
                          bed_on_device=True)
    census, dm = expected(bed, I, J)
    np.testing.assert_array_equal(d.census(), census)
    np.testing.assert_array_equal(d.double_missing(), dm)
    d.close()


def test_upload_in_slices(hx):
    """80 MB of BED: more than one slice of the upload."""
    I, J = 40000, 4000
    bed = np.random.default_rng(5).integers(0, 256, size=(2 * J, I // 4), dtype=np.uint8)
    d = hx.GB300Admix(bed, I, J, 2, bytes_per_snp=I // 4, n_snp=2 * J)
    census, dm = expected(bed, I, J)
    np.testing.assert_array_equal(d.census(), census)
    np.testing.assert_array_equal(d.double_missing(), dm)
    d.close()
