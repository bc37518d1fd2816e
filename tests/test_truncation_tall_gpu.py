"""Truncation results of flat and tall blocks, copied and transposed in parts of 32 columns and 128 rows."""
import numpy as np
import pytest

from qcmaquis_b200 import dmrg, heff

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 128, 129, 300, 2001])
def test_flat_and_tall_blocks(n):
    ctx = heff.Context(0)
    blocks = [np.random.default_rng([n, k]).standard_normal(s) for k, s in enumerate([(5, n), (n, 5), (33, n), (n, 65), (2, 2)])]
    got, _ = dmrg.truncate_svd(ctx, blocks, 10 ** 6, 1e-30)
    for a, (u, s, vt) in zip(blocks, got):
        k = s.size
        # backward error of the QR and the rotations: far below 100 sqrt(k) eps of the largest singular value
        assert u.shape == (a.shape[0], k) and vt.shape == (k, a.shape[1]) and k == min(a.shape)
        assert np.abs((u * s) @ vt - a).max() <= 100 * np.sqrt(k) * EPS * s[0]


@pytest.mark.parametrize("shape", [(1, 1), (40, 7), (7, 40), (50, 50)])
@pytest.mark.parametrize("keep", [1, 5, 50])
def test_one_block_cut(shape, keep):
    """A single block's kept columns, which are read back without a gather."""
    a = np.random.default_rng(8).standard_normal(shape)
    (u, s, vt), = dmrg.truncate_svd(heff.Context(0), [a], keep, 1e-30)[0]
    ru, rs, rvt = np.linalg.svd(a, full_matrices=False)
    k = min(keep + 1, rs.size)  # the cut lies at the value after the last of `keep`, and what is not below it is kept
    assert u.shape == (shape[0], k) and vt.shape == (k, shape[1])
    assert np.abs(s - rs[:k]).max() <= 100 * np.sqrt(rs.size) * EPS * rs[0]  # as above
    # the leading subspace: errors are amplified by the gap to the values cut off, none of which is within 1e-3 here
    assert np.abs((u * s) @ vt - (ru[:, :k] * rs[:k]) @ rvt[:k]).max() <= 1e3 * 100 * np.sqrt(rs.size) * EPS * rs[0]
