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
