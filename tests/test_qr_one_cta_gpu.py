"""QR and LQ of blocks that one CTA factorises: around a warp's and the CTA's rows and columns, flat and tall ones up to
the largest, and blocks with nothing to factorise."""
import numpy as np
import pytest

from qcmaquis_b200 import dmrg, heff

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps
SHAPES = [(1, 1), (2, 1), (1, 300), (300, 1), (31, 33), (32, 32), (33, 31), (64, 65), (112, 111), (112, 112), (5, 2000), (2000, 5),
          (12, 1045), (1045, 12), (1, 12544), (12544, 1)]


@pytest.mark.parametrize("lq", [False, True])
def test_one_cta_blocks(lq):
    ctx = heff.Context(0)
    blocks = [np.random.default_rng([m, n]).standard_normal((m, n)) for m, n in SHAPES]
    rank1 = np.outer(np.arange(1.0, 41.0), np.arange(1.0, 31.0))
    for a, (x, y) in zip(blocks + [rank1, rank1.T], dmrg.qr_blocks(ctx, blocks + [rank1, rank1.T], lq=lq)):
        q, r = (y.T, x.T) if lq else (x, y)  # A = L Q is A^T = Q^T L^T
        b = a.T if lq else a
        k = min(a.shape)
        tol = 20 * np.sqrt(max(a.shape) * k) * EPS  # k reflectors of unit-norm rounding on columns of norm sqrt(rows)
        assert np.abs(q @ r - b).max() <= 4 * tol * np.abs(b).max()
        assert np.abs(q.T @ q - np.eye(k)).max() <= tol
        assert np.array_equal(np.tril(r, -1), np.zeros_like(r))
        if a.shape in ((40, 30), (30, 40)):
            assert not np.diag(r)[1:].any()  # the rest of a negligible column is exactly zero


def test_blocks_with_nothing_to_factorise():
    ctx = heff.Context(0)
    bad = np.ones((20, 30))
    bad[3, 4] = np.nan
    got = dmrg.qr_blocks(ctx, [np.zeros((40, 30)), bad, np.eye(25)])
    assert np.array_equal(got[0][0], np.eye(40)[:, :30]) and not got[0][1].any()
    assert np.isnan(got[1][1]).any()
    assert np.array_equal(got[2][0], np.eye(25)) and np.array_equal(got[2][1], np.eye(25))
