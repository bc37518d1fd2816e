"""Factorisations of blocks at the edges of their kernels' work split: one CTA per block or a cluster of 2 to 16,
work arrays in shared memory or in global scratch, ragged shares of rows and columns."""
import numpy as np
import pytest

from qcmaquis_b200 import dmrg, heff

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps

# (rows, cols): around 48 and 88 columns (one CTA), 36 rows per CTA (2, 4, 8, 16 CTAs), the limits at 16 CTAs above which
# Q comes from the rotation log (about 420 columns) and G leaves shared memory (about 660), and beyond them
SVD_SHAPES = [(1, 1), (2, 1), (3, 3), (47, 48), (48, 49), (49, 49), (72, 73), (73, 75), (87, 88), (90, 89), (144, 145), (145, 149),
              (289, 291), (431, 437), (701, 699)]
# around the elements per block at which the QR splits (112, 128, 256, 512 squared), flat and tall blocks
QR_SHAPES = [(1, 1), (1, 7), (7, 1), (63, 65), (65, 65), (112, 112), (113, 112), (129, 127), (131, 131), (257, 256), (261, 263), (519, 517),
             (30, 900), (900, 30), (700, 701)]


def _decaying(m, n, seed):
    """Blocks with singular values down to 1e-7 of the largest (as the truncated two-site tensors have)."""
    rng = np.random.default_rng([seed, m, n])
    k = min(m, n)
    u, _ = np.linalg.qr(rng.standard_normal((m, k)))
    v, _ = np.linalg.qr(rng.standard_normal((n, k)))
    return (u * np.exp(-16.0 * (np.arange(k) + rng.uniform(0, 0.5, k)) / k)) @ v.T


@pytest.mark.parametrize("together", [False, True])
def test_svd_at_cluster_edges(together):
    ctx = heff.Context(0)
    blocks = [_decaying(m, n, 1) for m, n in SVD_SHAPES]
    batches = [blocks] if together else [[b] for b in blocks]
    for batch in batches:
        got, _ = dmrg.truncate_svd(ctx, batch, 10 ** 6, 1e-30)
        for a, (u, s, vt) in zip(batch, got):
            ref = np.linalg.svd(a, compute_uv=False)
            k = ref.size
            # backward error of the QR and the rotations: rounding of each of about 12 k transformations of a
            # column, adding up as a random walk, far below 100 sqrt(k) eps; columns are orthogonal to the
            # rotation threshold k eps, twice that with the QR's own rounding, times a safety of 5
            assert s.size == k
            assert np.abs(s - ref).max() <= 100 * np.sqrt(k) * EPS * ref[0]
            assert np.abs((u * s) @ vt - a).max() <= 100 * np.sqrt(k) * EPS * ref[0]
            for q in (u, vt.T):
                assert np.abs(q.T @ q - np.eye(k)).max() <= (10 * k + 100) * EPS


@pytest.mark.parametrize("lq", [False, True])
def test_qr_at_cluster_edges(lq):
    ctx = heff.Context(0)
    blocks = [np.random.default_rng([2, m, n]).standard_normal((m, n)) for m, n in QR_SHAPES]
    for a, (x, y) in zip(blocks, dmrg.qr_blocks(ctx, blocks, lq=lq)):
        q, r = (y.T, x.T) if lq else (x, y)  # A = L Q is A^T = Q^T L^T
        b = a.T if lq else a
        k = min(a.shape)
        tol = 20 * np.sqrt(max(a.shape)) * k ** 0.5 * EPS  # k reflectors of unit-norm rounding on columns of norm sqrt(rows)
        assert np.abs(q @ r - b).max() <= tol * np.abs(b).max() * 4
        assert np.abs(q.T @ q - np.eye(k)).max() <= tol
        assert np.array_equal(np.tril(r, -1), np.zeros_like(r))


def test_qr_of_nan_and_zero_blocks_ends():
    """Blocks without a comparable pivot (NaN) or with nothing to factorise (zero) come back without an error."""
    ctx = heff.Context(0)
    rng = np.random.default_rng(3)
    bad = rng.standard_normal((130, 131))
    bad[5, 7] = np.nan
    good = rng.standard_normal((130, 131))
    got = dmrg.qr_blocks(ctx, [bad, np.zeros((70, 80)), good])
    assert np.isnan(got[0][0]).any()
    assert np.array_equal(got[1][1], np.zeros((70, 80)))
    assert np.abs(got[2][0] @ got[2][1] - good).max() <= 1e-12
