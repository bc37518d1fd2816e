"""Block factorisations on a device (or partition) that cannot schedule the clusters they would best run in."""
import numpy as np
import pytest

from qcmaquis_b200 import _lib, dmrg, heff

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


@pytest.mark.parametrize("ctas", [1, 2, 8])
def test_factorisations_in_smaller_clusters(ctas):
    """The same blocks with at most `ctas` CTAs each: with one, Q is logged above 118 columns and G leaves shared memory
    above 167; with two and eight, later.  Bounds as for the clusters of the full device."""
    ctx = heff.Context(0)
    ctx.limit_clusters(ctas)
    svd, qr = [], []
    for k, (m, n) in enumerate([(60, 60), (119, 121), (166, 170), (300, 290), (431, 437), (690, 700)]):
        rng = np.random.default_rng([k, 5])
        r = min(m, n)
        u, _ = np.linalg.qr(rng.standard_normal((m, r)))
        v, _ = np.linalg.qr(rng.standard_normal((n, r)))
        svd.append((u * np.exp(-16.0 * (np.arange(r) + rng.uniform(0, 0.5, r)) / r)) @ v.T)
        qr.append(rng.standard_normal((m, n)))
    got, _ = dmrg.truncate_svd(ctx, svd, 10 ** 6, 1e-30)
    for a, (u, s, vt) in zip(svd, got):
        ref = np.linalg.svd(a, compute_uv=False)
        k = ref.size
        assert s.size == k
        # rounding of about 12 k transformations of a column, adding up as a random walk: far below 100 sqrt(k) eps;
        # columns orthogonal to the rotation threshold k eps, twice that with the QR, times a safety of 5
        assert np.abs(s - ref).max() <= 100 * np.sqrt(k) * EPS * ref[0]
        assert np.abs((u * s) @ vt - a).max() <= 100 * np.sqrt(k) * EPS * ref[0]
        for q in (u, vt.T):
            assert np.abs(q.T @ q - np.eye(k)).max() <= (10 * k + 100) * EPS
    qr += [np.random.default_rng(6).standard_normal(s) for s in ((30, 900), (900, 30))]
    for lq in (False, True):
        for a, (x, y) in zip(qr, dmrg.qr_blocks(ctx, qr, lq=lq)):
            q, r = (y.T, x.T) if lq else (x, y)
            b = a.T if lq else a
            k = min(a.shape)
            tol = 20 * np.sqrt(max(a.shape) * k) * EPS  # k reflectors of unit-norm rounding on columns of norm sqrt(rows)
            assert np.abs(q @ r - b).max() <= 4 * tol * np.abs(b).max()
            assert np.abs(q.T @ q - np.eye(k)).max() <= tol


def test_limits_that_are_no_cluster_size_are_refused():
    ctx = heff.Context(0)
    for ctas in (0, 3, 32):
        with pytest.raises(_lib.QcmError):
            ctx.limit_clusters(ctas)
