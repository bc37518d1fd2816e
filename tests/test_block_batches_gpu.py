"""Factorisations of batches that fill the device: cluster sizes are then chosen by the batch, down to one CTA a block."""
import numpy as np
import pytest

from qcmaquis_b200 import dmrg, heff

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps
# (rows, cols) of the blocks: as many as SMs and one more; mid-size ones with a few large ones among them; large ones
BATCHES = {"equal": [(118, 118)] * 148 + [(119, 120)], "mixed": [(90 + k % 60, 150 - k % 50) for k in range(110)] + [(300, 310), (440, 431)],
           "large": [(255 + k, 262 - k) for k in range(7)] * 4}


@pytest.mark.parametrize("name", list(BATCHES))
def test_batches_that_fill_the_device(name):
    ctx = heff.Context(0)
    rng = np.random.default_rng(9)
    svd = []
    for m, n in BATCHES[name]:
        k = min(m, n)
        a = rng.standard_normal((m, k)) * np.exp(-12.0 * np.arange(k) / k)
        svd.append(a @ rng.standard_normal((k, n)) / k)
    got, _ = dmrg.truncate_svd(ctx, svd, 10 ** 6, 1e-30)
    for a, (u, s, vt) in zip(svd, got):
        k = s.size
        ref = np.linalg.svd(a, compute_uv=False)
        # rounding of about 12 k transformations of a column, adding up as a random walk: far below 100 sqrt(k) eps;
        # columns orthogonal to the rotation threshold k eps, twice that with the QR, times a safety of 5
        assert k == min(a.shape) and np.abs(s - ref).max() <= 100 * np.sqrt(k) * EPS * ref[0]
        assert np.abs((u * s) @ vt - a).max() <= 100 * np.sqrt(k) * EPS * ref[0]
        for q in (u, vt.T):
            assert np.abs(q.T @ q - np.eye(k)).max() <= (10 * k + 100) * EPS
    qr = [rng.standard_normal(s) for s in BATCHES[name]]
    for lq in (False, True):
        for a, (x, y) in zip(qr, dmrg.qr_blocks(ctx, qr, lq=lq)):
            q, r = (y.T, x.T) if lq else (x, y)
            b = a.T if lq else a
            tol = 20 * np.sqrt(a.shape[0] * a.shape[1]) * EPS  # k reflectors of unit-norm rounding on columns of norm sqrt(rows)
            assert np.abs(q @ r - b).max() <= 4 * tol * np.abs(b).max()
            assert np.abs(q.T @ q - np.eye(min(a.shape))).max() <= tol
