"""Rounding of the truncation SVD's plane rotations: their cosines and sines must not drift from c^2 + s^2 = 1."""
import numpy as np
import pytest
import scipy.linalg

from qcmaquis_b200 import dmrg, heff

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


# one CTA per block, and clusters of 4, 8 and 16
@pytest.mark.parametrize("k", [60, 88, 142, 200, 300])
def test_column_norms_of_accumulated_rotations(k):
    """For the triangular factor of a pivoted QR, the truncation's own QR is the identity and U is the bare product of
    the rotations.  About 10 sweeps rotate a column 10 k times.  Rounding c (next to 1, steps of eps / 2, mostly small
    angles) to the nearest changes its squared norm by 0.3 eps rms each time: sqrt(10 k) eps / 2 in all with 1.6 times
    to spare, if no rotation is biased."""
    ctx = heff.Context(0)
    dev = []
    for seed in range(3):
        rng = np.random.default_rng([seed, k])
        u, _ = np.linalg.qr(rng.standard_normal((k, k)))
        v, _ = np.linalg.qr(rng.standard_normal((k, k)))
        a = (u * np.exp(-16.0 * (np.arange(k) + rng.uniform(0, 0.5, k)) / k)) @ v.T
        r = np.triu(scipy.linalg.qr(a, pivoting=True)[1])
        got, _ = dmrg.truncate_svd(ctx, [r], 10 ** 6, 1e-30)
        dev.append((got[0][0].astype(np.longdouble) ** 2).sum(0) - 1)
    assert float(np.sqrt((np.array(dev) ** 2).mean())) <= 0.5 * np.sqrt(10 * k) * EPS
