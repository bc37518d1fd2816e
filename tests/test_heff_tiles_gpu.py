"""H_eff . psi where sector sizes lie around the edges of the kernels' tiles and copies (fragments of 8 rows, K steps
of 16, tiles of 16, 32 and 64 rows and 64 or 128 columns; 16-byte copies for even sizes only), its adjoint over
the same, and lockstep solves of vectors of unlike lengths."""
import os
import sys

import numpy as np
import pytest

from oracle.oracle import heff_adjoint, heff_apply, site_problem
from qcmaquis_b200 import heff

from helpers import qc_system

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), ".."))
import bench  # noqa: E402

pytestmark = pytest.mark.gpu

L, SITE = 6, 2
PHYS = [(0, 0, 1), (1, 0, 1), (0, 1, 1), (1, 1, 1)]
# rows and K steps of one size class each, even and odd mixed; sector k of a bond takes size k of the list, cyclically
SIZES = {"fragments": [1, 7, 8, 9, 2], "steps": [15, 16, 17, 3, 14], "small tiles": [31, 32, 33, 18, 5],
         "large tiles": [63, 64, 65, 34, 1], "columns": [127, 6, 129, 64, 66], "even": [2, 64, 130, 16, 34]}


def problem(sizes, seed):
    """Site problem (blob and parsed) of the middle bond over bonds whose sectors have the given sizes."""
    up = L // 2
    bonds = []
    for i in range(L + 1):
        q = [(a, b) for a in range(up, -1, -1) for b in range(up, -1, -1)
             if max(a, b) <= i and up - min(a, b) <= L - i]
        bonds.append([(a, b, 1 if i in (0, L) else sizes[(k + i) % len(sizes)]) for k, (a, b) in enumerate(q)])
    sites = bench.synthetic_mps(PHYS, bonds, seed)
    snap = site_problem(qc_system(L)[5], [bench.qmps_blob(s) for s in sites], SITE)
    return snap, heff.parse_site_problem(snap)


@pytest.mark.parametrize("kind", list(SIZES))
def test_apply_at_tile_edges(gpu_ctx, kind):
    ts, blob = qc_system(L)[4:6]
    snap, p = problem(SIZES[kind], 7)
    plan = heff.plan_from_problem(gpu_ctx, p, ts, SITE)
    x = np.random.default_rng(1).standard_normal(plan.n)
    ref, _, _ = heff_apply(snap, blob, SITE, x)
    scale = np.abs(ref).max()
    assert np.abs(plan.apply(x) - ref).max() <= 1e-12 * scale  # the bound of every FP64 apply against the oracle
    for form in ("mixed", "mixed_tc"):
        assert np.abs(plan.apply(x, precision=form) - ref).max() <= 2e-6 * scale  # likewise (3xTF32 products, FP32 sums)


@pytest.mark.parametrize("kind", ["fragments", "steps", "small tiles", "large tiles", "even"])
def test_adjoint_at_tile_edges(gpu_ctx, kind):
    ts = qc_system(L)[4]
    snap, p = problem(SIZES[kind], 7)
    plan = heff.plan_from_problem(gpu_ctx, p, ts, SITE)
    x, ybar = np.random.default_rng(4).standard_normal((2, plan.n))
    pb, g = plan.adjoint(x, ybar)
    pb_ref, g_ref = heff_adjoint(snap, ts.blob(), SITE, x, ybar, g.size)
    # the bounds of every adjoint against the oracle
    assert np.abs(pb - pb_ref).max() <= 1e-12 * np.abs(pb_ref).max()
    assert np.abs(g - g_ref).max() <= 1e-11 * np.abs(g_ref).max()


def test_lockstep_solves_of_unlike_lengths(gpu_ctx):
    """Vectors below, around and far above the 4096 entries that a dot's threads take in one turn."""
    from qcmaquis_b200.dmrg import jd_solve
    ts = qc_system(L)[4]
    plans = [heff.plan_from_problem(gpu_ctx, problem(s, 5)[1], ts, SITE)
             for s in ([1, 2, 1], [6, 7, 5, 8], SIZES["steps"])]
    assert plans[0].n < 1024 < plans[1].n < 8192 < plans[2].n
    xs = [np.random.default_rng(k).standard_normal(q.n) for k, q in enumerate(plans)]
    xs = [x / np.linalg.norm(x) for x in xs]
    g = heff.HeffGroup(gpu_ctx, plans)
    ev, out, it, _ = g.jd_solve(g.pack(xs), 1e-10, 6)
    for k, (q, x) in enumerate(zip(plans, xs)):
        e1, _, it1 = jd_solve(q, x, 1e-10, 6)
        # the lowest value of the same six-dimensional spaces, orthogonalised differently
        assert int(it[k]) == it1 and abs(ev[k] - e1) <= 1e-10 * abs(e1)
