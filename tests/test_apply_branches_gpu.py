"""H_eff . psi on inputs that take the rarer branches of a plan: partials of all tile shapes in one region, MPO indices
of a boundary cohort that share a block, blocks of a cohort that no MPO index refers to."""
import numpy as np
import pytest

from oracle.oracle import heff_apply
from qcmaquis_b200 import heff

from helpers import qc_system
from test_heff_tiles_gpu import L, SITE, problem

pytestmark = pytest.mark.gpu
TOL = 1e-12  # the bound of every FP64 apply against the oracle


def test_partials_in_one_region(gpu_ctx):
    """Sizes for which a region per tile shape would pass the allocation-free scratch, and one shared region does not."""
    ts, blob = qc_system(L)[4:6]
    snap, p = problem([33, 11, 4, 66], 7)
    plan = heff.plan_from_problem(gpu_ctx, p, ts, SITE)
    assert plan.info["launches"] == 6  # T, S, and the two L.S kernels once for each of two shapes
    x = np.random.default_rng(1).standard_normal(plan.n)
    ref, _, _ = heff_apply(snap, blob, SITE, x)
    y = plan.apply(x)
    assert np.abs(y - ref).max() <= TOL * np.abs(ref).max()
    torch = pytest.importorskip("torch")
    xd = torch.from_numpy(x).cuda()
    yd = torch.zeros_like(xd)
    torch.cuda.synchronize()
    plan.apply_device_noalloc(xd.data_ptr(), yd.data_ptr())
    gpu_ctx.synchronize()
    assert np.array_equal(yd.cpu().numpy(), y)


def altered(p, side, change):
    """The problem with change(offsets of the cohort, its block size, its data) on its diagonal cohorts of at least two
    blocks (no other cohort reads their data)."""
    b = p[side]
    offsets, data = b["offsets"].reshape(-1, b["aux"]).copy(), b["data"].copy()
    n = 0
    for c in range(len(b["cohort_bra"])):
        at = np.flatnonzero(offsets[c] >= 0)
        if b["tr"][c] or b["cohort_bra"][c] != b["cohort_ket"][c] or at.size < 2:
            continue
        size = int(b["lsz"][c]) * int(b["rsz"][c])
        change(offsets[c], at, size, data[int(b["data_offset"][c]):])
        n += 1
    assert n
    return {**p, side: {**b, "offsets": offsets.ravel(), "data": data}}


@pytest.mark.parametrize("sizes", [[3, 17, 8, 5], [6, 34, 64, 2]])
def test_mpo_indices_sharing_a_block(gpu_ctx, sizes):
    """Two indices of a right boundary cohort on one block, against two blocks of the same values."""
    ts = qc_system(L)[4]
    p = problem(sizes, 3)[1]

    def same(o, at, size, d):
        i, j = o[at[0]], o[at[-1]]
        d[j:j + size] = d[i:i + size]

    def shared(o, at, size, d):
        same(o, at, size, d)
        o[at[-1]] = o[at[0]]

    plans = [heff.plan_from_problem(gpu_ctx, altered(p, "R", f), ts, SITE) for f in (same, shared)]
    x = np.random.default_rng(2).standard_normal(plans[0].n)
    ref, y = (q.apply(x) for q in plans)
    assert np.abs(y - ref).max() <= TOL * np.abs(ref).max()


@pytest.mark.parametrize("sizes", [[3, 17, 8, 5], [6, 34, 64, 2]])
def test_blocks_without_an_mpo_index(gpu_ctx, sizes):
    """A block of left boundary cohorts that no index refers to (its values are not used), against a block of zeros."""
    ts = qc_system(L)[4]
    p = problem(sizes, 3)[1]

    def zeros(o, at, size, d):
        d[o[at[-1]]:o[at[-1]] + size] = 0.0

    def left_out(o, at, size, d):
        o[at[-1]] = -1

    plans = [heff.plan_from_problem(gpu_ctx, altered(p, "L", f), ts, SITE) for f in (zeros, left_out)]
    x = np.random.default_rng(2).standard_normal(plans[0].n)
    ref, y = (q.apply(x) for q in plans)
    assert np.abs(y - ref).max() <= TOL * np.abs(ref).max()
    plan = plans[1]
    plan.apply(2.0 * x)  # other contents of the scratch that the next applies start from
    assert np.array_equal(plan.apply(x), y)
    whole = plan.info
    plan.chunk_apply(8 * (whole["t_len"] + whole["s_len"] + whole["w_len"]) // 3)
    assert np.abs(plan.apply(x) - ref).max() <= TOL * np.abs(ref).max()
