"""Timed cases of the two-site DMRG path: H_eff . psi in its forms, its adjoint, the lockstep solve of many
small problems, the truncation of a step and a whole sweep, each through the package's public calls.

The Hamiltonian is the package's seeded synthetic ab-initio one (L orbitals, N = L electrons, Sz = 0).  The
MPS has the bond sectors that a converged state of it has: sizes peak at half filling of the left part and fall
off as a Gaussian in its spin projection (wider in the middle of the chain), cut at the full space of either side; its entries are drawn from the seed, its sites right-normalised.
"""
import math
from functools import lru_cache
from itertools import combinations

import numpy as np
import torch

from qcmaquis_b200 import dmrg, heff
from qcmaquis_b200.fcidump import synthetic_integrals
from qcmaquis_b200.mpo import MPO

PHYS = [(1, 1, 1), (1, 0, 1), (0, 1, 1), (0, 0, 1)]  # (N_up, N_down, size) of one orbital, in sector order
# weight of a sector by how far its electron number is from half filling
NUMBER = {0: 1.0, 1: 0.3, 2: 0.27, 3: 0.03}


def listed():
    return [
        # the plain validation size (eight orbitals, M = 64) with host vectors: the smallest solver callback,
        # where launches and copies are most of the time
        dict(name="apply_host_L8_M64", kind="apply", L=8, M=64, site=3, form="fp64", host=True),
        # an odd bond dimension, off the middle of the chain
        dict(name="apply_L12_M101", kind="apply", L=12, M=101, site=3, form="fp64", host=False),
        # ordinary solver callbacks on device vectors, at the middle bond
        dict(name="apply_L16_M256", kind="apply", L=16, M=256, site=7, form="fp64", host=False),
        dict(name="apply_L24_M512", kind="apply", L=24, M=512, site=11, form="fp64", host=False),
        # a large one
        dict(name="apply_L24_M1024", kind="apply", L=24, M=1024, site=11, form="fp64", host=False),
        # the mixed-precision form of the callback
        dict(name="mixed_L20_M600", kind="apply", L=20, M=600, site=9, form="mixed", host=False),
        # the callback under a memory bound: coefficient blocks generated chunk by chunk in every apply
        dict(name="streamed_L20_M384", kind="streamed", L=20, M=384, site=9, mib=64),
        # the adjoint of the apply at the size of the gradient configuration (host vectors)
        dict(name="adjoint_L16_M256", kind="adjoint", L=16, M=256, site=7),
        # many independent small problems solved together (eight lockstep Jacobi-Davidson iterations)
        dict(name="group_jd_16xL12_M128", kind="group", L=12, M=128, site=5, members=16),
        # the truncation of one step at the middle bond of an M = 512 and of an M = 2048 state
        dict(name="svd_M512", kind="svd", L=24, M=512),
        dict(name="svd_M2048", kind="svd", L=24, M=2048),
        # one whole sweep of a run that has converged (all steps: boundaries, solve, truncation)
        dict(name="sweep_L16_M256", kind="sweep", L=16, M=256),
    ]


def draw(rng):
    def log_int(lo, hi):
        return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))
    kind = rng.choice(["apply", "apply", "apply", "mixed", "streamed", "adjoint", "group", "svd", "svd", "sweep"])
    L = rng.choice([8, 10, 12, 14, 16, 18, 20, 22, 24])
    site = min(L - 2, max(0, L // 2 - 1 + rng.choice([0, 0, 0, 1, -1, 2, -3])))
    if kind == "apply":
        return dict(kind="apply", L=L, M=log_int(24, 1000), site=site, form="fp64", host=rng.random() < 0.4)
    if kind == "mixed":
        return dict(kind="apply", L=L, M=log_int(48, 900), site=site, form="mixed", host=rng.random() < 0.4)
    if kind == "streamed":
        return dict(kind="streamed", L=L, M=log_int(48, 384), site=site, mib=rng.choice([16, 64, 200]))
    if kind == "adjoint":
        return dict(kind="adjoint", L=min(L, 18), M=log_int(32, 300), site=min(site, min(L, 18) - 2))
    if kind == "group":
        return dict(kind="group", L=min(L, 12), M=log_int(24, 128), site=min(site, min(L, 12) - 2), members=rng.randint(2, 16))
    if kind == "svd":
        return dict(kind="svd", L=L, M=log_int(48, 2000))
    return dict(kind="sweep", L=min(L, 16), M=log_int(32, 256))


# ---------------------------------------------------------------------------
# inputs

@lru_cache(maxsize=None)
def bond_sectors(L, M):
    """Sectors [(N_up, N_down, size)] of every bond 0 .. L of an MPS with bond dimension M."""
    n = L // 2
    bonds = []
    for i in range(L + 1):
        var_d = max(0.4, 0.78 * L * 4 * (i / L) * (1 - i / L))
        cap, w = {}, {}
        for a in range(n + 1):
            for b in range(n + 1):
                c = min(math.comb(i, a) * math.comb(i, b), math.comb(L - i, n - a) * math.comb(L - i, n - b))
                if c > 0:
                    cap[a, b] = c
                    w[a, b] = NUMBER.get(abs(a + b - i), 0.001) * math.exp(-((a - b) ** 2) / (1.2 * var_d))
        lo, hi = 0.0, 1e12
        for _ in range(200):  # the scale at which the capped sizes add up to M
            mid = (lo + hi) / 2
            lo, hi = (mid, hi) if sum(min(cap[q], int(mid * w[q] + 0.5)) for q in cap) < M else (lo, mid)
        bonds.append({q: min(cap[q], int(hi * w[q] + 0.5)) for q in cap})
    while True:  # a block's rows fit in its columns and its columns in its rows
        new = [dict(b) for b in bonds]
        for i in range(L):
            for (a, b), s in new[i].items():
                new[i][a, b] = min(s, sum(new[i + 1].get((a + p, b + q), 0) for p, q, _ in PHYS))
        for i in range(L, 0, -1):
            for (a, b), s in new[i].items():
                new[i][a, b] = min(s, sum(new[i - 1].get((a - p, b - q), 0) for p, q, _ in PHYS))
        if new == bonds:
            break
        bonds = new
    return [sorted(((a, b, s) for (a, b), s in d.items() if s > 0), reverse=True) for d in bonds]


def random_mps(L, M, seed):
    """Site tensors in the package's right-paired layout, sites 1 .. L - 1 right-normalised, norm 1."""
    rng = np.random.default_rng([seed, L, M])
    bonds = bond_sectors(L, M)
    sites, carry = [], None
    for i in range(L - 1, -1, -1):
        left, right = bonds[i], bonds[i + 1]
        size = {(a, b): s for a, b, s in right}
        blocks, lower = [], {}
        for a, b, ls in left:
            parts = []
            for p, q, _ in PHYS:
                rc = (a + p, b + q)
                if rc in size:
                    x = rng.standard_normal((ls, size[rc]))
                    parts.append(x if carry is None else x @ carry[rc])
            x = np.concatenate(parts, axis=1)
            if i > 0:
                qm, rm = np.linalg.qr(x.T)  # x = rm^T qm^T
                x, lower[a, b] = qm.T, rm.T / np.sqrt(ls)
            blocks.append(((a, b), x))
        carry = lower
        sites.insert(0, dict(phys=list(PHYS), left=left, right=right, blocks=blocks))
    norm = math.sqrt(sum(float((b * b).sum()) for _, b in sites[0]["blocks"]))
    sites[0]["blocks"] = [(c, b / norm) for c, b in sites[0]["blocks"]]
    return sites


@lru_cache(maxsize=None)
def hamiltonian(L, seed):
    h, V, _ = synthetic_integrals(L, seed)
    return h, V


@lru_cache(maxsize=2)
def mpo_of(L, seed):
    return MPO.qc(*hamiltonian(L, seed))


@lru_cache(maxsize=1)
def context():
    return heff.Context(0)


def site_plan(L, M, site, seed):
    """The plan of a two-site problem, its start vector, and the run that owns its boundaries."""
    d = dmrg.DMRG.from_mps(context(), mpo_of(L, seed), random_mps(L, M, seed), M, initial_site=site)
    plan, x = d.pending_plan()
    return d, plan, x


def svd_blocks(L, M, seed):
    """The two-site tensor at the middle bond, block by left-pair charge, with the decay of singular values
    that a converged state has (about 1e-6 at the truncated bond); the vectors are the seed's, the spectrum
    the state's."""
    rng, spectrum = np.random.default_rng([seed, L, M]), np.random.default_rng([L, M])
    bonds = bond_sectors(L, M)
    left = {(a, b): s for a, b, s in bonds[L // 2 - 1]}
    right = {(a, b): s for a, b, s in bonds[L // 2 + 1]}
    mid = {}
    for (a, b), s in left.items():
        for p, q, _ in PHYS:
            mid[a + p, b + q] = mid.get((a + p, b + q), 0) + s
    blocks = []
    for (a, b), m in sorted(mid.items(), reverse=True):
        n = sum(right.get((a + p, b + q), 0) for p, q, _ in PHYS)
        k = min(m, n)
        if k == 0:
            continue
        u, _ = np.linalg.qr(rng.standard_normal((m, k)))
        v, _ = np.linalg.qr(rng.standard_normal((n, k)))
        top = math.exp(-((a + b - L // 2 * 2) ** 2) / 2 - abs(a - b) / 2) * spectrum.uniform(0.3, 1.0)
        s = top * np.exp(-14.0 * (np.arange(k) + spectrum.uniform(0, 0.6, k)) / k)
        blocks.append(np.asfortranarray((u * s) @ v.T))
    return blocks


# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind, L, M = case["kind"], case["L"], case["M"]
    st = dict(case=case)
    if kind in ("apply", "streamed", "adjoint"):
        st["run"], plan, x = site_plan(L, M, case["site"], seed)
        st["plan"] = plan
        if kind == "streamed":
            plan.stream_coefficients(case["mib"] << 20)
        if kind == "adjoint" or case.get("host"):
            st["x"] = x
            st["ybar"] = np.random.default_rng([seed, 1]).standard_normal(plan.n)
        else:
            st["x"] = torch.from_numpy(x).cuda()
            st["y"] = torch.zeros(plan.n, dtype=torch.float64, device="cuda")
    elif kind == "group":
        made = [site_plan(L, M, case["site"], 1000 * seed + k) for k in range(case["members"])]
        st["runs"] = [m[0] for m in made]
        st["group"] = heff.HeffGroup(context(), [m[1] for m in made])
        st["x"] = st["group"].pack([m[2] for m in made])
    elif kind == "svd":
        st["ctx"], st["blocks"] = context(), svd_blocks(L, M, seed)
    else:
        # two sweeps bring the run near convergence: the steps' sectors hardly change from there on
        st["run"] = dmrg.DMRG.from_mps(context(), mpo_of(L, seed), random_mps(L, M, seed), M)
        for _ in range(2):
            st["run"].sweep()
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "apply" and case["host"]:
        return st["plan"].apply(st["x"], precision=case["form"])
    if kind == "apply":
        st["plan"].apply_device(st["x"].data_ptr(), st["y"].data_ptr(), precision=case["form"])
        return st["y"]
    if kind == "streamed":
        st["plan"].apply_device(st["x"].data_ptr(), st["y"].data_ptr())
        return st["y"]
    if kind == "adjoint":
        psi_bar, coeff_bar = st["plan"].adjoint(st["x"], st["ybar"])
        return dict(psi_bar=psi_bar, coeff_bar=coeff_bar)
    if kind == "group":
        ev, out, iters, applies = st["group"].jd_solve(st["x"], tol=1e-10, maxiter=8)
        return dict(evals=ev, vectors=out, iters=iters, applies=applies)
    if kind == "svd":
        kept, res = dmrg.truncate_svd(st["ctx"], st["blocks"], case["M"], 1e-16)
        return dict(U=np.concatenate([u.ravel() for u, _, _ in kept]), S=np.concatenate([s for _, s, _ in kept]),
                    Vt=np.concatenate([v.ravel() for _, _, v in kept]), keep=np.array([s.size for _, s, _ in kept]),
                    weight=res["truncated_weight"], smallest=res["smallest_ev"])
    # The state itself is defined up to the gauge of its bonds, and what a step cuts off (the default cutoff,
    # 1e-16 of the largest singular value) is rounding: the energy of every step is what a sweep determines.
    return st["run"].sweep()[0]


@lru_cache(maxsize=None)
def _work(key):
    case = dict(key)
    kind = case["kind"]
    if kind == "svd":
        # thin SVD of a dense block with both factors (Golub & Van Loan): 6 m k^2 + 20 k^3
        shapes = [b.shape for b in svd_blocks(case["L"], case["M"], 0)]
        return dict(bytes=float(sum(8 * (m * n + (m + n + 1) * min(m, n)) for m, n in shapes)),
                    flops=float(sum(6 * max(m, n) * min(m, n) ** 2 + 20 * min(m, n) ** 3 for m, n in shapes)))
    if kind == "sweep":
        st = prepare(case, 0)
        run(st)
        before = st["run"].stats()["hpsi_flops"]
        run(st)
        flops = st["run"].stats()["hpsi_flops"] - before
        bonds = bond_sectors(case["L"], case["M"])
        mps = sum(s * sum(r for x, y, r in bonds[i + 1] for p, q, _ in PHYS if (x, y) == (a + p, b + q))
                  for i in range(case["L"]) for a, b, s in bonds[i])
        return dict(bytes=8.0 * 2 * mps, flops=float(flops))
    st = prepare(dict(case, members=1) if kind == "group" else case, 0)
    info = st["group"].info if kind == "group" else st["plan"].info
    if kind == "group":
        plan = st["group"].plans[0].info
        return dict(bytes=8.0 * case["members"] * (plan["l_len"] + plan["r_len"] + 2 * plan["vec_len"]),
                    flops=9.0 * case["members"] * info["flops"])
    # the reference's count of one H.psi; the adjoint does the contractions of two (H ybar, and T(x) with its cotangents)
    times = 2 if kind == "adjoint" else 1
    return dict(bytes=8.0 * (info["l_len"] + info["r_len"] + 2 * times * info["vec_len"]), flops=float(times * info["flops"]))


def work(case):
    return _work(tuple(sorted((k, v) for k, v in case.items() if k != "name")))


# ---------------------------------------------------------------------------
# values in plain numpy

def exact(case, seed):
    kind, L, M = case["kind"], case["L"], case["M"]
    if kind == "svd":
        if M > 1200:
            return None
        s = [np.linalg.svd(b, compute_uv=False) for b in svd_blocks(L, M, seed)]
        top = np.sort(np.concatenate(s))[::-1]
        cut = top[M] if top.size > M else 0.0  # the value after the M-th stays: ties with it are kept
        S = [x[x >= cut] for x in s]
        # singular vectors are defined up to a sign, and the discarded weight is a small difference
        return dict(U=None, S=np.concatenate(S), Vt=None, keep=np.array([x.size for x in S]), weight=None, smallest=None)
    if L > 8 or kind in ("group", "sweep"):
        return None
    sites = random_mps(L, M, seed)
    if kind == "adjoint":
        n = _twin(sites, case["site"]).size
        ybar = np.random.default_rng([seed, 1]).standard_normal(n)
        return dict(psi_bar=_heff_dense(L, seed, sites, case["site"], ybar), coeff_bar=None)
    return _heff_dense(L, seed, sites, case["site"], _twin(sites, case["site"]))


def _dense_site(site):
    """A[state, l, r] of a right-paired site tensor."""
    lo = {(a, b): o for (a, b, _), o in zip(site["left"], np.cumsum([0] + [s[2] for s in site["left"]]))}
    ro = {(a, b): (o, s) for (a, b, s), o in zip(site["right"], np.cumsum([0] + [s[2] for s in site["right"]]))}
    A = np.zeros((4, sum(s[2] for s in site["left"]), sum(s[2] for s in site["right"])))
    for (a, b), blk in site["blocks"]:
        col = 0
        for k, (p, q, _) in enumerate(PHYS):
            if (a + p, b + q) in ro:
                o, s = ro[a + p, b + q]
                A[k, lo[a, b]:lo[a, b] + blk.shape[0], o:o + s] = blk[:, col:col + s]
                col += s
    return A


def _twin_columns(left, right, a, b):
    """Columns of a twin block: (state of the first site, state of the second, slice of the right index), in
    the order of the pair's charges (descending) and of the pairs within a charge."""
    ro = {(x, y): (o, s) for (x, y, s), o in zip(right, np.cumsum([0] + [s[2] for s in right]))}
    pairs = {}
    for k1, (p1, q1, _) in enumerate(PHYS):
        for k2, (p2, q2, _) in enumerate(PHYS):
            pairs.setdefault((p1 + p2, q1 + q2), []).append((k1, k2))
    for c in sorted(pairs, reverse=True):
        if (a + c[0], b + c[1]) in ro:
            o, s = ro[a + c[0], b + c[1]]
            for k1, k2 in pairs[c]:
                yield k1, k2, slice(o, o + s)


def _pack_twin(theta, left, right):
    out, row = [], 0
    for a, b, ls in left:
        for k1, k2, sl in _twin_columns(left, right, a, b):
            out.append(theta[row:row + ls, k1, k2, sl].T.ravel())
        row += ls
    return np.concatenate(out)


def _unpack_twin(x, left, right):
    theta = np.zeros((sum(s[2] for s in left), 4, 4, sum(s[2] for s in right)))
    row = at = 0
    for a, b, ls in left:
        for k1, k2, sl in _twin_columns(left, right, a, b):
            n = sl.stop - sl.start
            theta[row:row + ls, k1, k2, sl] = x[at:at + ls * n].reshape(n, ls).T
            at += ls * n
        row += ls
    return theta


def _twin(sites, site):
    theta = np.einsum("alm,bmr->labr", _dense_site(sites[site]), _dense_site(sites[site + 1]))
    return _pack_twin(theta, sites[site]["left"], sites[site + 1]["right"])


def _heff_dense(L, seed, sites, site, x):
    """P^T H P x with the Hamiltonian in the full space and P the two outer parts of the MPS."""
    left = np.ones((1, 1))
    for s in sites[:site]:
        left = np.einsum("fl,alr->far", left, _dense_site(s)).reshape(-1, sum(q[2] for q in s["right"]))
    right = np.ones((1, 1))
    for s in reversed(sites[site + 2:]):
        right = np.einsum("alr,fr->afl", _dense_site(s), right).reshape(-1, sum(q[2] for q in s["left"]))
    theta = _unpack_twin(x, sites[site]["left"], sites[site + 1]["right"])
    full = np.einsum("fl,labr,gr->fabg", left, theta, right, optimize=True)
    out = _hamiltonian_on(L, seed, full.ravel()).reshape(full.shape)
    theta = np.einsum("fl,fabg,gr->labr", left, out, right, optimize=True)
    return _pack_twin(theta, sites[site]["left"], sites[site + 1]["right"])


def _hamiltonian_on(L, seed, full):
    """H |full> in second quantisation: modes in the order (orbital 0 up, orbital 0 down, orbital 1 up, ...)."""
    h, V = hamiltonian(L, seed)
    n = L // 2
    basis = [sum(1 << 2 * o for o in up) | sum(2 << 2 * o for o in dn)
             for up in combinations(range(L), n) for dn in combinations(range(L), n)]
    bits = np.array(basis, dtype=np.int64)
    at = {b: i for i, b in enumerate(basis)}
    state = {(1, 1): 0, (1, 0): 1, (0, 1): 2, (0, 0): 3}  # (up, down) -> its place in PHYS
    place = np.zeros(bits.size, dtype=np.int64)
    look = np.array([[state[u, d] for d in (0, 1)] for u in (0, 1)])
    for o in range(L):
        place = 4 * place + look[(bits >> 2 * o) & 1, (bits >> 2 * o + 1) & 1]
    pos = np.full(1 << 2 * L, -1, dtype=np.int64)
    pos[bits] = np.arange(bits.size)

    def parity(m):
        for s in (16, 8, 4, 2, 1):
            m = m ^ (m >> s)
        return 1.0 - 2.0 * (m & 1)

    def hop(p, q):  # sum over spins of a+_p a_q: (target, source, sign)
        t, s, g = [], [], []
        for spin in (0, 1):
            mp, mq = 2 * p + spin, 2 * q + spin
            src = np.nonzero((bits >> mq) & 1)[0]
            b = bits[src]
            sign = parity(b & ((1 << mq) - 1))
            b = b ^ (1 << mq)
            ok = ((b >> mp) & 1) == 0
            src, b, sign = src[ok], b[ok], sign[ok]
            t.append(pos[b | (1 << mp)]); s.append(src); g.append(sign * parity(b & ((1 << mp) - 1)))
        return np.concatenate(t), np.concatenate(s), np.concatenate(g)

    c = full[place]
    hops = [hop(p, q) for p in range(L) for q in range(L)]

    def act(k, v):
        t, s, g = hops[k]
        return np.bincount(t, weights=g * v[s], minlength=bits.size)

    one = (h - 0.5 * np.einsum("prrq->pq", V)).ravel()
    D = np.stack([act(k, c) for k in range(L * L)])
    G = 0.5 * V.reshape(L * L, L * L) @ D
    sigma = sum(act(k, one[k] * c + G[k]) for k in range(L * L))
    out = np.zeros_like(full)
    out[place] = sigma
    return out
