"""Workloads of the engine as its users run them, through the package's public entry points.

Every case is a seeded system of noci-rs-like shape (a few reference determinants, all their singles
and doubles) and one call, or one short run of calls, that a NOCI, NOCI-PT2, selected-NOCI or
NOCI-QMC program makes over and over:

* ``hs``         (H, S) of determinant pairs, device buffers (``eval_pairs_device``);
* ``hs_host``    the same from and to host buffers (``eval_pairs``), the drop-in of
                 calculate_hs_pairs_wicks_batched;
* ``fs``         (F, S) of pairs (``eval_fs_pairs_device``), the SNOCI / PT2 element;
* ``build``      the intermediates of every ordered reference pair, then a batch of pairs over them:
                 a new geometry or a new reference set;
* ``pt2_solve``  one NOCI-PT2 correction: the candidate operator and its GMRES solve;
* ``pt2_apply``  one product with the stored candidate operator;
* ``qmc``        NOCI-QMC report blocks;
* ``overlap``    the overlap action y = S x over the resident basis.

Results are compared with ``exact``: the generalised Slater-Condon expressions in terms of the minors of
the occupied overlap, written with plain torch in 64 bits.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "noci-rs_b200"))

import nociwick  # noqa: E402
from nociwick import synthetic as sy  # noqa: E402

_MAX_WORK = 64 ** 4 * 36   # nmo^4 nref^2 of the largest system (15 GB of intermediates)


def listed():
    return [
        # the smallest call: a few rows of H and S asked for by a driver, latency and launches count
        {"name": "hs_small", "kind": "hs", "nmo": 30, "nocc": 3, "nref": 3, "npairs": 512, "pairs": "any", "zero": 0},
        # one spawning step of a 10^6-walker program: uniform pairs, same-parent pairs among them
        {"name": "hs_step", "kind": "hs", "nmo": 40, "nocc": 4, "nref": 3, "npairs": 1_000_003, "pairs": "any", "zero": 0},
        # a large batch across references: the H6 / cc-pVDZ NOCISD(3) dimensions of the benchmark
        {"name": "hs_large", "kind": "hs", "nmo": 30, "nocc": 3, "nref": 3, "npairs": 10_000_000, "pairs": "across",
         "zero": 0},
        # reference pairs with zero-overlap orbitals among well-behaved ones, contraction ranks 0-4 uniform: the
        # benchmark's stress system (64 orbitals, 6 + 6 electrons), intermediates far larger than L2
        {"name": "hs_zero_overlap", "kind": "hs", "nmo": 64, "nocc": 6, "nref": 6, "npairs": 20_000_000,
         "pairs": "ranks", "zero": 3},
        # the host-buffer drop-in call with pinned arrays, at the size of a host-driven spawning step
        {"name": "hs_host", "kind": "hs_host", "nmo": 30, "nocc": 3, "nref": 3, "npairs": 300_001, "pairs": "any",
         "zero": 0},
        # Fock elements for selected NOCI at F2 / cc-pVDZ dimensions (9 + 9 electrons)
        {"name": "fs_large", "kind": "fs", "nmo": 28, "nocc": 9, "nref": 3, "npairs": 4_000_000, "pairs": "across",
         "zero": 0},
        # intermediates of a new geometry, small molecule, and the first elements from them
        {"name": "build_small", "kind": "build", "nmo": 30, "nocc": 3, "nref": 3, "npairs": 20_000, "pairs": "across",
         "zero": 0, "transform": "fp64"},
        # the same at 64 orbitals, one reference pair with a zero-overlap orbital
        {"name": "build_large", "kind": "build", "nmo": 64, "nocc": 4, "nref": 3, "npairs": 20_000, "pairs": "across",
         "zero": 1, "transform": "fp64"},
        # one PT2 correction over a screened candidate set: operator build and GMRES to 1e-8
        {"name": "pt2_solve", "kind": "pt2_solve", "nmo": 28, "nocc": 9, "nref": 3, "ncand": 12_000},
        # the product that a solve repeats, at a candidate count whose matrix streams from HBM
        {"name": "pt2_apply", "kind": "pt2_apply", "nmo": 28, "nocc": 9, "nref": 3, "ncand": 50_001},
        # 20 steps of NOCI-QMC with 10^6 walkers: the H8 / cc-pVDZ NOCISD(3) dimensions of the benchmark
        {"name": "qmc_blocks", "kind": "qmc", "nmo": 40, "nocc": 4, "nref": 3, "walkers": 1_000_000, "reports": 2},
        # the population update of the direct-overlap propagator over the same space
        {"name": "overlap_action", "kind": "overlap", "nmo": 40, "nocc": 4, "nref": 3},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hs", "hs", "hs_host", "fs", "build", "pt2_solve", "pt2_apply", "qmc", "overlap"])
    if kind in ("hs", "hs_host", "fs", "build"):
        nmo = rng.randint(10, 40 if kind == "fs" else 64)
        nocc = rng.randint(2, 9 if kind == "fs" else 6)
        nocc = min(nocc, nmo // 3)
        nref = rng.randint(2, 3 if kind == "build" else 8)
        while nmo ** 4 * nref ** 2 > _MAX_WORK:
            nref -= 1
        # kept below the largest listed basis
        while nref * _block(nmo, nocc) > 1_100_000:
            nocc -= 1
        zero = rng.choice([0, 0, 1]) if kind in ("hs", "build") else 0
        npairs = {"hs": _log(rng, 300, 10_000_000), "hs_host": _log(rng, 300, 1_000_000),
                  "fs": _log(rng, 1000, 4_000_000), "build": _log(rng, 1000, 50_000)}[kind]
        c = {"kind": kind, "nmo": nmo, "nocc": nocc, "nref": nref, "npairs": npairs,
             "pairs": rng.choice(["across", "ranks"] if kind in ("fs", "build") or zero else ["any", "across", "ranks"]),
             "zero": zero}
        if kind == "build":
            c["transform"] = rng.choice(["fp64", "fp64", "chol_int8"])
        return c
    if kind in ("pt2_solve", "pt2_apply"):
        nmo, nocc = rng.randint(16, 28), rng.randint(3, 9)
        nocc = min(nocc, nmo // 3)
        most = min(12_000 if kind == "pt2_solve" else 50_000, 3 * _block(nmo, nocc) - 3)
        return {"kind": kind, "nmo": nmo, "nocc": nocc, "nref": 3, "ncand": _log(rng, min(500, most), most)}
    nmo, nocc = rng.randint(16, 40), rng.randint(2, 4)
    if kind == "qmc":
        return {"kind": kind, "nmo": nmo, "nocc": nocc, "nref": 3, "walkers": _log(rng, 10_000, 1_000_000), "reports": 2}
    return {"kind": kind, "nmo": nmo, "nocc": nocc, "nref": rng.choice([2, 3])}


def _strings(nmo, nocc):
    """Occupation strings of one spin reached by at most two excitations of a reference."""
    v = nmo - nocc
    return 1 + nocc * v + math.comb(nocc, 2) * math.comb(v, 2)


def _block(nmo, nocc):
    """Determinants of one reference: itself, all singles and doubles."""
    s, d = nocc * (nmo - nocc), math.comb(nocc, 2) * math.comb(nmo - nocc, 2)
    return 1 + 2 * s + 2 * d + s * s


def _system(case, seed):
    n, o, nref, kind = case["nmo"], case["nocc"], case["nref"], case["kind"]
    if kind in ("pt2_solve", "pt2_apply", "qmc", "overlap", "fs"):
        eps = np.concatenate([np.linspace(-1.5 if o > 4 else -1.0, -0.5, o), np.linspace(0.2, 2.5, n - o)])
        return sy.make_system(n, o, o, nref, 4 * n, seed, sigma_h=0.02, sigma_l=0.02, k_scale=0.3, uhf_like=True,
                              orbital_energies=eps)
    zero = [z for z in ((0, 1, 1, 0), (2, 3, 0, 2), (4, 5, 1, 1))[:case["zero"]] if max(z[:2]) < nref and max(z[2:]) <= o]
    return sy.make_system(n, o, o, nref, 4 * n, seed, k_scale=0.08, zero_pairs=zero, uhf_like=nref <= 3)


def _basis(case):
    return sy.sd_basis(case["nmo"], case["nocc"], case["nocc"], case["nref"])


def _pairs(case, basis, seed):
    """Determinant pairs (a <= b), int32 on the device: uniform over all pairs ("any"), over pairs of
    different references ("across"), or with the total excitation rank uniform over 0..4 ("ranks")."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    m, nref = case["npairs"], case["nref"]
    per = basis.shape[0] // nref

    def below(k):
        return (torch.rand(m, generator=g, device="cuda", dtype=torch.float64) * k).long()

    if case["pairs"] == "ranks":
        rank = (basis["rank_a"][:per].astype(np.int64) + basis["rank_b"][:per])
        order = torch.from_numpy(np.argsort(rank, kind="stable")).cuda()
        size = torch.from_numpy(np.bincount(rank, minlength=3)).cuda()
        off = torch.cumsum(size, 0) - size
        t = below(5)
        lo = torch.clamp(t - 2, min=0)
        rx = lo + below(torch.clamp(t, max=2) - lo + 1)
        local = [order[off[r] + below(size[r])] for r in (rx, t - rx)]
    else:
        local = [below(per), below(per)]
    px = below(nref)
    pw = below(nref) if case["pairs"] == "any" else (px + 1 + below(nref - 1)) % nref
    ab = torch.stack([px * per + local[0], pw * per + local[1]], dim=1)
    return torch.sort(ab, dim=1).values.to(torch.int32).contiguous()


def _engine(case, system, basis, transform="fp64"):
    # "build" uses the exact convention for zero-overlap reference pairs, the others the default one
    conv = "exact" if case["kind"] == "build" else "reference"
    chol = system.chol if transform != "fp64" else None
    w = nociwick.WicksShared(system.s, system.h, None if chol is not None else system.eri, system.enuc, system.refs,
                             tol=1e-8, convention=conv, chol=chol)
    if chol is not None:
        w.set_transform(transform)
    return w.build().set_basis(basis) if case["kind"] != "overlap" else w.set_basis(basis)


def _references(basis):
    return np.nonzero((basis["rank_a"] == 0) & (basis["rank_b"] == 0))[0].astype(np.uint32)


def prepare(case, seed):
    kind = case["kind"]
    system, basis = _system(case, seed), _basis(case)
    w = _engine(case, system, basis, case.get("transform", "fp64"))
    st = {"case": case, "w": w, "stream": torch.cuda.current_stream().cuda_stream}
    if kind in ("hs", "fs", "build", "hs_host"):
        st["pairs"] = _pairs(case, basis, seed)
        if kind == "fs":
            w.update_fock(*sy.reference_fock(system, 0))
        if kind == "hs_host":
            st["host_pairs"] = st["pairs"].cpu().pin_memory().numpy().view(np.uint32)
            st["host_out"] = torch.empty((case["npairs"], 2), dtype=torch.float64).pin_memory().numpy()
        st["out"] = torch.empty((case["npairs"], 2), dtype=torch.float64, device="cuda")
        return st
    if kind == "overlap":
        g = torch.Generator(device="cuda").manual_seed(seed)
        st["x"] = torch.randn(basis.shape[0], dtype=torch.float64, device="cuda", generator=g)
        st["y"] = torch.zeros_like(st["x"])
        w.apply_overlap_device(st["x"].data_ptr(), st["y"].data_ptr(), st["stream"])   # the factor tables
        return st
    refs = _references(basis)
    hr, sr = w.build_hs_matrix(refs, refs)
    er, cr = w.general_evp(hr, sr, project=True, tol=1e-8)
    c = cr[:, 0]
    rng = np.random.default_rng(seed)
    if kind == "qmc":
        # walkers as they lie in a run: on the references first, with a tail over the whole space
        c0 = np.zeros(basis.shape[0])
        c0[refs] = c
        q = nociwick.Qmc(w, c0, refs, dt=1e-3, initial_population=case["walkers"], target_population=case["walkers"],
                         shift_damping=0.5, initial_shift=float(er[0]), ncycles=10, propagator="unshifted",
                         seed=seed % (1 << 31) + 1, max_attempts=48_000_000)
        pop = rng.normal(size=basis.shape[0]) * rng.pareto(2.0, size=basis.shape[0])
        pop *= 0.6 * case["walkers"] / np.abs(pop).sum()
        pop[refs] += 0.4 * case["walkers"] * c / np.abs(c).sum()
        q.set_populations(pop)
        st["q"] = q
        return st
    cand = np.setdiff1d(np.arange(basis.shape[0]), refs)
    cand = np.sort(rng.choice(cand, case["ncand"], replace=False)).astype(np.uint32)
    w.update_fock(*sy.reference_fock(system, 0))
    fr, _ = w.build_fs_matrix(refs, refs)
    e0 = float(c @ fr @ c)
    st.update(cand=cand, e0=e0)
    if kind == "pt2_apply":
        st["pt2"] = w.pt2(cand, e0)
        st["x"] = rng.normal(size=case["ncand"])
        return st
    h_ar, s_ar = w.build_hs_matrix(cand, refs, symmetric=False)
    f_ar, _ = w.build_fs_matrix(cand, refs, symmetric=False)
    f_ra, s_ra = w.build_fs_matrix(refs, cand, symmetric=False)
    s_a0 = s_ar @ c
    st.update(s_a0=s_a0, f_a0=f_ar @ c, s_0a=s_ra.T @ c, f_0a=f_ra.T @ c, rhs=-(h_ar @ c - float(er[0]) * s_a0))
    return st


def run(state):
    case, w = state["case"], state["w"]
    kind = case["kind"]
    if kind == "hs":
        w.eval_pairs_device(state["pairs"].data_ptr(), case["npairs"], state["out"].data_ptr(), state["stream"])
        return state["out"]
    if kind == "hs_host":
        return w.eval_pairs(state["host_pairs"], state["host_out"])
    if kind == "fs":
        w.eval_fs_pairs_device(state["pairs"].data_ptr(), case["npairs"], state["out"].data_ptr(), state["stream"])
        return state["out"]
    if kind == "build":
        w.build()
        w.eval_pairs_device(state["pairs"].data_ptr(), case["npairs"], state["out"].data_ptr(), state["stream"])
        return state["out"]
    if kind == "overlap":
        state["y"].zero_()
        w.apply_overlap_device(state["x"].data_ptr(), state["y"].data_ptr(), state["stream"])
        return state["y"]
    if kind == "pt2_apply":
        return state["pt2"].apply_m(state["x"])
    if kind == "pt2_solve":
        with w.pt2(state["cand"], state["e0"]) as p:
            x, _ = p.solve(state["e0"], state["s_a0"], state["s_0a"], state["f_a0"], state["f_0a"], state["rhs"],
                           max_iter=60, restart=30, res_tol=1e-8)
        return x
    rep = state["q"].run(case["reports"])
    return {"reports": {k: rep[k] for k in nociwick.Qmc.REPORT_FIELDS}, "populations": state["q"].populations()}


def work(case):
    n, o, nref, kind = case["nmo"], case["nocc"], case["nref"], case["kind"]
    ndet = nref * _block(n, o)
    if kind in ("hs", "hs_host", "fs"):
        # pair, result, and the entries of the intermediates of a (2, 2) pair (every table at most once)
        per = 8 * (16 + 2 + 16) if kind != "fs" else 8 * 16
        table = nref ** 2 * 8 * (3 * n ** 4 + 8 * n * n if kind != "fs" else 8 * n * n)
        m = case["npairs"]
        return {"bytes": 24.0 * m + 32.0 * ndet + min(float(per) * m, float(table)), "flops": (150.0 if kind != "fs" else 60.0) * m}
    if kind == "build":
        # Coulomb tensor (or factors) in, intermediates out; (aa|aa), (aa|bb), (bb|bb) of every ordered pair
        chol = case["transform"] != "fp64"
        flops = nref ** 2 * (3 * 2.0 * n ** 4 * (4 * n) if chol else 10 * 2.0 * n ** 5)
        return {"bytes": 8.0 * ((4 * n ** 3 if chol else n ** 4) + nref ** 2 * (3 * n ** 4 + 8 * n * n)), "flops": flops}
    if kind in ("pt2_solve", "pt2_apply"):
        half = case["ncand"] * (case["ncand"] + 1) / 2
        if kind == "pt2_apply":
            return {"bytes": 8.0 * half + 16.0 * case["ncand"], "flops": 4.0 * half}
        return {"bytes": 8.0 * half * 20, "flops": half * (60.0 + 4.0 * 20)}
    if kind == "qmc":
        m = 10.0 * case["reports"] * case["walkers"]
        return {"bytes": 24.0 * m + 10.0 * case["reports"] * 24 * ndet, "flops": 150.0 * m}
    # the two single-spin tables of every ordered pair of references, and x B^T then A U on the occupied pattern
    ns = _strings(n, o)
    return {"bytes": nref * (nref - 1) * 2 * 8.0 * ns * ns + 16.0 * ndet,
            "flops": nref * (nref - 1) * 4.0 * _block(n, o) * ns}


# ---------------------------------------------------------------------------------------------------
# The same results in 64 bits with plain torch.  With M = <x occupied | w occupied> of one spin,
# S = det M_a det M_b and H follows from M's first and second minors, without dividing by det M.
# ---------------------------------------------------------------------------------------------------
def _occupied(dets, spin, nocc):
    """Ascending occupied orbitals of every determinant, one spin."""
    rank = dets["rank_a" if spin == 0 else "rank_b"].astype(np.int64)
    idx = dets["idx_a" if spin == 0 else "idx_b"].astype(np.int64)
    occ = np.tile(np.arange(nocc), (dets.shape[0], 1))
    for k in range(int(rank.max(initial=0))):
        on = np.nonzero(rank > k)[0]
        occ[on, idx[on, k]] = idx[on, 4 + k]
    return torch.from_numpy(np.sort(occ, axis=1)).cuda()


def _det(m):
    """Determinants of small matrices by expansion along the first row."""
    k = m.shape[-1]
    if k == 0:
        return torch.ones(m.shape[:-2], dtype=m.dtype, device=m.device)
    if k == 1:
        return m[..., 0, 0]
    if k > 4:
        return torch.linalg.det(m)
    tot = 0.0
    for c in range(k):
        rest = [j for j in range(k) if j != c]
        tot = tot + (-1.0) ** c * m[..., 0, c] * _det(m[..., 1:, :][..., rest])
    return tot


def _without(m, rows, cols):
    k = m.shape[-1]
    return m[..., [r for r in range(k) if r not in rows], :][..., [c for c in range(k) if c not in cols]]


def _first_minors(m):
    k = m.shape[-1]
    return torch.stack([torch.stack([(-1.0) ** (r + c) * _det(_without(m, (r,), (c,))) for c in range(k)], -1)
                        for r in range(k)], -2)


def _groups(basis, pairs, nref):
    par = torch.from_numpy(basis["parent"].astype(np.int64)).cuda()
    key = par[pairs[:, 0].long()] * nref + par[pairs[:, 1].long()]
    for p in range(nref * nref):
        sel = torch.nonzero(key == p).flatten()
        if sel.numel():
            yield p // nref, p % nref, sel


def _exact_hs(case, system, basis, pairs):
    o, nref = case["nocc"], case["nref"]
    occ = [_occupied(basis, s, o) for s in (0, 1)]
    chol, h = torch.from_numpy(system.chol).cuda(), torch.from_numpy(system.h).cuda()
    out = torch.empty((pairs.shape[0], 2), dtype=torch.float64, device="cuda")
    c = [[torch.from_numpy(np.ascontiguousarray(r[2 * s])).cuda() for s in (0, 1)] for r in system.refs]
    comb = [(i, j) for i in range(o) for j in range(i + 1, o)]
    for x, w, sel in _groups(basis, pairs, nref):
        n = case["nmo"]
        ov = [c[x][s].T @ c[w][s] for s in (0, 1)]
        h1 = [c[x][s].T @ h @ c[w][s] for s in (0, 1)]
        b = [torch.einsum("mp,kmn,nq->kpq", c[x][s], chol, c[w][s]).reshape(chol.shape[0], n * n) for s in (0, 1)]
        eri = [(b[0].T @ b[0]).reshape(-1), (b[1].T @ b[1]).reshape(-1), (b[0].T @ b[1]).reshape(-1)]
        for part in torch.split(sel, 250_000):
            det, minors, one, same = [], [], 0.0, []
            ix, iw = [], []
            for s in (0, 1):
                ox, ow = occ[s][pairs[part, 0].long()], occ[s][pairs[part, 1].long()]
                ix.append(ox)
                iw.append(ow)
                m = ov[s][ox[:, :, None], ow[:, None, :]]
                det.append(_det(m))
                minors.append(_first_minors(m))
                two = torch.zeros_like(det[s])
                for (i, j) in comb:
                    for (k, l) in comb:
                        sec = (-1.0) ** (i + j + k + l) * _det(_without(m, (i, j), (k, l)))
                        direct = eri[s][((ox[:, i] * n + ow[:, k]) * n + ox[:, j]) * n + ow[:, l]]
                        swap = eri[s][((ox[:, i] * n + ow[:, l]) * n + ox[:, j]) * n + ow[:, k]]
                        two += sec * (direct - swap)
                same.append(two)
            for s in (0, 1):
                hs = h1[s][ix[s][:, :, None], iw[s][:, None, :]]
                one = one + ((hs * minors[s]).sum((1, 2)) + same[s]) * det[1 - s]
            mixed = torch.zeros_like(det[0])
            for i in range(o):
                for k in range(o):
                    e = ((ix[0][:, i] * n + iw[0][:, k]) * n * n)[:, None, None]
                    e = eri[2][e + ix[1][:, :, None] * n + iw[1][:, None, :]]
                    mixed += minors[0][:, i, k] * (e * minors[1]).sum((1, 2))
            sv = det[0] * det[1]
            out[part, 0] = one + mixed + system.enuc * sv
            out[part, 1] = sv
    return out


def _exact_fs(case, system, basis, pairs):
    o, nref = case["nocc"], case["nref"]
    occ = [_occupied(basis, s, o) for s in (0, 1)]
    eri, h = torch.from_numpy(system.eri).cuda(), torch.from_numpy(system.h).cuda()
    c = [[torch.from_numpy(np.ascontiguousarray(r[2 * s])).cuda() for s in (0, 1)] for r in system.refs]
    d = [c[0][s][:, :o] @ c[0][s][:, :o].T for s in (0, 1)]
    j = torch.einsum("pqrs,rs->pq", eri, d[0] + d[1])
    fock = [h + j - torch.einsum("prqs,rs->pq", eri, d[s]) for s in (0, 1)]
    out = torch.empty((pairs.shape[0], 2), dtype=torch.float64, device="cuda")
    for x, w, sel in _groups(basis, pairs, nref):
        ov = [c[x][s].T @ c[w][s] for s in (0, 1)]
        f1 = [c[x][s].T @ fock[s] @ c[w][s] for s in (0, 1)]
        for part in torch.split(sel, 250_000):
            det, tr = [], []
            for s in (0, 1):
                ox, ow = occ[s][pairs[part, 0].long()], occ[s][pairs[part, 1].long()]
                m = ov[s][ox[:, :, None], ow[:, None, :]]
                f = f1[s][ox[:, :, None], ow[:, None, :]]
                det.append(torch.linalg.det(m))
                tr.append(torch.diagonal(torch.linalg.solve(m, f), dim1=1, dim2=2).sum(1))
            sv = det[0] * det[1]
            out[part, 0] = sv * (tr[0] + tr[1])
            out[part, 1] = sv
    return out


def _exact_overlap(case, system, basis, seed):
    o, nref, per = case["nocc"], case["nref"], basis.shape[0] // case["nref"]
    x = torch.randn(basis.shape[0], dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))
    ids, strings = [], []
    for s in (0, 1):
        u, inv = torch.unique(_occupied(basis[:per], s, o), dim=0, return_inverse=True)
        strings.append(u)
        ids.append(inv)
    c = [[torch.from_numpy(np.ascontiguousarray(r[2 * s])).cuda() for s in (0, 1)] for r in system.refs]
    y = x.clone()     # determinants of one reference are orthonormal
    for p in range(nref):
        dense = torch.zeros((strings[0].shape[0], strings[1].shape[0]), dtype=torch.float64, device="cuda")
        dense[ids[0], ids[1]] = x[p * per:(p + 1) * per]
        for q in range(nref):
            if p == q:
                continue
            tab = []
            for s in (0, 1):
                ov = c[q][s].T @ c[p][s]
                t = [_det(ov[rows[:, None, :, None], strings[s][None, :, None, :]]) for rows in torch.split(strings[s], 256)]
                tab.append(torch.cat(t))
            y[q * per:(q + 1) * per] += (tab[0] @ dense @ tab[1].T)[ids[0], ids[1]]
    return y


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("hs", "hs_host", "fs", "build", "overlap"):
        return None               # stochastic, or too many elements
    if kind in ("hs", "hs_host", "build") and case["nocc"] > 4:
        return None               # too many second minors
    if kind == "hs" and case["zero"]:
        return None               # the default convention differs from the exact element there
    system, basis = _system(case, seed), _basis(case)
    if kind == "overlap":
        return _exact_overlap(case, system, basis, seed)
    pairs = _pairs(case, basis, seed)
    value = _exact_fs(case, system, basis, pairs) if kind == "fs" else _exact_hs(case, system, basis, pairs)
    return value.cpu().numpy() if kind == "hs_host" else value
