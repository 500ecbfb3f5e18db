"""Packed candidate matrix from single-spin string pairs against the dense (F, S) matrices of the pair
evaluation: products with M over unsorted, repeated and single-parent candidates, ranks up to 4 per spin,
zero-overlap reference pairs, both conventions, on both sides of the size rule.

An entry is the same expression on both routes, so a product differs by the summation order and a few
roundings an entry: bound 16 n 2^-53 max_a sum_b |M_ab| |x_b|.
"""
import numpy as np
import pytest

import nociwick
from nociwick import synthetic as sy

pytestmark = pytest.mark.gpu


def _check(w, cand, e0, seed):
    f, s = w.build_fs_matrix(cand, cand, symmetric=False)
    up = np.triu(f - e0 * s)
    m = up + np.triu(up, 1).T
    rng = np.random.default_rng(seed)
    with nociwick.Pt2(w, cand, e0) as pt:
        for _ in range(3):
            x = rng.normal(size=cand.shape[0])
            bound = 16 * cand.shape[0] * 2.0 ** -53 * np.max(np.abs(m) @ np.abs(x))
            assert np.max(np.abs(pt.apply_m(x) - m @ x)) <= bound
    return m


@pytest.mark.parametrize("convention", ["reference", "exact"])
@pytest.mark.parametrize("zero_pairs", [[], [(0, 1, 1, 0)], [(0, 1, 0, 2), (1, 2, 1, 1)]])
def test_product_all_ranks(zero_pairs, convention):
    system = sy.make_system(8, 3, 3, 3, 20, seed=1, k_scale=0.3, zero_pairs=zero_pairs, enuc=0.37)
    basis = sy.sd_basis(8, 3, 3, 3, orders=(1, 2, 3, 4))
    rng = np.random.default_rng(5)
    fa = system.h + np.diag(rng.normal(size=8))
    fb = system.h - np.diag(rng.normal(size=8))
    nd = basis.shape[0]
    with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8,
                              convention=convention) as w:
        w.build().set_basis(basis)
        w.update_fock(fa, fb)
        for n in (1023, 1024, 1537):
            _check(w, rng.choice(nd, n, replace=True).astype(np.uint32), -1.25, n)   # unsorted, repeated


def test_single_parent_zeros_and_rule():
    """One parent: exact zeros beyond doubles; sorted candidates of all parents; too few repeats."""
    system = sy.make_system(12, 4, 3, 3, 40, seed=2, k_scale=0.3)
    basis = sy.sd_basis(12, 4, 3, 3)
    nd = basis.shape[0]
    per = nd // 3
    with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8) as w:
        w.build().set_basis(basis)
        w.update_fock(system.h, 0.9 * system.h)
        m = _check(w, np.arange(per, 2 * per, dtype=np.uint32)[:1100], 0.75, 1)
        assert (m == 0.0).mean() > 0.1
        _check(w, np.arange(0, nd, 2, dtype=np.uint32), -0.5, 2)
        # only doubles in one spin: every candidate has its own string
        own = np.nonzero((basis["rank_a"] == 2) | (basis["rank_b"] == 2))[0].astype(np.uint32)
        _check(w, own[:1200], -0.5, 3)


def test_matrix_and_vectors_kept_between_operators():
    """Operators of other sizes made, used and destroyed in turn on one context, two alive at once: the kept
    matrix and GMRES vectors hold nothing of an earlier operator."""
    system = sy.make_system(12, 4, 3, 3, 40, seed=2, k_scale=0.3)
    basis = sy.sd_basis(12, 4, 3, 3)
    nd = basis.shape[0]
    rng = np.random.default_rng(1)

    def product(w, cand, x):
        with nociwick.Pt2(w, cand, -0.5) as pt:
            return pt.apply_m(x)

    sizes = (1500, 700, 1600, 1500)
    cands = [rng.choice(nd, n, replace=False).astype(np.uint32) for n in sizes]
    xs = [rng.normal(size=n) for n in sizes]
    fresh, solved = [], []
    opts = dict(max_iter=12, restart=5, res_tol=1e-10)

    def solve(pt, n, x):
        z = np.zeros(n)
        return pt.solve(0.0, z, z, z, z, x, **opts)

    for cand, x in zip(cands, xs):
        with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8) as w:
            w.build().set_basis(basis)
            w.update_fock(system.h, system.h)
            fresh.append(product(w, cand, x))
            with nociwick.Pt2(w, cand, -0.5) as pt:
                solved.append(solve(pt, cand.shape[0], x))
    with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8) as w:
        w.build().set_basis(basis)
        w.update_fock(system.h, system.h)
        for cand, x, y, (sx, si) in zip(cands, xs, fresh, solved):
            # column sums reach y by FP64 atomics in no fixed order
            assert np.max(np.abs(product(w, cand, x) - y)) <= 1e-11 * max(1.0, np.max(np.abs(y)))
            with nociwick.Pt2(w, cand, -0.5) as pt, nociwick.Pt2(w, cands[1], -0.5) as other:
                gx, gi = solve(pt, cand.shape[0], x)
                assert gi["iterations"] == si["iterations"]
                assert np.max(np.abs(gx - sx)) <= 1e-6 * max(1.0, np.max(np.abs(sx)))
                assert np.max(np.abs(other.apply_m(xs[1]) - fresh[1])) <= 1e-11 * max(1.0, np.max(np.abs(fresh[1])))


def test_operator_outlives_its_context():
    """An operator destroyed after its context gives its matrix back to the device, not to the context."""
    system = sy.make_system(10, 3, 3, 3, 24, seed=7, k_scale=0.3)
    basis = sy.sd_basis(10, 3, 3, 3)
    w = nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8)
    w.build().set_basis(basis)
    w.update_fock(system.h, system.h)
    pt = nociwick.Pt2(w, np.arange(1200, dtype=np.uint32), -0.5)
    w.close()
    pt.close()


def test_rows_beyond_shared_memory():
    """More strings than a staged pair of table rows holds (220 KB: 14080 strings of both spins): columns of M
    against the elements of the pair evaluation, which agree to a few roundings of terms of order 10."""
    system = sy.make_system(28, 9, 9, 3, 112, seed=2, sigma_h=0.02, sigma_l=0.02, k_scale=0.3, uhf_like=True)
    basis = sy.sd_basis(28, 9, 9, 3)
    rng = np.random.default_rng(6)
    kinds = [((2, 0), 6900), ((0, 2), 6900), ((1, 1), 16200)]
    cand = np.concatenate([rng.choice(np.nonzero((basis["rank_a"] == a) & (basis["rank_b"] == b))[0], k, replace=False)
                           for (a, b), k in kinds])
    cand = rng.permutation(cand).astype(np.uint32)
    n = cand.shape[0]
    strings = [len({(int(d["parent"]), int(d[r]), d[i].tobytes()) for d in basis[cand]})
               for r, i in (("rank_a", "idx_a"), ("rank_b", "idx_b"))]
    assert sum(strings) > 14080 and strings[0] ** 2 + strings[1] ** 2 <= n * (n + 1) // 8
    e0 = -0.75
    with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8) as w:
        w.build().set_basis(basis)
        w.update_fock(*sy.reference_fock(system, 0))
        with nociwick.Pt2(w, cand, e0) as pt:
            for k in (0, 1, n // 2, n - 2, n - 1):
                x = np.zeros(n)
                x[k] = 1.0
                pos = np.arange(n)
                pairs = np.stack([cand[np.minimum(pos, k)], cand[np.maximum(pos, k)]], axis=1)
                fs = w.eval_fs_pairs(pairs)
                assert np.max(np.abs(pt.apply_m(x) - (fs[:, 0] - e0 * fs[:, 1]))) <= 1e-12


@pytest.mark.parametrize("restart", [4, 7, 40])
def test_long_solves_replay_the_step(restart):
    """Solves beyond the plain steps, in one cycle and over several (the step is replayed as a graph), against the
    matrix-free operator, whose steps are always launched one by one; a second solve starts afresh."""
    system = sy.make_system(12, 4, 3, 3, 40, seed=2, k_scale=0.3)
    basis = sy.sd_basis(12, 4, 3, 3)
    rng = np.random.default_rng(4)
    cand = rng.choice(basis.shape[0], 1300, replace=False).astype(np.uint32)
    vecs = [0.01 * rng.normal(size=1300) for _ in range(5)]
    with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8) as w:
        w.build().set_basis(basis)
        w.update_fock(system.h, system.h)
        for max_iter in (5, 6, 7, 20, 41):
            got = []
            for free in (False, True):
                with nociwick.Pt2(w, cand, -30.0, matrix_free=free) as pt:
                    a = pt.solve(-30.0, *vecs, max_iter=max_iter, restart=restart, res_tol=1e-13)
                    b = pt.solve(-30.0, *vecs, max_iter=max_iter, restart=restart, res_tol=1e-13)
                assert a[1]["iterations"] == b[1]["iterations"]
                got += [a[0], b[0]]
            scale = max(1.0, np.max(np.abs(got[2])))
            for x in got:
                assert np.max(np.abs(x - got[2])) <= 1e-9 * scale
