"""Four-index tensors of the build (csrc/transform.cu) against the FP64 oracle: every tile count of the
fused half transforms (n = 1 .. 64 in steps of 8 orbitals, with odd and even remainders) and the
quarter-transform route that larger orbital spaces and tensors without the permutation symmetry of
real orbitals take.  Same-parent, mirrored (w, x) and zero-overlap reference pairs are all evaluated.

Tolerance: both builds are FP64 sums of the same terms in other orders.  Elements are of order 10, and each
passes through four sums of n <= 65 terms and two divisions by the singular values: with the smallest non-zero
paired singular value above 0.1, 4 * 65 * 2^-53 * 10 * 10^2 is 3e-11, so 1e-10 Eh holds with room.  Reference
pairs that a forced zero overlap leaves nearly singular (below 0.1) are outside that premise and left out."""
import numpy as np
import pytest

import nociwick
from nociwick import synthetic as sy
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu
ATOL = 1e-10


def _check(system, basis, pairs, convention="exact"):
    orc = Oracle.from_system(system, tol=1e-8, with_mo_cache=False)
    h, s = orc.eval_pairs(orc.oracle_basis(basis), pairs, exact=(convention == "exact"))
    with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8,
                              convention=convention).build() as w:
        w.set_basis(basis)
        hs = w.eval_pairs(pairs)
    oa, ob = system.nocc_a, system.nocc_b
    smin = np.array([[min(v[v > 1e-8].min() for v in (np.linalg.svd(x[k][:, :o].T @ w[k][:, :o], compute_uv=False)
                                                      for k, o in ((0, oa), (2, ob)))) for w in system.refs]
                     for x in system.refs])
    sel = smin[basis["parent"][pairs[:, 0]], basis["parent"][pairs[:, 1]]] >= 0.1
    assert sel.mean() > 0.5
    assert np.max(np.abs(hs[sel, 0] - h[sel])) <= ATOL
    assert np.max(np.abs(hs[sel, 1] - s[sel])) <= ATOL


@pytest.mark.parametrize("n", [4, 7, 8, 9, 16, 17, 23, 24, 25, 32, 33, 40, 41, 48, 55, 56, 57, 63, 64, 65])
def test_every_tile_count(n):
    oa, ob = (1, 2) if n < 8 else (2, 3)
    zero = [(0, 1, 1, 0)] if n in (9, 24, 41, 64) else []
    system = sy.make_system(n, oa, ob, 2 if n > 33 else 3, 2 * n, seed=100 + n, k_scale=0.05, zero_pairs=zero, enuc=0.3)
    basis = sy.sd_basis(n, oa, ob, len(system.refs))
    pairs = sy.sample_pairs(basis, 3000, seed=n, distinct_parents=n % 2 == 0, canonical=False)
    _check(system, basis, pairs)


def test_tensor_without_permutation_symmetry():
    """(mu nu|lam sig) with a part that is not symmetric: the general route, and the oracle's general sums."""
    system = sy.make_system(12, 2, 3, 3, 24, seed=7, k_scale=0.05, zero_pairs=[(0, 1, 1, 0)])
    rng = np.random.default_rng(3)
    system.eri = system.eri + 1e-3 * rng.standard_normal(system.eri.shape)
    basis = sy.sd_basis(12, 2, 3, 3)
    pairs = sy.sample_pairs(basis, 3000, seed=5, distinct_parents=True, canonical=False)
    _check(system, basis, pairs, convention="reference")


def _split_classes():
    """A system and a tolerance between the singular values that the two orders of one reference pair
    compute for the same orbital pair: (1, 0) has no zero-overlap orbital and (0, 1) has one."""
    for seed in range(60):
        system = sy.make_system(10, 3, 3, 2, 24, seed=seed, k_scale=0.3, enuc=0.2)
        (xa, _, xb, _), (wa, _, wb, _) = system.refs
        s = min(np.linalg.svd(x[:, :3].T @ w[:, :3], compute_uv=False)[-1] for x, w in ((xa, wa), (xb, wb)))
        if s < 0.2:
            continue
        for k in range(-12, 13):
            tol = float(s + k * np.spacing(s))
            with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=tol).build() as w:
                m = w.zero_counts().sum(axis=2)
            if (m[1, 0] == 0) != (m[0, 1] == 0):
                if m[1, 0] > 0:
                    system.refs.reverse()
                return system, tol
    raise AssertionError("no pair whose two orders round apart")


def test_orders_of_a_pair_classed_apart():
    """The order without zero-overlap orbitals keeps its own tensors where the other order has some: its
    elements are the exact ones, in a full build and in every block of a blocked evaluation."""
    import torch
    system, tol = _split_classes()
    basis = sy.sd_basis(10, 3, 3, 2)
    per = basis.shape[0] // 2
    rng = np.random.default_rng(2)
    pairs = np.stack([per + rng.integers(0, per, 3000), rng.integers(0, per, 3000)], axis=1).astype(np.uint32)
    orc = Oracle.from_system(system, tol=1e-8, with_mo_cache=False)
    h, s = orc.eval_pairs(orc.oracle_basis(basis), pairs)
    with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=tol).build() as w:
        w.set_basis(basis)
        hs = w.eval_pairs(pairs)
        slab = w.info()["slab_bytes"]
        assert np.max(np.abs(hs[:, 0] - h)) <= ATOL and np.max(np.abs(hs[:, 1] - s)) <= ATOL
        stream = torch.cuda.current_stream().cuda_stream
        dp = torch.from_numpy(pairs.view(np.int32)).cuda()
        out = torch.full((pairs.shape[0], 2), float("nan"), dtype=torch.float64, device="cuda")
        assert w.eval_pairs_blocked(dp.data_ptr(), pairs.shape[0], out.data_ptr(), slab // 2, stream) >= 2
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), hs)
