"""One-kernel pair evaluation (small requests; every (F, S) request without zero-overlap reference pairs)
against the sorted pipeline, which serial class timing selects, and the oracle.

Both routes evaluate the same expressions in FP64; the compiler may contract them differently, so they
agree to a few roundings of the largest term of an element (1e-12 here: terms of at most about 1e2 for
these systems, 2^-53 each, a few tens of them), and the oracle to the tolerance of the other parity tests.
"""
import numpy as np
import pytest

import nociwick
from nociwick import synthetic as sy
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu
ROUTES = 1e-12
ATOL = 1e-9


def _both(w, torch, pairs, fs):
    stream = torch.cuda.current_stream().cuda_stream
    dp = torch.from_numpy(np.ascontiguousarray(pairs.astype(np.uint32)).view(np.int32)).cuda()
    call = w.eval_fs_pairs_device if fs else w.eval_pairs_device
    outs = []
    for serial in (False, True):
        w.set_timing(serial, serial_classes=serial)
        out = torch.full((pairs.shape[0], 2), float("nan"), dtype=torch.float64, device="cuda")
        call(dp.data_ptr(), pairs.shape[0], out.data_ptr(), stream)
        w.sync(stream)
        outs.append(out.cpu().numpy())
    w.set_timing(False)
    return outs


@pytest.mark.parametrize("zero_pairs", [[], [(0, 1, 1, 0)], [(0, 1, 0, 2), (1, 2, 1, 1)]])
@pytest.mark.parametrize("fs", [False, True])
def test_routes_agree(zero_pairs, fs):
    """Ranks up to 8 per spin (the runtime path), same-parent pairs beyond doubles, tile and warp edges."""
    torch = pytest.importorskip("torch")
    system = sy.make_system(8, 3, 3, 3, 20, seed=1, k_scale=0.3, zero_pairs=zero_pairs, enuc=0.37)
    basis = sy.sd_basis(8, 3, 3, 3, orders=(1, 2, 3, 4))
    rng = np.random.default_rng(3)
    fock = []
    for _ in range(2):
        a = rng.normal(0.0, 0.3, (8, 8))
        fock.append(system.h + 0.5 * (a + a.T))
    orc = Oracle.from_system(system, tol=1e-8)
    orc.set_fock(*fock)
    ob = orc.oracle_basis(basis)
    with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8) as w:
        w.build().set_basis(basis)
        w.update_fock(*fock)
        for n in (1, 31, 33, 148 * 32 + 1, 20000, 131072, 131073, 148 * 1024 + 7, 393216, 393217):
            pairs = sy.sample_pairs(basis, n, seed=n, distinct_parents=False)
            one, srt = _both(w, torch, pairs, fs)
            assert np.all(np.isfinite(one)) and np.max(np.abs(one - srt)) <= ROUTES, n
            k = min(n, 2000)
            if fs:
                _, h_ref, s_ref = orc.eval_m_pairs(ob, pairs[-k:], 0.0)
            else:
                h_ref, s_ref = orc.eval_pairs(ob, pairs[-k:])
            assert np.max(np.abs(one[-k:, 0] - h_ref)) <= ATOL and np.max(np.abs(one[-k:, 1] - s_ref)) <= ATOL, n


@pytest.mark.parametrize("fs", [False, True])
def test_out_of_range_and_one_class(fs):
    """An index beyond the basis gives NaN and the error, its neighbours their values; a request of one
    determinant pair repeated fills every tile with one class."""
    torch = pytest.importorskip("torch")
    system = sy.make_system(10, 3, 3, 3, 24, seed=7, k_scale=0.3, enuc=0.5)
    basis = sy.sd_basis(10, 3, 3, 3)
    per = basis.shape[0] // 3
    with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8) as w:
        w.build().set_basis(basis)
        w.update_fock(system.h, system.h)
        pairs = np.tile(np.array([[per - 1, 2 * per - 1]]), (3000, 1))
        one, srt = _both(w, torch, pairs, fs)
        assert np.max(np.abs(one - srt)) <= ROUTES and np.all(one == one[0])
        pairs[1234, 1] = basis.shape[0]
        stream = torch.cuda.current_stream().cuda_stream
        dp = torch.from_numpy(pairs.astype(np.uint32).view(np.int32)).cuda()
        out = torch.zeros((3000, 2), dtype=torch.float64, device="cuda")
        (w.eval_fs_pairs_device if fs else w.eval_pairs_device)(dp.data_ptr(), 3000, out.data_ptr(), stream)
        with pytest.raises(nociwick.NwError):
            w.sync(stream)
        got = out.cpu().numpy()
        assert np.all(np.isnan(got[1234])) and np.array_equal(np.delete(got, 1234, 0), np.delete(one, 1234, 0))


@pytest.mark.parametrize("zero_pairs", [[], [(0, 1, 1, 0)]])
def test_pinned_host_chunks(zero_pairs):
    """Pinned host buffers around the smallest pipelined request, chunks of whole and ragged size."""
    torch = pytest.importorskip("torch")
    system = sy.make_system(10, 3, 3, 3, 24, seed=7, k_scale=0.3, enuc=0.5, zero_pairs=zero_pairs)
    basis = sy.sd_basis(10, 3, 3, 3)
    with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8) as w:
        w.build().set_basis(basis)
        for n in ((1 << 17) - 1, 1 << 17, 200_001, 393_216, 393_217, 600_001):
            pairs = sy.sample_pairs(basis, n, seed=n, distinct_parents=False)
            host = torch.from_numpy(pairs.astype(np.uint32).view(np.int32)).pin_memory()
            out = torch.full((n, 2), float("nan"), dtype=torch.float64).pin_memory()
            w.eval_pairs(host.numpy().view(np.uint32), out.numpy())
            assert np.max(np.abs(out.numpy() - _both(w, torch, pairs, False)[0])) <= ROUTES, n


@pytest.mark.parametrize("n,nref,limit", [(8, 3, 393216), (16, 8, 303104), (16, 17, 131072), (41, 2, 131072)])
def test_route_by_references(n, nref, limit):
    """Both sides of every line of the (H, S) size rule: the largest one-kernel request agrees with the sorted
    pipeline, and one pair more is the sorted pipeline's own result, bit for bit."""
    torch = pytest.importorskip("torch")
    system = sy.make_system(n, 2, 2, nref, 2 * n, seed=3, k_scale=0.05, enuc=0.2)
    basis = sy.sd_basis(n, 2, 2, nref)
    with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8) as w:
        w.build().set_basis(basis)
        pairs = sy.sample_pairs(basis, limit + 1, seed=n, distinct_parents=False)
        one, srt = _both(w, torch, pairs[:limit], False)
        assert np.all(np.isfinite(one)) and np.max(np.abs(one - srt)) <= ROUTES
        one, srt = _both(w, torch, pairs, False)
        assert np.array_equal(one, srt)


def test_autotune_small_request():
    """The tuner's settings are the sorted pipeline's: on a request that the one kernel takes, a budget that only
    clears and scans more counters (2^22 or 2^23 for 1000 pairs: 27 MB at these 6.7 10^6 keys, against 64 KB) is
    never the fastest, and the results are the request's own."""
    torch = pytest.importorskip("torch")
    system = sy.make_system(40, 4, 4, 3, 80, seed=3, k_scale=0.05)
    basis = sy.sd_basis(40, 4, 4, 3)
    pairs = sy.sample_pairs(basis, 1000, seed=1, distinct_parents=False)
    with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8) as w:
        w.build().set_basis(basis)
        one, _ = _both(w, torch, pairs, False)
        stream = torch.cuda.current_stream().cuda_stream
        dp = torch.from_numpy(np.ascontiguousarray(pairs.astype(np.uint32)).view(np.int32)).cuda()
        for _ in range(8):
            out = torch.full((1000, 2), float("nan"), dtype=torch.float64, device="cuda")
            rep = w.autotune(dp.data_ptr(), 1000, out.data_ptr(), stream)
            assert rep["trials"] == 19 and rep["key_budget"] < 1 << 22
            assert np.array_equal(out.cpu().numpy(), one)


@pytest.mark.parametrize("fs", [False, True])
def test_blocks_of_a_matrix_take_one_route(fs):
    """A dense matrix in row blocks of 2^24 pairs, the last one small: every element as the device call gives it
    for all pairs at once, bit for bit, with zero-overlap reference pairs."""
    torch = pytest.importorskip("torch")
    system = sy.make_system(8, 3, 3, 3, 20, seed=1, k_scale=0.3, zero_pairs=[(0, 1, 1, 0)], enuc=0.37)
    basis = sy.sd_basis(8, 3, 3, 3)
    rng = np.random.default_rng(3)
    left, right = (rng.integers(0, basis.shape[0], 4100).astype(np.uint32) for _ in range(2))
    with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8) as w:
        w.build().set_basis(basis)
        w.update_fock(system.h, system.h)
        got = (w.build_fs_matrix if fs else w.build_hs_matrix)(left, right, symmetric=False)
        pairs = np.stack([np.repeat(left, 4100), np.tile(right, 4100)], axis=1)
        dp = torch.from_numpy(pairs.view(np.int32)).cuda()
        out = torch.empty((pairs.shape[0], 2), dtype=torch.float64, device="cuda")
        stream = torch.cuda.current_stream().cuda_stream
        (w.eval_fs_pairs_device if fs else w.eval_pairs_device)(dp.data_ptr(), pairs.shape[0], out.data_ptr(), stream)
        w.sync(stream)
        want = out.cpu().numpy().reshape(4100, 4100, 2)
    assert np.array_equal(got[0], want[:, :, 0]) and np.array_equal(got[1], want[:, :, 1])


def test_one_reference_pair_among_many():
    """A request for one reference pair in a context of many keeps the one kernel where pairs of all references are
    sorted: both give the same elements."""
    torch = pytest.importorskip("torch")
    system = sy.make_system(16, 2, 2, 20, 32, seed=3, k_scale=0.05, enuc=0.2)
    basis = sy.sd_basis(16, 2, 2, 20)
    per = basis.shape[0] // 20
    rng = np.random.default_rng(7)
    i, j = 3 * per + rng.integers(0, per, 140000), 11 * per + rng.integers(0, per, 140000)
    exc = nociwick.lib.exc_caches(basis)
    with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8) as w:
        w.build().set_basis(basis)
        got = w.eval_batched(3, 11, exc[i], exc[j], basis["phase"][i] * basis["phase"][j])
        want = _both(w, torch, np.stack([i, j], axis=1), False)[1]
    assert np.all(np.isfinite(got)) and np.max(np.abs(got - want)) <= ROUTES
