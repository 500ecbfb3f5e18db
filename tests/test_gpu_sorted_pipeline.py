"""The sorted pipeline at sizes beyond the one-kernel evaluation's (393216 pairs for these systems, 131072 with
zero-overlap reference pairs): its own settings, work counter, sub-buckets and skip keys."""
import numpy as np
import pytest

import nociwick
from nociwick import synthetic as sy

pytestmark = pytest.mark.gpu


def _device(w, torch, pairs, call):
    stream = torch.cuda.current_stream().cuda_stream
    dp = torch.from_numpy(np.ascontiguousarray(pairs.astype(np.uint32)).view(np.int32)).cuda()
    out = torch.full((pairs.shape[0], 2), float("nan"), dtype=torch.float64, device="cuda")
    call(dp.data_ptr(), pairs.shape[0], out.data_ptr(), stream)
    w.sync(stream)
    return out.cpu().numpy()


@pytest.mark.parametrize("zero_pairs,npairs", [([], 393217), ([], 600001), ([(0, 1, 1, 0)], 131073)])
def test_tuned_settings_keep_every_bit(zero_pairs, npairs):
    torch = pytest.importorskip("torch")
    system = sy.make_system(14, 3, 3, 3, 28, seed=5, k_scale=0.2, zero_pairs=zero_pairs, enuc=0.2)
    basis = sy.sd_basis(14, 3, 3, 3)
    pairs = sy.sample_pairs(basis, npairs, seed=13, distinct_parents=False)
    with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8) as w:
        w.build().set_basis(basis)
        before = _device(w, torch, pairs, w.eval_pairs_device)
        rep = {}

        def tune(pp, n, op, stream):
            rep.update(w.autotune(pp, n, op, stream))

        tuned = _device(w, torch, pairs, tune)
        after = _device(w, torch, pairs, w.eval_pairs_device)
    assert rep["trials"] == 19
    assert np.array_equal(before, tuned) and np.array_equal(before, after)


@pytest.mark.parametrize("fs", [False, True])
def test_zero_overlap_pairs_at_any_position(fs):
    """Ranks up to 8 per spin in the m > 0 evaluators: the same bits in a permuted request and a shorter one."""
    torch = pytest.importorskip("torch")
    system = sy.make_system(8, 3, 3, 3, 20, seed=4, k_scale=0.3, zero_pairs=[(0, 1, 1, 0), (1, 2, 0, 2)])
    basis = sy.sd_basis(8, 3, 3, 3, orders=(1, 2, 3, 4))
    pairs = sy.sample_pairs(basis, 200000, seed=21)
    perm = np.random.default_rng(5).permutation(pairs.shape[0])
    with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8) as w:
        w.build().set_basis(basis)
        w.update_fock(system.h, system.h)
        call = w.eval_fs_pairs_device if fs else w.eval_pairs_device
        first = _device(w, torch, pairs, call)
        assert np.all(np.isfinite(first))
        assert np.array_equal(first, _device(w, torch, pairs, call))
        assert np.array_equal(first[perm], _device(w, torch, pairs[perm], call))
        assert np.array_equal(first[:131073], _device(w, torch, pairs[:131073], call))


@pytest.mark.parametrize("npairs", [131072, 131073, 300000])
def test_blocked_evaluation_on_both_sides_of_the_limit(npairs):
    torch = pytest.importorskip("torch")
    system = sy.make_system(12, 3, 3, 3, 24, seed=5, k_scale=0.3, zero_pairs=[(0, 1, 1, 0)], enuc=0.2)
    basis = sy.sd_basis(12, 3, 3, 3, orders=(1, 2, 3))
    pairs = sy.sample_pairs(basis, npairs, seed=8, distinct_parents=False)
    with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8).build() as w:
        w.set_basis(basis)
        full = _device(w, torch, pairs, w.eval_pairs_device)
        slab = w.info()["slab_bytes"]
        nb = []

        def blocked(pp, n, op, stream):
            nb.append(w.eval_pairs_blocked(pp, n, op, slab // 3, stream))

        got = _device(w, torch, pairs, blocked)
    assert nb[0] >= 3 and np.array_equal(got, full)
