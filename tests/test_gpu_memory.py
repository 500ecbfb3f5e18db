"""Device memory that a context keeps between calls: given back when another allocation needs it, and no
larger than the work needs."""
import numpy as np
import pytest

import nociwick
from nociwick import synthetic as sy

pytestmark = pytest.mark.gpu


def test_kept_operator_memory_is_given_back():
    """After a candidate operator is gone its matrix and string tables stay with the context; the tables of the
    overlap action still fit where only their memory is left."""
    torch = pytest.importorskip("torch")
    system = sy.make_system(28, 9, 9, 3, 112, seed=2, sigma_h=0.02, sigma_l=0.02, k_scale=0.3, uhf_like=True)
    basis = sy.sd_basis(28, 9, 9, 3)
    nd = basis.shape[0]
    stream = torch.cuda.current_stream().cuda_stream
    x = torch.randn(nd, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    def apply(w):
        y = torch.zeros_like(x)
        w.apply_overlap_device(x.data_ptr(), y.data_ptr(), stream)
        torch.cuda.synchronize()
        return y

    args = (system.s, system.h, system.eri, system.enuc, system.refs)
    with nociwick.WicksShared(*args, tol=1e-8).build().set_basis(basis) as w:
        apply(w.set_basis(basis))   # the kernels and torch's buffers
        w.set_basis(basis)          # drops the tables
        before = free()
        want = apply(w)
        need = before - free()
    with nociwick.WicksShared(*args, tol=1e-8).build().set_basis(basis) as w:
        w.update_fock(system.h, system.h)
        cand = np.random.default_rng(3).choice(nd, 12000, replace=False).astype(np.uint32)
        before = free()
        with nociwick.Pt2(w, cand, -0.5) as pt:
            z = np.zeros(12000)
            pt.solve(0.0, z, z, z, z, np.ones(12000), max_iter=2, restart=2, res_tol=1e-12)
        kept = before - free()
        assert need > kept > 600 << 20
        hog = torch.empty(free() - (need - kept // 2), dtype=torch.uint8, device="cuda")
        try:
            assert free() < need
            got = apply(w)
        finally:
            del hog
            torch.cuda.empty_cache()
    # chunks of a long row are added by atomics, in no fixed order
    assert float((got - want).abs().max()) <= 1e-11 * float(want.abs().max())


def test_build_scratch_beyond_the_fused_transforms():
    """Above 64 orbitals a build takes three tensors a reference pair and a workspace of five (grown by a
    quarter), beside matrices of n^2 and what the driver rounds up; the context's own memory is not counted."""
    torch = pytest.importorskip("torch")
    n = 72
    system = sy.make_system(n, 2, 2, 1, 2 * n, seed=4)
    for _ in range(2):              # the first one loads the kernels
        with nociwick.WicksShared(system.s, system.h, system.eri, system.enuc, system.refs, tol=1e-8) as w:
            torch.cuda.synchronize()
            before = torch.cuda.mem_get_info()[0]
            w.build()
            used = before - torch.cuda.mem_get_info()[0]
    assert used <= 8 * n ** 4 * (3 + 1.25 * 5) + (64 << 20)
