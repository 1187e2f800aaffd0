"""Repeated preconditioner applications: kernels launched one by one, and from a handle's second call on as one graph."""
import numpy as np
import pytest

from pargemslr_b200 import _abi
from pargemslr_b200 import params as P
from pargemslr_b200 import problems

pytestmark = pytest.mark.gpu


def _handle(precision):
    from pargemslr_b200.handle import GemslrHandle
    p = P.workload_params("lap3d_128")
    A = problems.laplacian(20, 18, 16)
    return GemslrHandle.from_matrix(A, p, precision=precision), p, np.random.default_rng(8)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_graph_repeats_the_direct_launches(precision):
    """The first call launches the kernels, the later ones the graph: the same bits, also between solves of other
    Krylov dimensions, and before and after the wait limit is set (which drops the graph)."""
    h, p, rng = _handle(precision)
    try:
        b = rng.standard_normal((2, h.n))
        fresh = []
        for v in b:  # the first application of a handle each
            other, _, _ = _handle(precision)
            fresh.append(other.apply(v))
            other.close()
        for k in (0, 1, 0, 1):
            np.testing.assert_array_equal(h.apply(b[k]), fresh[k])
        for kdim in (20, 30):
            q = p.copy()
            q[P.SOLVER_KDIM] = kdim
            x, r = h.solve(b[0], params=q)
            assert r["status"] == 0 and r["true_rel_res"] <= 1e-8
            np.testing.assert_array_equal(h.apply(b[1]), fresh[1])
        _abi.check(_abi.lib().pgx_gemslr_set_wait_limit(h._h, 1 << 20))
        for k in (0, 1, 0):
            np.testing.assert_array_equal(h.apply(b[k]), fresh[k])
    finally:
        h.close()


def test_applications_without_device_memory_left():
    """A handle that was applied once goes on being applied where no memory for a graph is left."""
    import torch
    h, _, rng = _handle("fp64")
    keep = []
    try:
        v = torch.from_numpy(rng.standard_normal(h.n)).cuda()
        z = torch.zeros_like(v)
        want = torch.zeros_like(v)
        lib = _abi.lib()
        _abi.check(lib.pgx_gemslr_precond_apply(h._h, want.data_ptr(), v.data_ptr(), _abi.LOCATION_DEVICE))
        size = 16 << 30
        while size >= 1 << 20:
            try:
                keep.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.cuda.OutOfMemoryError:
                size //= 2
        for _ in range(3):
            z.zero_()
            torch.cuda.synchronize()
            _abi.check(lib.pgx_gemslr_precond_apply(h._h, z.data_ptr(), v.data_ptr(), _abi.LOCATION_DEVICE))
            assert torch.equal(z, want)
    finally:
        keep.clear()
        torch.cuda.empty_cache()
        h.close()


def test_a_failed_commit_leaves_nothing_to_solve_with():
    """A handle whose commit was refused answers as one that was never committed, and can be committed again."""
    from pargemslr_b200.handle import import_structures, init
    from pargemslr_b200.structures import GemslrStructures, LevelStructures, empty_csr
    init(0)
    n = 40
    eye = (np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), np.ones(n), n, n)
    rp = np.zeros(n + 1, np.int32)
    rp[8:] = 1  # one entry, in row 7, on the wrong side of the diagonal
    bad = (rp, np.array([9], np.int32), np.ones(1), n, n)

    def structures(L):
        lv = LevelStructures(ncomp=1, dom_ptr=np.array([0, n], np.int32), L=L, U=empty_csr(n, n), dinv=np.ones(n), B=eye)
        return GemslrStructures(n=n, A=eye, pperm=np.arange(n, dtype=np.int32), qperm=None,
                                lev_ptr=np.array([0, n], np.int32), levels=[lv], inner_enable=0)

    lib = _abi.lib()
    h = import_structures(structures(bad), "fp64")
    try:
        assert lib.pgx_gemslr_commit(h) != 0
        v, z = np.ones(n), np.zeros(n)
        assert lib.pgx_gemslr_precond_apply(h, _abi.ptr(z), _abi.ptr(v), _abi.LOCATION_HOST) != 0
        assert b"before commit" in lib.pgx_last_error()
        keep = []
        desc = _abi.Level()
        lv = structures(empty_csr(n, n)).levels[0]
        keep += [np.ascontiguousarray(lv.dom_ptr, np.int32), _abi.doubles(lv.dinv)]
        desc.ncomp, desc.dom_ptr, desc.dinv = 1, _abi.ptr(keep[0]), _abi.ptr(keep[1])
        for name in ("L", "U", "B"):
            setattr(desc, name, _abi.csr_struct(*getattr(lv, name), keep=keep))
        import ctypes as C
        _abi.check(lib.pgx_gemslr_set_level(h, 0, C.byref(desc)))
        _abi.check(lib.pgx_gemslr_commit(h))
        _abi.check(lib.pgx_gemslr_precond_apply(h, _abi.ptr(z), _abi.ptr(v), _abi.LOCATION_HOST))
        np.testing.assert_array_equal(z, v)
    finally:
        lib.pgx_gemslr_destroy(h)
