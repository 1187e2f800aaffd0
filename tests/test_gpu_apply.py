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
