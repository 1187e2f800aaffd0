"""The SpMV plan made on the device against the host's rule."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_spmv_plan_on_the_device():
    """The variant taken for device arrays is the host plan's: each side of every limit of the rule."""
    import ctypes as C

    import torch

    from pargemslr_b200 import _abi
    from pargemslr_b200.handle import init
    init(0)
    lib = _abi.lib()
    rng = np.random.default_rng(2)
    lens = [[1], [0, 0, 3], [8] * 9 + [9], [8] * 8 + [9] * 2, [16] * 90 + [17] * 10, [16] * 89 + [17] * 11,
            [32] * 900 + [200] * 100, [64] * 9 + [65] * 2, [5] * 990 + [128] * 10, [5] * 990 + [129] * 10,
            [4] * 3000 + [140] * 10, [4] * 3000 + [300] * 5, [200] * 50, [3] * 70000 + [4000] * 2,
            [2] * 3000 + [1500] * 40]
    for ln in lens:
        ln = rng.permutation(np.array(ln))
        n, cols = len(ln), 5000
        rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
        cj = rng.integers(0, cols, rp[-1]).astype(np.int32)
        va = rng.standard_normal(rp[-1])
        x = rng.standard_normal(cols)
        dev = [torch.from_numpy(a).cuda() for a in (rp, cj, va)]
        xd = torch.from_numpy(x).cuda()
        host = _abi.Csr(n, cols, len(cj), rp.ctypes.data, cj.ctypes.data, va.ctypes.data)
        dcsr = _abi.Csr(n, cols, len(cj), *[t.data_ptr() for t in dev])
        lanes, merge = C.c_int32(), C.c_int32()
        _abi.check(lib.pgx_csr_spmv_plan(C.byref(host), C.byref(lanes), C.byref(merge)))
        y = [torch.full((n,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(3)]
        for k in range(3):
            _abi.check(lib.pgx_csr_spmv_device_variant(C.byref(dcsr), k, 1.0, xd.data_ptr(), 0.0, y[k].data_ptr()))
        assert torch.equal(y[0], y[2 if merge.value else 1]), ln[:20]
        ref = np.bincount(np.repeat(np.arange(n), ln), weights=va * x[cj], minlength=n)
        mag = np.bincount(np.repeat(np.arange(n), ln), weights=np.abs(va * x[cj]), minlength=n)
        for k in (1, 2):
            assert np.all(np.abs(y[k].cpu().numpy() - ref) <= 4000 * 2.3e-16 * mag)


@pytest.mark.parametrize("rows", [1023, 1024, 1025, 3000])
def test_plan_on_both_sides_of_the_rows_planned_on_the_host(rows):
    """Matrices around the row count up to which the host chooses: the variant is the same rule's on either side."""
    import ctypes as C

    import torch

    from pargemslr_b200 import _abi
    from pargemslr_b200.handle import init
    init(0)
    lib = _abi.lib()
    rng = np.random.default_rng(rows)
    cols = 5000
    for ln in ([1], [0, 0, 3], [8] * 9 + [9], [8] * 8 + [9] * 2, [16] * 89 + [17] * 11, [32] * 90 + [200] * 10,
               [5] * 90 + [128], [5] * 90 + [129], [2] * 70 + [1500]):
        ln = rng.permutation(np.resize(np.array(ln), rows))
        rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
        cj = rng.integers(0, cols, rp[-1]).astype(np.int32)
        va = rng.standard_normal(rp[-1])
        x, y0 = rng.standard_normal(cols), rng.standard_normal(rows)
        dev = [torch.from_numpy(a).cuda() for a in (rp, cj, va)]
        xd = torch.from_numpy(x).cuda()
        host = _abi.Csr(rows, cols, len(cj), rp.ctypes.data, cj.ctypes.data, va.ctypes.data)
        dcsr = _abi.Csr(rows, cols, len(cj), *[t.data_ptr() for t in dev])
        lanes, merge = C.c_int32(), C.c_int32()
        _abi.check(lib.pgx_csr_spmv_plan(C.byref(host), C.byref(lanes), C.byref(merge)))
        y = [torch.from_numpy(y0).cuda() for _ in range(3)]
        for k in range(3):
            _abi.check(lib.pgx_csr_spmv_device_variant(C.byref(dcsr), k, 2.0, xd.data_ptr(), 0.5, y[k].data_ptr()))
        assert torch.equal(y[0], y[2 if merge.value else 1]), ln[:20]
        ref = 2.0 * np.bincount(np.repeat(np.arange(rows), ln), weights=va * x[cj], minlength=rows) + 0.5 * y0
        mag = 2.0 * np.bincount(np.repeat(np.arange(rows), ln), weights=np.abs(va * x[cj]), minlength=rows) + np.abs(y0)
        for k in (1, 2):
            assert np.all(np.abs(y[k].cpu().numpy() - ref) <= 4000 * 2.3e-16 * mag)
