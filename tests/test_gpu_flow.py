"""The per-subdomain triangular solve at the edges of its tasks, groups and ring, against plain substitution."""
import numpy as np
import pytest

from pargemslr_b200.structures import GemslrStructures, LevelStructures, empty_csr

pytestmark = pytest.mark.gpu


def _factors(dom, deg, back, seed, cplx, longrow=0):
    """A random factor pair, block diagonal over `dom`: up to `deg` entries a row, at most `back` rows away."""
    rng = np.random.default_rng(seed)
    n = dom[-1]
    out = []
    for up in (False, True):
        rp, cj = [0], []
        for a, e in zip(dom[:-1], dom[1:]):
            for i in range(a, e):
                room = e - 1 - i if up else i - a
                want = min(room, longrow if longrow and i % 97 == 96 else int(rng.integers(0, deg + 1)))
                d = np.unique(1 + rng.integers(0, min(room, max(back, want)), want)) if want else np.zeros(0, np.int64)
                cj.append(np.sort(i + d if up else i - d))
                rp.append(rp[-1] + len(d))
        cj = np.concatenate(cj).astype(np.int32)
        rp = np.array(rp, np.int32)
        va = rng.uniform(-1, 1, len(cj)) / (1.0 + np.repeat(np.diff(rp), np.diff(rp)))
        if cplx:
            va = va + 1j * rng.uniform(-1, 1, len(cj)) / 4
        out.append((rp, cj, va, n, n))
    return out[0], out[1], 1.0 + 0.2 * rng.uniform(-1, 1, n) + (0.1j if cplx else 0.0)


def _substitute(L, U, dinv, b):
    y = b.astype(np.result_type(b, dinv))
    for M, up in ((L, False), (U, True)):
        rp, cj, va = M[:3]
        for i in (range(len(b) - 1, -1, -1) if up else range(len(b))):
            y[i] -= va[rp[i]:rp[i + 1]] @ y[cj[rp[i]:rp[i + 1]]]
            if up:
                y[i] *= dinv[i]
    return y


CASES = {
    "one row": ([0, 1], 0, 1, 0),
    "a task and a row": ([0, 33], 3, 20, 0),
    "diagonal": ([0, 1300], 0, 1, 0),
    "chains": ([0, 400], 1, 1, 0),
    "a row a level": ([0, 300], 3, 2, 0),
    "two narrow subdomains and an empty one": ([0, 517, 517, 900], 6, 40, 0),
    "long rows": ([0, 2500], 6, 150, 90),
    "ring wraps": ([0, 20000], 4, 30, 0),
    "operands older than the ring": ([0, 24000], 4, 9000, 0),
}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("cplx", [False, True], ids=["real", "complex"])
@pytest.mark.parametrize("name", CASES)
def test_pass_pair(name, cplx, precision):
    from pargemslr_b200.handle import GemslrHandle
    dom, deg, back, longrow = CASES[name]
    L, U, dinv = _factors(dom, deg, back, len(name), cplx, longrow)
    n = dom[-1]
    eye = (np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), np.ones(n, dinv.dtype), n, n)
    lv = LevelStructures(ncomp=len(dom) - 1, dom_ptr=np.array(dom, np.int32), L=L, U=U, dinv=dinv, B=eye)
    st = GemslrStructures(n=n, A=eye, pperm=np.arange(n, dtype=np.int32), qperm=None,
                          lev_ptr=np.array([0, n], np.int32), levels=[lv], inner_enable=0)
    rng = np.random.default_rng(1)
    b = rng.standard_normal(n) + (1j * rng.standard_normal(n) if cplx else 0.0)
    h = GemslrHandle(st, precision=precision)
    try:
        if name in ("one row", "diagonal"):
            assert "product of the inverses" in h.describe()
        elif name not in ("a task and a row", "chains"):  # those are about as deep as the limit
            assert "dataflow" in h.describe()
        z = h.apply(b)
    finally:
        h.close()
    ref = _substitute(L, U, dinv, b)
    # |x| stays of order |b| (row sums of the factors are below 1): rounding of 90 products a row at most
    tol = 1e-13 if precision == "fp64" else 2e-5
    assert np.linalg.norm(z - ref) <= tol * np.linalg.norm(ref)


def _one_level(dom, L, U, dinv):
    n = dom[-1]
    eye = (np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), np.ones(n, dinv.dtype), n, n)
    lv = LevelStructures(ncomp=len(dom) - 1, dom_ptr=np.array(dom, np.int32), L=L, U=U, dinv=dinv, B=eye)
    return GemslrStructures(n=n, A=eye, pperm=np.arange(n, dtype=np.int32), qperm=None,
                            lev_ptr=np.array([0, n], np.int32), levels=[lv], inner_enable=0)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("cplx", [False, True], ids=["real", "complex"])
@pytest.mark.parametrize("name", [k for k in CASES if k not in ("one row", "diagonal")])
def test_lanes_repeat_the_single_lane(name, cplx, precision):
    """The same solves through slots of one, two and four lanes: the same results bit for bit, on every pass."""
    from pargemslr_b200 import params as P
    from pargemslr_b200.handle import GemslrHandle
    dom, deg, back, longrow = CASES[name]
    if name in ("a task and a row", "chains"):
        deg, back = 3, 2  # one row a level: well above the depth of one product
    L, U, dinv = _factors(dom, deg, back, len(name), cplx, longrow)
    n = dom[-1]
    rng = np.random.default_rng(2)
    B = rng.standard_normal((4, n)) + (1j * rng.standard_normal((4, n)) if cplx else 0.0)
    p = P.workload_params("lap2d_256")
    h = GemslrHandle(_one_level(dom, L, U, dinv), precision=precision)
    try:
        assert "dataflow" in h.describe()
        want = [h.solve(b, params=p)[0] for b in B]
        for lanes in (2, 4):
            h.set_lanes(lanes)
            h.set_slots(1 + 4 // lanes)
            for _ in range(2):
                X, R = h.solve_batch(B, params=p)
                assert all(r["status"] == 0 for r in R)
                for k in range(4):
                    np.testing.assert_array_equal(X[k], want[k])
    finally:
        h.close()


@pytest.mark.parametrize("levels", [2, 7, 8, 9])
@pytest.mark.parametrize("cplx", [False, True], ids=["real", "complex"])
def test_shallow_factors(levels, cplx):
    """Factors on both sides of the depth at which one product takes the place of the two passes."""
    from pargemslr_b200.handle import GemslrHandle
    n, seps = 999, 999 // levels
    rng = np.random.default_rng(levels)
    rp = np.zeros(n + 1, np.int32)
    coupled = np.arange(n) % seps == 3  # a few chains of `levels` rows
    rows = np.flatnonzero(coupled)[1:levels]
    rp[rows + 1] = 1
    rp = np.cumsum(rp).astype(np.int32)
    cj = (rows - seps).astype(np.int32)
    va = rng.uniform(-1, 1, len(rows)) + (1j * rng.uniform(-1, 1, len(rows)) if cplx else 0.0)
    L = (rp, cj, va, n, n)
    up = np.zeros(n + 1, np.int32)
    up[cj + 1] = 1
    U = (np.cumsum(up).astype(np.int32), rows.astype(np.int32), va[::-1].copy(), n, n)
    dinv = 1.0 + rng.random(n) + (0.3j if cplx else 0.0)
    eye = (np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), np.ones(n, dinv.dtype), n, n)
    lv = LevelStructures(ncomp=1, dom_ptr=np.array([0, n], np.int32), L=L, U=U, dinv=dinv, B=eye)
    st = GemslrStructures(n=n, A=eye, pperm=np.arange(n, dtype=np.int32), qperm=None,
                          lev_ptr=np.array([0, n], np.int32), levels=[lv], inner_enable=0)
    b = rng.standard_normal(n) + (1j * rng.standard_normal(n) if cplx else 0.0)
    h = GemslrHandle(st, precision="fp64")
    try:
        assert ("product of the inverses" in h.describe()) == (levels <= 8)
        z = h.apply(b)
    finally:
        h.close()
    ref = _substitute(L, U, dinv, b)
    assert np.linalg.norm(z - ref) <= 1e-14 * np.linalg.norm(ref)


@pytest.mark.parametrize("size", [0.5, 300.0, 1e12])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_shallow_factors_that_grow_keep_their_passes(size, precision):
    """Five levels of large multipliers: the product of the inverses would hold entries of size^4 times those of D^-1
    (at 1e12 beyond a float's range), and results that need none of them would be lost."""
    from pargemslr_b200.handle import GemslrHandle
    n, step = 1000, 200  # five rows a chain
    rows = np.arange(step, n)
    rp = np.concatenate([np.zeros(step, np.int32), np.arange(n - step + 1, dtype=np.int32)])
    up = np.concatenate([np.arange(n - step + 1, dtype=np.int32), np.full(step, n - step, np.int32)])
    rng = np.random.default_rng(7)
    L = (rp, (rows - step).astype(np.int32), size * rng.uniform(0.5, 1, n - step), n, n)
    U = (up, rows.astype(np.int32), size * rng.uniform(0.5, 1, n - step), n, n)
    dinv = 1.0 + rng.random(n)
    b = rng.standard_normal(n)
    b[:600] = 0.0  # what is left reaches two levels on
    b[600:] *= 1e-9 if size > 1e6 else 1.0
    h = GemslrHandle(_one_level([0, n], L, U, dinv), precision=precision)
    try:
        assert ("product of the inverses" in h.describe()) == (size < 1)
        z = h.apply(b)
    finally:
        h.close()
    kind = np.float64 if precision == "fp64" else np.float32
    y = b.astype(kind)
    for i in range(step, n):
        y[i] -= kind(L[2][i - step]) * y[i - step]
    y *= dinv.astype(kind)
    with np.errstate(over="ignore"):  # the rows that leave a float's range are not looked at
        for i in range(n - step - 1, -1, -1):
            y[i] -= kind(dinv[i]) * kind(U[2][i]) * y[i + step]
    fin = np.isfinite(y)
    assert fin[600:].all()
    # two steps each way, a few roundings each, in either order
    tol = 1e-14 if precision == "fp64" else 5e-6
    for a in (600, 800):
        assert np.linalg.norm(z[a:a + step] - y[a:a + step]) <= tol * np.linalg.norm(y[a:a + step].astype(np.float64))


@pytest.mark.parametrize("bad", ["L", "U"])
def test_factor_that_is_not_triangular_is_refused(bad):
    from pargemslr_b200 import _abi
    from pargemslr_b200.handle import GemslrHandle
    n = 40
    eye = (np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), np.ones(n), n, n)
    lv = LevelStructures(ncomp=1, dom_ptr=np.array([0, n], np.int32), L=empty_csr(n, n), U=empty_csr(n, n),
                         dinv=np.ones(n), B=eye)
    rp = np.zeros(n + 1, np.int32)
    rp[8:] = 1  # one entry, in row 7
    setattr(lv, bad, (rp, np.array([9 if bad == "L" else 5], np.int32), np.ones(1), n, n))
    st = GemslrStructures(n=n, A=eye, pperm=np.arange(n, dtype=np.int32), qperm=None,
                          lev_ptr=np.array([0, n], np.int32), levels=[lv], inner_enable=0)
    with pytest.raises(_abi.PgxError, match="triangular"):
        GemslrHandle(st, precision="fp64").close()


def _many_far(n, deg):
    """One subdomain, about `deg` entries a row anywhere before (after) it: levels of hundreds of rows."""
    rng = np.random.default_rng(n)
    out = []
    for up in (False, True):
        rows = np.repeat(np.arange(n, dtype=np.int64), deg)
        cols = rng.integers(0, n, rows.size)
        keep = cols > rows if up else cols < rows
        key = np.unique(rows[keep] * n + cols[keep])
        rp = np.concatenate([[0], np.cumsum(np.bincount(key // n, minlength=n))]).astype(np.int32)
        out.append((rp, (key % n).astype(np.int32), rng.uniform(-1, 1, key.size) / deg, n, n))
    return out[0], out[1], 1.0 + 0.2 * rng.uniform(-1, 1, n)


@pytest.mark.parametrize("n,kernel", [(40000, "dataflow"), (90000, "segmented")])
def test_factors_of_mostly_far_operands(n, kernel):
    """On both sides of the number of far operands from which a subdomain leaves one SM; lanes follow their handle."""
    from pargemslr_b200 import params as P
    from pargemslr_b200.handle import GemslrHandle
    L, U, dinv = _many_far(n, 40)
    h = GemslrHandle(_one_level([0, n], L, U, dinv), precision="mixed")
    try:
        assert h.describe().count(kernel) >= 2  # the lower and the upper factor
        B = np.random.default_rng(4).standard_normal((4, n))
        ref = _substitute(L, U, dinv, B[0])
        assert np.linalg.norm(h.apply(B[0]) - ref) <= 2e-5 * np.linalg.norm(ref)
        p = P.workload_params("serve")
        want = [h.solve(b, params=p)[0] for b in B]
        h.set_lanes(4)
        h.set_slots(2)
        X, _ = h.solve_batch(B, params=p)
        for k in range(4):
            np.testing.assert_array_equal(X[k], want[k])
    finally:
        h.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("cplx", [False, True], ids=["real", "complex"])
@pytest.mark.parametrize("name", ["two narrow subdomains and an empty one", "long rows", "operands older than the ring"])
def test_infinities_and_nan_pass_through(name, cplx, precision):
    """A result that is not finite is a result: rows that depend on it are not finite either, in class as plain
    substitution has them (real values), and all others are as without it."""
    from pargemslr_b200.handle import GemslrHandle
    dom, deg, back, longrow = CASES[name]
    L, U, dinv = _factors(dom, deg, back, len(name), cplx, longrow)
    n = dom[-1]
    h = GemslrHandle(_one_level(dom, L, U, dinv), precision=precision)
    try:
        assert "dataflow" in h.describe()
        b = np.random.default_rng(3).standard_normal(n) + (1j if cplx else 0.0)
        import torch
        for bad in (np.inf, -np.inf, np.nan):
            for at in (n - 2, n // 2):  # reaches few rows, and many
                v = b.copy()
                v[at] = bad
                with np.errstate(all="ignore"):
                    ref = _substitute(L, U, dinv, v)
                vd = torch.from_numpy(v).cuda()
                zd = torch.zeros_like(vd)
                from pargemslr_b200 import _abi
                _abi.check(_abi.lib().pgx_gemslr_precond_apply(h._h, zd.data_ptr(), vd.data_ptr(), _abi.LOCATION_DEVICE))
                z = zd.cpu().numpy()
                fin = np.isfinite(ref)
                assert fin.any() and not fin.all()
                np.testing.assert_array_equal(np.isfinite(z), fin)
                if not cplx:
                    np.testing.assert_array_equal(np.isnan(z), np.isnan(ref))
                    np.testing.assert_array_equal(np.sign(z[np.isinf(z)]), np.sign(ref[np.isinf(ref)]))
                tol = 1e-13 if precision == "fp64" else 2e-5
                assert np.linalg.norm(z[fin] - ref[fin]) <= tol * np.linalg.norm(ref[fin])
    finally:
        h.close()
