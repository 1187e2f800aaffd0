"""The measured cases: what a program of this library has the GPU do, through its public entry points.

Every case is a dict of plain values; `kind` says which entry point it calls:

  spmv      pgx_csr_spmv_device on device arrays: y = A x
  apply     pgx_gemslr_precond_apply on device vectors, the preconditioner set up by GemslrHandle.from_matrix
  imported  the same call on a handle imported level by level (GemslrHandle of GemslrStructures): block ILU(0) on slabs,
            separator planes as the second level, a low-rank correction
  solve     GemslrHandle.solve_device: one GeMSLR-preconditioned FGMRES solve
  batch     GemslrHandle.solve_batch_ptr: many right-hand sides over multi-lane slots
  block     the same call with one 16-lane slot of a complex handle (imported)
  systems   SystemsBatch.solve_ptrs: many systems of uneven sizes in one launch

Parameter sets are the library's named workloads; the right-hand sides are b = A x with x = 2u - 1 from the seed.
"""
import math

import numpy as np
import torch

from pargemslr_b200 import _abi
from pargemslr_b200 import params as P
from pargemslr_b200 import problems
from pargemslr_b200.handle import GemslrHandle, init
from pargemslr_b200.structures import GemslrStructures, LevelStructures
from pargemslr_b200.systems import SystemsBatch

SHIFT = 0.05 + 0.01j  # of the complex workload


def listed():
    return [
        # the smallest product: the 2D grid of the first configuration
        {"name": "spmv_lap2d_256", "kind": "spmv", "matrix": "lap", "nx": 256, "ny": 256, "nz": 1},
        # the product of every Krylov step of the headline grid
        {"name": "spmv_lap3d_128", "kind": "spmv", "matrix": "lap", "nx": 128, "ny": 128, "nz": 128},
        # a few long rows among many short ones: the merge-path product
        {"name": "spmv_skewed_60k", "kind": "spmv", "matrix": "skewed", "n": 60000},
        # the smallest preconditioner call, where launches and latency count
        {"name": "apply_lap2d_64_fp64", "kind": "apply", "workload": "lap2d_256", "nx": 64, "ny": 64, "nz": 1,
         "precision": "fp64"},
        # a preconditioner call inside a caller's own Krylov method, on a 3D problem
        {"name": "apply_lap3d_48_mixed", "kind": "apply", "workload": "lap3d_128", "nx": 48, "ny": 48, "nz": 48,
         "precision": "mixed"},
        # a preconditioner that another code set up, ragged sizes, full precision
        {"name": "imported_61x55x64_fp64", "kind": "imported", "nx": 61, "ny": 55, "nz": 64, "slabs": 6, "rank": 16,
         "precision": "fp64"},
        # the first configuration as a whole: one solve in full precision
        {"name": "solve_lap2d_256_fp64", "kind": "solve", "workload": "lap2d_256", "nx": 256, "ny": 256, "nz": 1,
         "precision": "fp64"},
        # one right-hand side at a time on a 3D grid, mixed precision
        {"name": "solve_lap3d_64_mixed", "kind": "solve", "workload": "lap3d_128", "nx": 64, "ny": 64, "nz": 64,
         "precision": "mixed"},
        # a served matrix: random, nonsymmetric, one request
        {"name": "solve_random_60k_mixed", "kind": "solve", "workload": "serve", "nx": 60000, "ny": 1, "nz": 1,
         "precision": "mixed"},
        # throughput: the headline's four-lane slots, 24 right-hand sides at once
        {"name": "batch_lap3d_48_mixed", "kind": "batch", "workload": "lap3d_128", "nx": 48, "ny": 48, "nz": 48,
         "precision": "mixed", "nrhs": 24, "lanes": 4},
        # the complex configuration: 16 right-hand sides as one block
        {"name": "block_complex_24_mixed", "kind": "block", "nx": 24, "ny": 24, "nz": 24, "slabs": 4, "rank": 32,
         "precision": "mixed", "nrhs": 16},
        # uneven convection-diffusion systems in one launch
        {"name": "systems_convdiff_40", "kind": "systems", "count": 40, "edge_min": 32, "edge_max": 112,
         "precision": "mixed"},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "apply", "apply", "imported", "imported", "solve", "solve", "batch", "block",
                       "systems"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "spmv":
        if rng.random() < 0.35:
            return {"kind": kind, "matrix": rng.choice(["skewed", "random"]), "n": _logint(rng, 2000, 60000)}
        if rng.random() < 0.5:
            return {"kind": kind, "matrix": "lap", "nx": _logint(rng, 40, 1000), "ny": _logint(rng, 40, 1000), "nz": 1}
        return {"kind": kind, "matrix": "lap", "nx": _logint(rng, 20, 128), "ny": _logint(rng, 20, 128),
                "nz": _logint(rng, 20, 128)}
    if kind == "imported":
        return {"kind": kind, "nx": _logint(rng, 9, 61), "ny": _logint(rng, 9, 55), "nz": _logint(rng, 20, 64),
                "slabs": rng.randint(2, 8), "rank": rng.choice([4, 8, 16, 24]), "precision": precision}
    if kind == "block":
        return {"kind": kind, "nx": rng.randint(11, 24), "ny": rng.randint(11, 24), "nz": rng.randint(12, 24),
                "slabs": rng.randint(2, 4), "rank": rng.choice([8, 16, 32]), "precision": precision, "nrhs": 16}
    if kind == "systems":
        lo = rng.randint(24, 48)
        return {"kind": kind, "count": rng.randint(8, 40), "edge_min": lo, "edge_max": rng.randint(lo + 8, 112),
                "precision": precision}
    if kind == "batch":
        return {"kind": kind, "workload": "lap3d_128", "nx": _logint(rng, 16, 48), "ny": _logint(rng, 16, 48),
                "nz": _logint(rng, 16, 48), "precision": precision, "nrhs": rng.randint(2, 24),
                "lanes": rng.choice([1, 2, 4])}
    what = rng.choice(["2d", "3d", "random"])
    if what == "random":
        return {"kind": kind, "workload": "serve", "nx": _logint(rng, 1500, 60000), "ny": 1, "nz": 1,
                "precision": precision}
    if what == "2d":
        return {"kind": kind, "workload": "lap2d_256", "nx": _logint(rng, 40, 256), "ny": _logint(rng, 40, 256),
                "nz": 1, "precision": precision}
    return {"kind": kind, "workload": "lap3d_128", "nx": _logint(rng, 14, 64), "ny": _logint(rng, 14, 64),
            "nz": _logint(rng, 14, 64), "precision": precision}


# ------------------------------------------------------------------ matrices
def _laplacian(nx, ny, nz, shift=0.0):
    """(rowptr, colidx, values) of the 5- or 7-point stencil (the entries of problems.laplacian)."""
    n = nx * ny * nz
    idx = np.arange(n, dtype=np.int64)
    k, r = idx // (nx * ny), idx % (nx * ny)
    i, j = r // nx, r % nx
    mask = np.stack([k > 0, k < nz - 1, i > 0, i < ny - 1, j > 0, j < nx - 1, np.ones(n, bool)], axis=1)
    cols = idx[:, None] + np.array([-nx * ny, nx * ny, -nx, nx, -1, 1, 0])
    vals = np.empty((n, 7), np.result_type(shift, np.float64))
    vals[:, :6] = -1.0
    vals[:, 6] = (4.0 if min(nx, ny, nz) == 1 else 6.0) - shift
    rp = np.zeros(n + 1, np.int32)
    np.cumsum(mask.sum(axis=1), out=rp[1:])
    return rp, cols[mask].astype(np.int32), vals[mask]


def _matrix(case, seed):
    if case.get("matrix") == "skewed":
        return problems.random_skewed(case["n"], seed)
    if case.get("matrix") == "random":
        return problems.random_diag_dominant(case["n"], seed)
    if case.get("workload") == "serve":
        return problems.random_diag_dominant(case["nx"], seed)
    return _laplacian(case["nx"], case["ny"], case["nz"])


def _multiply(A, x):
    rp, cj, va = A
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    t = va * x[cj]
    if np.iscomplexobj(t):
        return (np.bincount(rows, weights=t.real, minlength=len(rp) - 1)
                + 1j * np.bincount(rows, weights=t.imag, minlength=len(rp) - 1))
    return np.bincount(rows, weights=t, minlength=len(rp) - 1)


def _csr(shape, rows, cols, vals):
    order = np.lexsort((cols, rows))
    rp = np.zeros(shape[0] + 1, np.int32)
    np.cumsum(np.bincount(rows, minlength=shape[0]), out=rp[1:])
    return rp, cols[order].astype(np.int32), vals[order], shape[0], shape[1]


class _Block:
    """ILU(0) of the stencil on an nx x ny x nz box with diagonal `diag`: factors and, in 64 bits, the solve."""

    def __init__(self, nx, ny, nz, diag):
        self.shape = (nz, ny, nx)
        self.diag = diag
        k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
        front = (i + j + k).ravel()
        order = np.argsort(front, kind="stable")
        cut = np.searchsorted(front[order], np.arange(nx + ny + nz - 1))
        self.fronts = np.split(order, cut[1:])
        pos = {"x": i.ravel(), "y": j.ravel(), "z": k.ravel()}
        self.nb = [(pos["x"], nx, 1), (pos["y"], ny, nx), (pos["z"], nz, nx * ny)]
        self.n = nx * ny * nz
        d = np.zeros(self.n, np.result_type(diag, np.float64))
        for f in self.fronts:
            t = np.full(f.size, diag, d.dtype)
            for p, _, s in self.nb:
                has = p[f] > 0
                t[has] -= 1.0 / d[f[has] - s]
            d[f] = t
        self.d = d

    def parts(self):
        """rows, cols, vals of L, U and the box's own matrix; the inverse diagonal."""
        idx = np.arange(self.n)
        low = [(idx[p > 0], idx[p > 0] - s) for p, _, s in self.nb]
        up = [(idx[p < m - 1], idx[p < m - 1] + s) for p, m, s in self.nb]
        lr, lc = (np.concatenate([t[q] for t in low]) for q in (0, 1))
        ur, uc = (np.concatenate([t[q] for t in up]) for q in (0, 1))
        off = -np.ones(ur.size, self.d.dtype)
        L = (lr, lc, -1.0 / self.d[lc])
        U = (ur, uc, off)
        B = (np.concatenate([lr, ur, idx]), np.concatenate([lc, uc, idx]),
             np.concatenate([off, off, np.full(self.n, self.diag, self.d.dtype)]))
        return L, U, B, 1.0 / self.d

    def solve(self, b):
        y = b.astype(np.result_type(b, self.d))
        for f in self.fronts:
            for p, _, s in self.nb:
                has = f[p[f] > 0]
                y[has] += y[has - s] / self.d[has - s]
        for f in self.fronts[::-1]:
            for p, m, s in self.nb:
                has = f[p[f] < m - 1]
                y[has] += y[has + s]
            y[f] /= self.d[f]
        return y


class _Slabs:
    """Two levels: slabs of the grid, block ILU(0); the planes between them, ILU(0); a low-rank correction."""

    def __init__(self, case, cplx):
        nx, ny, nz, ns = case["nx"], case["ny"], case["nz"], case["slabs"]
        diag = 6.0 - SHIFT if cplx else 6.0
        self.A = _laplacian(nx, ny, nz, SHIFT if cplx else 0.0)
        plane = nx * ny
        self.n = n = plane * nz
        seps = [(q + 1) * nz // ns for q in range(ns - 1)]
        edges = [-1] + seps + [nz]
        spans = [(a + 1, b) for a, b in zip(edges[:-1], edges[1:])]
        order = [np.arange(a * plane, b * plane) for a, b in spans] + [np.arange(s * plane, (s + 1) * plane)
                                                                       for s in seps]
        self.perm = np.concatenate(order)
        self.nl = n - plane * len(seps)
        self.m = n - self.nl
        self.slabs = [_Block(nx, ny, b - a, diag) for a, b in spans]
        self.planes = [_Block(nx, ny, 1, diag) for _ in seps]
        where = np.empty(n, np.int64)
        where[self.perm] = np.arange(n)
        r = np.concatenate([np.arange(s * plane, (s + 1) * plane) for s in seps])
        rows = np.concatenate([where[r], where[r]]) - self.nl
        cols = np.concatenate([where[r - plane], where[r + plane]])
        self.E = (rows, cols, -np.ones(rows.size, self.A[2].dtype))
        rng = np.random.default_rng(11)
        w = rng.standard_normal((self.m, case["rank"]))
        if cplx:
            w = w + 1j * rng.standard_normal(w.shape)
        self.W = np.linalg.qr(w)[0]
        self.WH = self.W * np.linspace(0.2, 0.02, case["rank"])

    def structures(self, inner):
        levels = []
        for blocks, last in ((self.slabs, False), (self.planes, True)):
            off = np.concatenate([[0], np.cumsum([b.n for b in blocks])])
            got = [b.parts() for b in blocks]
            nl = int(off[-1])
            L, U, B = (_csr((nl, nl), *(np.concatenate([g[q][t] + (o if t < 2 else 0) for g, o in zip(got, off)])
                                        for t in range(3))) for q in range(3))
            lv = LevelStructures(ncomp=len(blocks), dom_ptr=off.astype(np.int32), L=L, U=U,
                                 dinv=np.concatenate([g[3] for g in got]), B=B)
            if not last:
                lv.E = _csr((self.m, self.nl), *self.E)
                lv.F = _csr((self.nl, self.m), self.E[1], self.E[0], self.E[2])
                lv.rank = self.W.shape[1]
                lv.W = self.W.ravel(order="F")
                lv.WH = self.WH.ravel(order="F")
            levels.append(lv)
        return GemslrStructures(n=self.n, A=(*self.A, self.n, self.n), pperm=self.perm.astype(np.int32), qperm=None,
                                lev_ptr=np.array([0, self.nl, self.n], np.int32), levels=levels, inner_enable=inner)

    def apply(self, v):
        r = v[self.perm]
        ru, rl = r[:self.nl], r[self.nl:]

        def blocks(bs, t):
            off = np.cumsum([0] + [b.n for b in bs])
            return np.concatenate([b.solve(t[o:o + b.n]) for b, o in zip(bs, off)])

        z = rl.copy()
        zu = blocks(self.slabs, ru)
        np.add.at(z, self.E[0], zu[self.E[1]])  # z = r_l - E z_u, E = -1
        z = z + self.WH @ (self.W.conj().T @ z)
        xl = blocks(self.planes, z)
        t = ru.copy()
        np.add.at(t, self.E[1], xl[self.E[0]])
        out = np.empty_like(r)
        out[self.perm] = np.concatenate([blocks(self.slabs, t), xl])
        return out


# --------------------------------------------------------------------- inputs
def _x(n, seed, k=0, cplx=False):
    rng = np.random.default_rng([seed, k])
    if cplx:
        return rng.standard_normal(n) + 1j * rng.standard_normal(n)
    return 2.0 * rng.random(n) - 1.0


def _system_list(case, seed):
    """Edges log-uniform over the range, the largest and the smallest among them; convection of either sign."""
    rng = np.random.default_rng(seed)
    c, lo, hi = case["count"], math.log(case["edge_min"]), math.log(case["edge_max"])
    edges = [int(round(math.exp(lo + (hi - lo) * q / (c - 1)))) for q in range(c)]
    return [problems.upwind_convdiff_2d(e, e, rng.uniform(-50, 50), rng.uniform(-50, 50)) for e in edges]


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def prepare(case, seed):
    init(0)
    kind = case["kind"]
    if kind == "spmv":
        A = _matrix(case, seed)
        n = len(A[0]) - 1
        keep = [_dev(a) for a in A]
        csr = _abi.Csr(n, n, len(A[1]), *[t.data_ptr() for t in keep])
        return {"kind": kind, "A": csr, "keep": keep, "x": _dev(_x(n, seed)), "y": torch.zeros(n, dtype=torch.float64,
                                                                                             device="cuda")}
    if kind == "systems":
        p = P.workload_params("convdiff")
        mats = _system_list(case, seed)
        handles = [GemslrHandle.from_matrix(A, p, precision=case["precision"]) for A in mats]
        batch = SystemsBatch(handles)
        off = np.cumsum([0] + [h.n for h in handles])
        b = _dev(np.concatenate([_multiply(A, _x(len(A[0]) - 1, seed, q)) for q, A in enumerate(mats)]))
        return {"kind": kind, "batch": batch, "handles": handles, "b": b, "off": off[:-1], "p": p}
    if kind == "imported":
        s = _Slabs(case, False)
        h = GemslrHandle(s.structures(0), precision=case["precision"])
        return {"kind": kind, "h": h, "b": _dev(_x(s.n, seed))}
    if kind == "block":
        s = _Slabs(case, True)
        h = GemslrHandle(s.structures(1), precision=case["precision"])
        h.set_lanes(16)
        h.set_slots(2)
        b = _dev(np.stack([_multiply(s.A, _x(s.n, seed, q, True)) for q in range(case["nrhs"])]))
        return {"kind": kind, "h": h, "b": b, "p": P.workload_params("zlap3d_96")}
    A = _matrix(case, seed)
    p = P.workload_params(case["workload"])
    h = GemslrHandle.from_matrix(A, p, precision=case["precision"])
    if kind == "apply":
        return {"kind": kind, "h": h, "b": _dev(_x(h.n, seed))}
    if kind == "solve":
        return {"kind": kind, "h": h, "b": _dev(_multiply(A, _x(h.n, seed))), "p": p}
    h.set_lanes(case["lanes"])
    h.set_slots(1 + -(-case["nrhs"] // case["lanes"]))
    b = _dev(np.stack([_multiply(A, _x(h.n, seed, q)) for q in range(case["nrhs"])]))
    return {"kind": kind, "h": h, "b": b, "p": p}


def run(state):
    kind, lib = state["kind"], _abi.lib()
    if kind == "spmv":
        _abi.check(lib.pgx_csr_spmv_device(_abi.C.byref(state["A"]), 1.0, state["x"].data_ptr(), 0.0,
                                           state["y"].data_ptr()))
        return state["y"]
    b = state["b"]
    if kind in ("apply", "imported"):
        z = torch.empty_like(b)
        _abi.check(lib.pgx_gemslr_precond_apply(state["h"]._h, z.data_ptr(), b.data_ptr(), _abi.LOCATION_DEVICE))
        return z
    x = torch.zeros_like(b)  # the initial guess
    torch.cuda.current_stream().synchronize()  # the library works on its own streams
    if kind == "systems":
        at, of = x.data_ptr(), b.data_ptr()
        state["batch"].solve_ptrs([at + 8 * int(o) for o in state["off"]], [of + 8 * int(o) for o in state["off"]],
                                  _abi.LOCATION_DEVICE, state["p"])
    elif kind == "solve":
        state["h"].solve_device(x.data_ptr(), b.data_ptr(), state["p"])
    else:
        n = state["h"].n
        state["h"].solve_batch_ptr(b.shape[0], x.data_ptr(), n, b.data_ptr(), n, _abi.LOCATION_DEVICE, state["p"])
    return x


# ----------------------------------------------------------------- bookkeeping
# entries of the ILUT factors per row and FGMRES iterations of the named workloads (measured on the library's setup)
FILL = {"lap2d_256": 11.6, "lap3d_128": 53.0, "serve": 32.0}
ITERS = {"lap2d_256": 20, "lap3d_128": 14, "serve": 5}


def work(case):
    """Inputs read once, outputs written once; the operations of the products and triangular solves."""
    kind = case["kind"]
    wide = {"mixed": 4, "fp64": 8}[case.get("precision", "fp64")]
    if kind == "spmv":
        if case["matrix"] == "lap":
            n = case["nx"] * case["ny"] * case["nz"]
            nnz = n * (5 if case["nz"] == 1 else 7)
        else:
            n = case["n"]
            nnz = n * (27 if case["matrix"] == "skewed" else 17)
        return {"bytes": 12.0 * nnz + 20.0 * n, "flops": 2.0 * nnz}
    if kind == "systems":
        lo, hi = math.log(case["edge_min"]), math.log(case["edge_max"])
        n = sum(math.exp(2 * (lo + (hi - lo) * q / (case["count"] - 1))) for q in range(case["count"]))
        return {"bytes": n * (11.6 * (wide + 4) + 5 * 12 + 16), "flops": 15 * n * 2.0 * (7 * 11.6 + 5)}
    n = case["nx"] * case["ny"] * case["nz"]
    if kind in ("imported", "block"):
        c = 2 if kind == "block" else 1
        m = (case["slabs"] - 1) * case["nx"] * case["ny"]
        per = n * 6.0 * (c * wide + 4) + 2.0 * m * case["rank"] * c * wide
        if kind == "imported":
            return {"bytes": per + 16.0 * n, "flops": 2.0 * (12.0 * n + 2.0 * m * case["rank"])}
        return {"bytes": per + n * (7 * 20.0 + case["nrhs"] * 32.0), "flops": 40 * case["nrhs"] * 8.0 * n * 50}
    fill = FILL[case["workload"]]
    a = 17 if case["workload"] == "serve" else 5 if case["nz"] == 1 else 7
    inner = 1 if case["workload"] == "serve" else 7  # triangular solves a preconditioner call makes with each factor
    if kind == "apply":
        return {"bytes": n * (fill * (wide + 4) + 16.0), "flops": 2.0 * n * fill * inner}
    rhs = case.get("nrhs", 1)
    return {"bytes": n * (fill * (wide + 4) + 12.0 * a + 16.0 * rhs),
            "flops": rhs * ITERS[case["workload"]] * 2.0 * n * (fill * inner + a)}


def tolerance(case):
    """About four times what two correct implementations were seen to differ by."""
    kind = case["kind"]
    if kind == "spmv":
        return {"rel": 5e-15 if case["matrix"] == "skewed" else 1e-15}  # rows of up to 2000 entries, else of up to 27
    single = case["precision"] == "mixed"
    if kind == "imported":
        return {"rel": 1e-6 if single else 2e-15}
    if kind == "apply":
        return {"rel": 2e-5 if single else 1e-13}
    # iterates that meet the residual tolerance of 1e-8 differ by that times the condition number of the matrix
    return {"rel": {"lap2d_256": 2e-4, "lap3d_128": 1e-5, "serve": 1e-7}.get(case.get("workload"), 5e-6)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "spmv":
        A = _matrix(case, seed)
        return _multiply(A, _x(len(A[0]) - 1, seed))
    if kind == "apply":
        return None  # the factors are the library's own
    if kind == "imported":
        s = _Slabs(case, False)
        return s.apply(_x(s.n, seed))
    if kind == "systems":
        return np.concatenate([_x(len(A[0]) - 1, seed, q) for q, A in enumerate(_system_list(case, seed))])
    n = case["nx"] * case["ny"] * case["nz"]
    if kind == "block":
        return np.stack([_x(n, seed, q, True) for q in range(case["nrhs"])])
    if kind == "batch":
        return np.stack([_x(n, seed, q) for q in range(case["nrhs"])])
    return _x(n, seed)
