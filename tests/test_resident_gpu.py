"""Chip-resident forms of single-system solves against the paths whose sums they
reproduce: the resident loop (cg_resident.cu) against the graph loop, the solve
spread over all SMs (cg_wide.cu) against the cluster solve. Both keep the other
path's order of additions, so solutions, iteration counts and statuses are
compared bit for bit; the other paths are held to the oracle elsewhere."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from cumat_b200 import problems as P  # noqa: E402


def cm():
    import cumat_b200
    return cumat_b200


def _banded(n, offsets, seed):
    """A symmetric diagonally dominant matrix with entries at +-offsets."""
    rng = np.random.default_rng(seed)
    offs = sorted({0, *offsets, *(-o for o in offsets)})
    w = {o: -rng.uniform(0.2, 1.0, n).astype(np.float32) for o in offsets}
    rows, cols, vals = [], [], []
    diag = np.full(n, 0.05)
    r = np.arange(n)
    for o in offsets:
        ok = r + o < n
        rows += [r[ok], r[ok] + o]
        cols += [r[ok] + o, r[ok]]
        vals += [w[o][ok], w[o][ok]]
        diag[r[ok]] -= w[o][ok]
        diag[r[ok] + o] -= w[o][ok]
    rows.append(r), cols.append(r), vals.append(diag)
    rows, cols, vals = map(np.concatenate, (rows, cols, vals))
    order = np.lexsort((cols, rows))
    row_ptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    assert len(offs) <= 7
    return row_ptr, cols[order].astype(np.int32), vals[order].astype(np.float32)


def _system(kind, size, seed=3):
    if kind == "2d":
        p = P.poisson2d(size, seed)
        return p.row_ptr, p.col, p.val, p.b
    if kind == "fv":
        p = P.fv2d_batch(1, size, size, 0.5, seed)
        return p.row_ptr, p.col, p.val, p.b
    if kind == "3d":
        p = P.fv3d(size, 0.5, seed)
        return p.row_ptr, p.col, p.val, p.b
    n, offsets = size
    row_ptr, col, val = _banded(n, offsets, seed)
    return row_ptr, col, val, P.uniform(seed, n)


def _solver(monkeypatch, A, env, precond):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    m = cm()
    cg = m.ConjugateGradient(A, m.DiagonalPreconditioner if precond else m.IdentityPreconditioner)
    for k in env:
        monkeypatch.delenv(k)
    return cg


NO_OTHER = {"CUMAT_CG_CLUSTER": "0", "CUMAT_CG_COOP": "0"}
GRAPH = {**NO_OTHER, "CUMAT_CG_RESIDENT": "0"}

# one tile; a part tile; one quad per thread and two; rows not a multiple of 4
# (the update's sums in row order); windows wider than a CTA's rows; offsets
# that are no multiple of 4, and far apart
RESIDENT = [("2d", 15), ("2d", 64), ("2d", 151), ("fv", 333), ("2d", 390), ("2d", 780), ("fv", 1023), ("2d", 1024),
            ("3d", 33), ("3d", 64), ("3d", 101), ("band", (50001, (1,))), ("band", (60000, (3, 7))),
            ("band", (40000, (1, 15000))), ("band", (30010, (2, 9, 6001))), ("band", (262145, (5, 1001, 70003)))]


@pytest.mark.parametrize("precond", [True, False])
@pytest.mark.parametrize("kind,size", RESIDENT)
def test_resident_equals_graph_fp32(cuda, monkeypatch, kind, size, precond):
    m = cm()
    row_ptr, col, val, b = _system(kind, size)
    n = b.size
    A = m.SparseMatrix(m.SparsityPattern.csr(n, n, row_ptr, col)).setData(val)
    bt = torch.from_numpy(b).to(cuda)
    guess = torch.from_numpy(P.uniform(9, n)).to(cuda)
    for g in (None, guess):
        out = []
        for env in (NO_OTHER, GRAPH):
            cg = _solver(monkeypatch, A, env, precond).setTolerance(1e-6).setMaxIterations(150).set_path(2)
            x = cg.solveWithGuess(bt, g).cpu().numpy()
            out.append((x, cg.system_stats(), cg.error()))
        assert np.array_equal(out[0][0], out[1][0])
        assert out[0][1]["iterations"][0] == out[1][1]["iterations"][0]
        assert out[0][1]["status"][0] == out[1][1]["status"][0]
        assert out[0][2] == out[1][2]
    assert m.Context.current().device_errors() == 0


@pytest.mark.parametrize("kind,size", [("2d", 150), ("fv", 301), ("2d", 500), ("2d", 770), ("3d", 40), ("3d", 75),
                                       ("band", (50001, (1, 15)))])
def test_resident_fp64_against_graph(cuda, monkeypatch, kind, size):
    # (the sums agree except in the last rows of a system whose size is 2 mod
    # 4: rounding-level differences at a tolerance of 1e-12)
    m = cm()
    row_ptr, col, val, b = _system(kind, size)
    n = b.size
    A = m.SparseMatrix(m.SparsityPattern.csr(n, n, row_ptr, col), dtype=torch.float64).setData(val.astype(np.float64))
    bt = torch.from_numpy(b.astype(np.float64)).to(cuda)
    out = []
    for env in (NO_OTHER, GRAPH):
        cg = _solver(monkeypatch, A, env, True).setTolerance(1e-12).set_path(2)
        x = cg.solve(bt).cpu().numpy()
        out.append((x, cg.system_stats()))
    assert out[0][1]["status"][0] == 0
    assert abs(int(out[0][1]["iterations"][0]) - int(out[1][1]["iterations"][0])) <= 2
    # both residuals are below 1e-12 |b|: the solutions differ by at most
    # 2e-12 |b| times the norm of the inverse, here below 1e3 times |x| / |b|
    assert np.linalg.norm(out[0][0] - out[1][0]) <= 2e-9 * np.linalg.norm(out[1][0])


@pytest.mark.parametrize("inner", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kind,size", [("3d", 26), ("3d", 64), ("3d", 90), ("fv", 150), ("fv", 401), ("2d", 1000),
                                       ("band", (20011, (1, 77, 6001)))])
def test_resident_mixed_equals_graph(cuda, monkeypatch, kind, size, inner):
    m = cm()
    row_ptr, col, val, b = _system(kind, size)
    n = b.size
    p = m.SparsityPattern.csr(n, n, row_ptr, col)
    A, A64 = m.SparseMatrix(p, dtype=inner).setData(val), m.SparseMatrix(p, dtype=torch.float64).setData(val)
    bt = torch.from_numpy(b.astype(np.float64)).to(cuda)
    monkeypatch.setenv("CUMAT_CG_BF16_FALLBACK", "0")
    out = []
    for env in (NO_OTHER, GRAPH):
        cg = _solver(monkeypatch, A, env, True).set_path(2).setMaxIterations(600)
        x = cg.solve_refined(bt, outer=A64, outer_tol=1e-11, max_outer=100).cpu().numpy()
        out.append((x, cg.system_stats()))
    assert np.array_equal(out[0][0], out[1][0])
    for k in ("iterations", "status", "outer", "error"):
        assert out[0][1][k][0] == out[1][1][k][0], k
    assert m.Context.current().device_errors() == 0


def test_resident_statuses(cuda, monkeypatch):
    # iteration limit, zero right-hand side, converged guess, indefinite matrix, NaN
    m = cm()
    row_ptr, col, val, b = _system("2d", 200)
    n = b.size
    p = m.SparsityPattern.csr(n, n, row_ptr, col)
    A, Neg = m.SparseMatrix(p).setData(val), m.SparseMatrix(p).setData(-val)
    bt = torch.from_numpy(b).to(cuda)
    bad = bt.clone()
    bad[n // 2] = float("nan")
    for M, rhs, limit in ((A, bt, 3), (A, bt, 0), (A, torch.zeros_like(bt), -1), (Neg, bt, -1), (A, bad, -1)):
        out = []
        for env in (NO_OTHER, GRAPH):
            cg = _solver(monkeypatch, M, env, True).setTolerance(1e-6).setMaxIterations(limit).set_path(2)
            x = cg.solve(rhs).cpu().numpy()
            st = cg.system_stats()
            out.append((x, int(st["iterations"][0]), int(st["status"][0])))
        assert out[0][1:] == out[1][1:]
        assert np.array_equal(out[0][0], out[1][0], equal_nan=True)


# the sizes at which a thread owns 1, 2, 4 and 8 rows; a last unit of one row;
# fewer units than SMs and a last cluster CTA that is nearly empty
WIDE = [("2d", 65), ("2d", 90), ("fv", 128), ("2d", 129), ("fv", 181), ("2d", 200), ("2d", 257), ("fv", 300),
        ("2d", 362), ("3d", 17), ("3d", 25), ("3d", 40), ("3d", 50), ("band", (4097, (1, 2))),
        ("band", (16385, (3, 7))), ("band", (131072, (1, 4099))), ("band", (32801, (1, 33, 1024)))]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("kind,size", WIDE)
def test_wide_equals_cluster(cuda, monkeypatch, kind, size, dtype):
    m = cm()
    row_ptr, col, val, b = _system(kind, size)
    n = b.size
    np_dt = np.float32 if dtype == torch.float32 else np.float64
    A = m.SparseMatrix(m.SparsityPattern.csr(n, n, row_ptr, col), dtype=dtype).setData(val.astype(np_dt))
    bt = torch.from_numpy(b.astype(np_dt)).to(cuda)
    guess = torch.from_numpy(P.uniform(9, n).astype(np_dt)).to(cuda)
    for precond in (True, False):
        for g in (None, guess):
            out = []
            for env in ({}, {"CUMAT_CG_WIDE": "0", "CUMAT_CG_RESIDENT": "0"}):
                cg = _solver(monkeypatch, A, env, precond).setTolerance(1e-6).setMaxIterations(200)
                x = cg.solveWithGuess(bt, g).cpu().numpy()
                out.append((x, cg.system_stats(), cg.error()))
            assert out[0][1]["iterations"][0] == out[1][1]["iterations"][0]
            assert out[0][1]["status"][0] == out[1][1]["status"][0]
            if dtype == torch.float32 or n <= 65536:   # (larger FP64 systems: the graph and resident loops)
                assert np.array_equal(out[0][0], out[1][0])
                assert out[0][2] == out[1][2]
    assert m.Context.current().device_errors() == 0


def test_wide_statuses(cuda, monkeypatch):
    m = cm()
    row_ptr, col, val, b = _system("2d", 100)
    n = b.size
    p = m.SparsityPattern.csr(n, n, row_ptr, col)
    A, Neg = m.SparseMatrix(p).setData(val), m.SparseMatrix(p).setData(-val)
    bt = torch.from_numpy(b).to(cuda)
    bad = bt.clone()
    bad[n // 3] = float("nan")
    for M, rhs, limit in ((A, bt, 3), (A, bt, 0), (A, torch.zeros_like(bt), -1), (Neg, bt, -1), (A, bad, -1)):
        out = []
        for env in ({}, {"CUMAT_CG_WIDE": "0"}):
            cg = _solver(monkeypatch, M, env, True).setTolerance(1e-6).setMaxIterations(limit)
            x = cg.solve(rhs).cpu().numpy()
            st = cg.system_stats()
            out.append((x, int(st["iterations"][0]), int(st["status"][0])))
        assert out[0][1:] == out[1][1:]
        assert np.array_equal(out[0][0], out[1][0], equal_nan=True)


@pytest.mark.parametrize("side,path", [(100, 0), (400, 2)])
def test_tagged_word_waits_run_out(cuda, monkeypatch, side, path):
    # the readers wait for a tag that is never written: every poll runs out, the
    # device error bit is set, nothing is reported converged, and the context works
    m = cm()
    row_ptr, col, val, b = _system("2d", side)
    n = b.size
    A = m.SparseMatrix(m.SparsityPattern.csr(n, n, row_ptr, col)).setData(val)
    bt = torch.from_numpy(b).to(cuda)
    ctx = m.Context.current()
    ctx.device_errors()
    cg = m.ConjugateGradient(A).setTolerance(1e-6).set_path(path)
    monkeypatch.setenv("CUMAT_TEST_GRID_SPINS", "2000")
    monkeypatch.setenv("CUMAT_TEST_GRID_EXTRA", "7")
    cg.solve(bt)
    assert ctx.device_errors() & 2
    assert cg.system_stats()["status"][0] != 0
    monkeypatch.delenv("CUMAT_TEST_GRID_SPINS")
    monkeypatch.delenv("CUMAT_TEST_GRID_EXTRA")
    cg.solve(bt)
    assert ctx.device_errors() == 0 and cg.system_stats()["status"][0] == 0


def test_a_sum_that_lacks_a_partial_is_not_accepted(cuda, monkeypatch):
    # one combining warp waits for a partial that no CTA publishes: the total it could
    # not form reaches no CTA, although the sum of what is there would converge
    m = cm()
    row_ptr, col, val, b = _system("2d", 400)
    n = b.size
    A = m.SparseMatrix(m.SparsityPattern.csr(n, n, row_ptr, col)).setData(val)
    bt = torch.from_numpy(b).to(cuda)
    ctx = m.Context.current()
    ctx.device_errors()
    # (r_1 = (4 - A) b / 4 here, about half of |b|: the first iteration converges)
    cg = _solver(monkeypatch, A, NO_OTHER, True).setTolerance(0.95).set_path(2)
    cg.solve(bt)
    assert cg.system_stats()["status"][0] == 0 and cg.system_stats()["iterations"][0] == 0
    monkeypatch.setenv("CUMAT_TEST_GRID_SPINS", "2000")
    monkeypatch.setenv("CUMAT_TEST_GRID_PARTIAL", "1")
    cg.solve(bt)
    assert ctx.device_errors() & 2
    assert cg.system_stats()["status"][0] != 0
    monkeypatch.delenv("CUMAT_TEST_GRID_SPINS")
    monkeypatch.delenv("CUMAT_TEST_GRID_PARTIAL")
    cg.solve(bt)
    assert ctx.device_errors() == 0 and cg.system_stats()["status"][0] == 0


@pytest.mark.parametrize("kind,size", [("3d", 40), ("fv", 401), ("2d", 1000)])
def test_resident_mixed_with_frequent_replacements(cuda, monkeypatch, kind, size):
    # a replacement whenever the residual fell by a tenth: every one reads x entries that
    # other CTAs have just folded
    m = cm()
    row_ptr, col, val, b = _system(kind, size)
    n = b.size
    p = m.SparsityPattern.csr(n, n, row_ptr, col)
    A, A64 = m.SparseMatrix(p).setData(val), m.SparseMatrix(p, dtype=torch.float64).setData(val)
    bt = torch.from_numpy(b.astype(np.float64)).to(cuda)
    out = []
    for env in (NO_OTHER, GRAPH):
        cg = _solver(monkeypatch, A, env, True).set_path(2).setMaxIterations(400).set_refinement(0, 0.9)
        x = cg.solve_refined(bt, outer=A64, outer_tol=1e-11, max_outer=400).cpu().numpy()
        out.append((x, cg.system_stats()))
    assert out[0][1]["outer"][0] > 20
    assert np.array_equal(out[0][0], out[1][0])
    for k in ("iterations", "status", "outer", "error"):
        assert out[0][1][k][0] == out[1][1][k][0], k
