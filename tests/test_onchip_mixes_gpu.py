"""Batched solves whose systems differ in shape: squares, long grids and bands of
one batch, for which the launch forms of cg_onchip.cu differ in their halos. The
solutions are held to their residual, formed with NumPy in 64 bits: a solve that
stops at |r| < tol |b| has a true residual within tol |b| plus the drift of the
recursion, at most (iterations) (unit roundoff) (|A| |x| / |b|), below 1e3 * 1e-16 *
1e3 for these systems in FP64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from cumat_b200 import problems as P  # noqa: E402
from test_resident_gpu import _banded  # noqa: E402


def cm():
    import cumat_b200
    return cumat_b200


def _pack(systems, seed):
    """Packed systems (rows, offsets): row offsets, CSR arrays, right-hand side."""
    parts = {}
    out = []
    for i, key in enumerate(systems):
        if key not in parts:
            parts[key] = _banded(*key, seed + i)
        out.append(parts[key])
    off = np.concatenate([[0], np.cumsum([k[0] for k in systems])]).astype(np.int64)
    nz = np.concatenate([[0], np.cumsum([p[1].size for p in out])])
    row_ptr = np.concatenate([p[0][:-1] + nz[i] for i, p in enumerate(out)] + [[nz[-1]]]).astype(np.int32)
    col = np.concatenate([p[1] + off[i] for i, p in enumerate(out)]).astype(np.int32)
    return off, row_ptr, col, np.concatenate([p[2] for p in out]), P.uniform(seed, int(off[-1]))


def _residuals(off, row_ptr, col, val, b, x):
    """|b - A x| / |b| per system, in 64 bits."""
    r = b.astype(np.float64) - np.add.reduceat(val.astype(np.float64) * x.astype(np.float64)[col], row_ptr[:-1])
    n2 = lambda v: np.sqrt(np.add.reduceat(v.astype(np.float64) ** 2, off[:-1]))  # noqa: E731
    return n2(r) / n2(b)


def _square(s):
    return (s * s, (1, s))


def _grid(w, h, d=0):
    return (w * h * max(d, 1), (1, w, w * h) if d else (1, w))


# systems of one batch that take different forms: a long grid whose halo spans more
# than a CTA's rows, and small systems that the batch's halo keeps out of the
# smallest forms; the last one is reached by FP32 values under FP64 vectors
MIXES = {"long_grid": [_square(100)] * 10 + [_grid(2200, 2)] + [_square(58)] * 2,
         "long_grid_3d": [(13000, (1, 100, 1300)), _grid(50, 70, 3), (9000, (1, 90, 900))],
         "band": [_square(128)] * 10 + [(5000, (1, 3500))],
         "band_alone": [(5000, (1, 2499)), (4100, (3, 2100)), (9000, (1, 3000)), (12000, (7, 3071))],
         "wide": [_square(64)] * 150 + [_grid(3000, 3), _grid(1025, 15), _square(20)],
         # (values, p and halo of an FP64 cluster at the shared memory's limit)
         "halo_2110": [_grid(2110, 7)] * 20 + [_grid(2109, 7)] * 130,
         "small": [_grid(700, 2), _grid(2, 700), _square(31), (50, (1,)), (3, (2,))] * 40}


@pytest.mark.parametrize("values", [torch.float64, torch.float32])
@pytest.mark.parametrize("name", sorted(MIXES))
def test_fp64_mixed_shapes(cuda, name, values):
    m = cm()
    off, row_ptr, col, val, b = _pack(MIXES[name], 11)
    n = b.size
    p = m.SparsityPattern.csr(n, n, row_ptr, col)
    p.set_systems(off)
    A = m.SparseMatrix(p, dtype=values).setData(val)
    cg = m.ConjugateGradient(A).setTolerance(1e-8).set_path(1)
    x = cg.solve(torch.from_numpy(b.astype(np.float64)).to(cuda)).cpu().numpy()
    assert np.all(cg.system_stats()["status"] == 0)
    assert np.all(_residuals(off, row_ptr, col, val, b, x) <= 1.1e-8)


# one system on each path that reads stencil patterns in the diagonal layout, and a batch
@pytest.mark.parametrize("systems,path", [([_square(31)] * 160, 0), ([_square(64)], 0), ([_square(100)], 0),
                                          ([_square(400)], 0), ([_square(40)], 2)])
@pytest.mark.parametrize("kind", ["fp32", "fp64", "mixed"])
def test_repeated_entries_add_up(cuda, systems, path, kind):
    # every entry stored as two (1/4 and 3/4 of it), which a product adds up
    m = cm()
    off, row_ptr, col, val, b = _pack(systems, 5)
    n = b.size
    quarter = (val * np.float32(0.25)).astype(np.float32)
    v2 = np.stack([quarter, val - quarter], 1).ravel()
    p = m.SparsityPattern.csr(n, n, row_ptr * 2, np.repeat(col, 2))
    if len(systems) > 1:
        p.set_systems(off)
    dt = torch.float64 if kind == "fp64" else torch.float32
    A = m.SparseMatrix(p, dtype=dt).setData(v2)
    bt = torch.from_numpy(b).to(cuda).to(torch.float32 if kind == "fp32" else torch.float64)
    cg = m.ConjugateGradient(A).setTolerance(1e-8 if kind == "fp64" else 1e-5).set_path(path)
    x = (cg.solve_refined(bt, outer_tol=1e-10) if kind == "mixed" else cg.solve(bt)).cpu().numpy()
    assert np.all(cg.system_stats()["status"] == 0)
    # (FP32: the recursion drifts by at most 100 iterations of 2^-24 |A| |x| / |b| <= 50)
    limit = {"fp32": 3.1e-4, "fp64": 1.1e-8, "mixed": 1.01e-10}[kind]
    assert np.all(_residuals(off, row_ptr * 2, np.repeat(col, 2), v2, b, x) <= limit)


# rows either side of the layout's 1024-row blocks, systems of one and two rows, three
# to seven offsets of a system, entries of a row in any order
LAYOUT = [(1, ()), (2, (1,)), (1023, (1, 31)), (1024, (2,)), (1025, (1, 32, 33)), (2049, (1, 5, 1024)), (3000, (7,))]


@pytest.mark.parametrize("order", ["ascending", "descending", "shuffled"])
@pytest.mark.parametrize("kind", ["fp32", "fp64", "mixed", "product"])
def test_entry_order_of_the_diagonal_layout(cuda, order, kind):
    m = cm()
    off, row_ptr, col, val, b = _pack(LAYOUT * 25, 3)
    n = b.size
    key = {"ascending": col, "descending": -col, "shuffled": np.random.RandomState(4).randint(0, 1 << 30, col.size)}[order]
    perm = np.lexsort((key, np.repeat(np.arange(n), np.diff(row_ptr))))
    col, val = col[perm], val[perm]
    p = m.SparsityPattern.csr(n, n, row_ptr, col)
    p.set_systems(off)
    A = m.SparseMatrix(p, dtype=torch.float64 if kind == "fp64" else torch.float32).setData(val)
    bt = torch.from_numpy(b).to(cuda).to(torch.float32 if kind == "fp32" else torch.float64)
    if kind == "product":   # the grid path's product in the layout: an iteration of it
        cg = m.ConjugateGradient(A).setTolerance(1e-8).set_path(2)
    else:
        cg = m.ConjugateGradient(A).setTolerance(1e-5 if kind == "fp32" else 1e-8).set_path(1)
    x = (cg.solve_refined(bt, outer_tol=1e-10) if kind == "mixed" else cg.solve(bt)).cpu().numpy()
    assert np.all(cg.system_stats()["status"] == 0)
    limit = {"fp32": 3.1e-4, "fp64": 1.1e-8, "mixed": 1.01e-10, "product": 1.1e-8}[kind]
    assert np.all(_residuals(off, row_ptr, col, val, b, x) <= limit)


@pytest.mark.parametrize("diagonals", [True, False])
def test_value_uploads_rebuild_the_layouts_read(cuda, monkeypatch, diagonals):
    # a mixed solve of systems either side of 8192 rows after a value upload: the scale,
    # the sliced values (FP64 residual above 8192 rows), the scaled diagonals and the unit
    # diagonal's flags, and the diagonals (FP64 residual below); on the sliced layout the
    # scale and both sliced copies
    m = cm()
    if not diagonals:
        monkeypatch.setenv("CUMAT_CG_DIA", "0")
    off, row_ptr, col, val, b = _pack([_square(100), _square(50)], 5)
    n = b.size
    p = m.SparsityPattern.csr(n, n, row_ptr, col)
    p.set_systems(off)
    A = m.SparseMatrix(p).setData(val)
    cg = m.ConjugateGradient(A).set_path(1)
    bt = torch.from_numpy(b.astype(np.float64)).to(cuda)
    launches = []
    for scale in (None, 1.0, 3.0):
        if scale is not None:
            A.setData(val * np.float32(scale))
        for again in (False, True):
            before = m.launch_count()
            x = cg.solve_refined(bt, outer_tol=1e-10).cpu().numpy()
            launches.append(m.launch_count() - before)
            assert np.all(_residuals(off, row_ptr, col, val * np.float32(scale or 1), b, x) <= 1.01e-10)
    solve = 2
    assert launches[1::2] == [solve] * 3
    assert launches[2::2] == [solve + (5 if diagonals else 3)] * 2


@pytest.mark.parametrize("kind", ["fp64", "mixed"])
def test_a_failed_tier_launch_waits_for_the_others(cuda, monkeypatch, kind):
    # the second launch of a solve of two forms fails: the call raises, and what follows
    # on the caller's stream comes after the first launch, which still writes x
    m = cm()
    systems = [_square(110)] * 600 + [_square(40)] * 50
    off, row_ptr, col, val, b = _pack(systems, 5)
    n = b.size
    p = m.SparsityPattern.csr(n, n, row_ptr, col)
    p.set_systems(off)
    A = m.SparseMatrix(p, dtype=torch.float64 if kind == "fp64" else torch.float32).setData(val)
    bt = torch.from_numpy(b.astype(np.float64)).to(cuda)
    solve = lambda cg, x: (cg.solve(bt, out=x) if kind == "fp64"  # noqa: E731
                           else cg.solve_refined(bt, outer_tol=1e-8, out=x))
    big = int(off[600])
    want = solve(m.ConjugateGradient(A).setTolerance(1e-8), None).cpu().numpy()   # (all layouts in place)
    monkeypatch.setenv("CUMAT_TEST_TIER_FAIL", "1")
    cg = m.ConjugateGradient(A).setTolerance(1e-8)
    monkeypatch.delenv("CUMAT_TEST_TIER_FAIL")
    x = torch.full((n,), float("nan"), dtype=torch.float64, device=cuda)
    for _ in range(2):
        x.fill_(float("nan"))
        with pytest.raises(m.CuMatError):
            solve(cg, x)
        got = x.cpu().numpy()
        assert np.array_equal(got[:big], want[:big]) and np.all(np.isnan(got[big:]))


@pytest.mark.parametrize("values", [torch.float64, torch.float32, torch.bfloat16])
@pytest.mark.parametrize("name", sorted(MIXES))
def test_fp64_guess_and_preconditioner(cuda, monkeypatch, name, values):
    # against the kernels the forms stand in for: the statuses, the iteration counts (the
    # sums differ in their order) and the true residual of every combination
    m = cm()
    off, row_ptr, col, val, b = _pack(MIXES[name], 13)
    n = b.size
    p = m.SparsityPattern.csr(n, n, row_ptr, col)
    p.set_systems(off)
    A = m.SparseMatrix(p, dtype=values).setData(val)
    val = A.getData().astype(np.float64).reshape(-1)   # (BF16: as stored)
    bt = torch.from_numpy(b.astype(np.float64)).to(cuda)
    guess = torch.from_numpy(P.uniform(17, n).astype(np.float64)).to(cuda)
    for precond in (m.DiagonalPreconditioner, m.IdentityPreconditioner):
        for g in (None, guess):
            stats = []
            for onchip in ("1", "0"):
                monkeypatch.setenv("CUMAT_CG_ONCHIP", onchip)
                cg = m.ConjugateGradient(A, precond).setTolerance(1e-8).set_path(1)
                x = cg.solveWithGuess(bt, g).cpu().numpy()
                stats.append(cg.system_stats())
                ok = stats[-1]["status"] == 0
                assert np.all(_residuals(off, row_ptr, col, val, b, x)[ok] <= 1.1e-8)
            assert np.array_equal(stats[0]["status"], stats[1]["status"])
            if values != torch.bfloat16:   # (rounded to 8 bits the matrices may lose definiteness)
                assert np.all(stats[0]["status"] == 0)
                assert np.all(np.abs(stats[0]["iterations"] - stats[1]["iterations"]) <= 2)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("rhs", ["one", "each"])
def test_value_sets_on_one_pattern(cuda, dtype, rhs):
    # several value sets on one packed pattern of mixed shapes, one right-hand side for all
    # or one each, with a guess
    m = cm()
    systems = [_square(100), _grid(700, 4), _square(58), (5000, (1, 1400)), _square(12)]
    off, row_ptr, col, val, b = _pack(systems, 7)
    n, B = b.size, 30
    p = m.SparsityPattern.csr(n, n, row_ptr, col)
    p.set_systems(off)
    vals = np.stack([val * np.float32(1 + 0.05 * i) for i in range(B)])
    bs = np.stack([P.uniform(i, n) for i in range(B)]) if rhs == "each" else b
    A = m.SparseMatrix(p, dtype=dtype, batches=B).setData(vals)
    tol = 1e-8 if dtype == torch.float64 else 1e-5
    cg = m.ConjugateGradient(A).setTolerance(tol).set_path(1)
    guess = torch.from_numpy(np.stack([P.uniform(50 + i, n) for i in range(B)])).to(cuda).to(dtype)
    for g in (None, guess):
        x = cg.solveWithGuess(torch.from_numpy(bs).to(cuda).to(dtype), g).cpu().numpy()
        assert np.all(cg.system_stats()["status"] == 0)
        for i in range(B):
            res = _residuals(off, row_ptr, col, vals[i], bs[i] if rhs == "each" else b, x[i])
            # (FP32: the recursion drifts by at most 100 iterations of 2^-24 |A| |x| / |b| <= 50)
            assert np.all(res <= (1.1e-8 if dtype == torch.float64 else 3.1e-4))


@pytest.mark.parametrize("name", sorted(MIXES))
def test_fp32_and_mixed_shapes_equal_persistent(cuda, monkeypatch, name):
    # these keep the order of sums of the kernels they stand in for: bit for bit
    m = cm()
    off, row_ptr, col, val, b = _pack(MIXES[name], 19)
    n = b.size
    p = m.SparsityPattern.csr(n, n, row_ptr, col)
    p.set_systems(off)
    A = m.SparseMatrix(p).setData(val)
    bt = torch.from_numpy(b).to(cuda)
    for mixed in (False, True):
        out = []
        for onchip in ("1", "0"):
            monkeypatch.setenv("CUMAT_CG_ONCHIP", onchip)
            cg = m.ConjugateGradient(A).setTolerance(1e-5).set_path(1)
            x = cg.solve_refined(bt.double(), outer_tol=1e-10) if mixed else cg.solve(bt)
            out.append((x.cpu().numpy(), cg.system_stats()))
        assert np.array_equal(out[0][0], out[1][0])
        for k in ("iterations", "status", "error"):
            assert np.array_equal(out[0][1][k], out[1][1][k]), k
        if mixed:
            assert np.all(_residuals(off, row_ptr, col, val, b, out[0][0]) <= 1.01e-10)
