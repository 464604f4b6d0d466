"""On-chip batched solves (cg_onchip.cu, cg_onchip_mixed.cu) against the kernels
they stand in for. The plain FP32 solve keeps the sums of the 1024-thread kernel
in every launch form and the mixed solve those of its kernel's tiers: bit for
bit. FP64 solves are compared by statuses, iteration counts and solutions, and
with the oracle elsewhere."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from cumat_b200 import problems as P  # noqa: E402
from test_resident_gpu import _banded  # noqa: E402


def cm():
    import cumat_b200
    return cumat_b200


def _packed(sides, dims, seed):
    """Packed finite-volume systems of the given sides."""
    parts = [P.fv2d_batch(1, s, s, 0.5, seed + i) if dims == 2 else P.fv3d(s, 0.5, seed + i)
             for i, s in enumerate(sides)]
    off = np.concatenate([[0], np.cumsum([p.n for p in parts])]).astype(np.int64)
    nz = np.concatenate([[0], np.cumsum([p.nnz for p in parts])])
    row_ptr = np.concatenate([p.row_ptr[:-1] + nz[i] for i, p in enumerate(parts)] + [[nz[-1]]]).astype(np.int32)
    col = np.concatenate([p.col + off[i] for i, p in enumerate(parts)]).astype(np.int32)
    return off, row_ptr, col, np.concatenate([p.val for p in parts]), np.concatenate([p.b for p in parts])


# every launch form and its edges: rows at and around 2048, 4096, 8192, 16384
# (45^2 = 2025, 46^2, 64^2, 65^2, 90^2, 91^2, 128^2), tiny systems, 7-point systems
BATCHES = {"all_forms": (2, [128, 1, 2, 91, 90, 65, 64, 46, 45, 33, 32, 31, 127, 7, 90, 64] * 20),
           "few": (2, [128, 45, 90, 3]), "one": (2, [64]), "small": (2, [16, 17, 45, 31] * 60),
           "middle": (2, [64, 65, 90, 89] * 50), "cubes": (3, [12, 13, 16, 5, 20, 24] * 30), "cube": (3, [20])}


def _solve(monkeypatch, onchip, make):
    if not onchip:
        monkeypatch.setenv("CUMAT_CG_ONCHIP", "0")
    try:
        return make()
    finally:
        monkeypatch.delenv("CUMAT_CG_ONCHIP", raising=False)


@pytest.mark.parametrize("values", [torch.float32, torch.float64, torch.bfloat16])
@pytest.mark.parametrize("name", sorted(BATCHES))
def test_fp32_equals_persistent(cuda, monkeypatch, name, values):
    m = cm()
    dims, sides = BATCHES[name]
    off, row_ptr, col, val, b = _packed(sides, dims, 5)
    n = b.size
    p = m.SparsityPattern.csr(n, n, row_ptr, col)
    p.set_systems(off)
    A = m.SparseMatrix(p, dtype=values).setData(val)
    bt = torch.from_numpy(b).to(cuda)
    guess = torch.from_numpy(P.uniform(3, n)).to(cuda)
    for precond in (m.DiagonalPreconditioner, m.IdentityPreconditioner):
        for g in (None, guess):
            out = []
            for onchip in (True, False):
                def make():
                    cg = m.ConjugateGradient(A, precond).setTolerance(1e-6).setMaxIterations(120).set_path(1)
                    return cg.solveWithGuess(bt, g).cpu().numpy(), cg.system_stats()
                out.append(_solve(monkeypatch, onchip, make))
            assert np.array_equal(out[0][0], out[1][0])
            for k in ("iterations", "status", "error"):
                assert np.array_equal(out[0][1][k], out[1][1][k]), k


def test_fp32_batched_values_and_statuses(cuda, monkeypatch):
    # value batches on one pattern, a right-hand side per batch: a NaN, a zero
    # right-hand side and a negative definite set stop alone
    m = cm()
    p1 = P.fv2d_batch(1, 40, 40, 0.5, 4)
    n, B = p1.n, 6
    rng = np.random.default_rng(0)
    vals = np.stack([p1.val * (1 + 0.1 * i) for i in range(B)])
    vals[2] = -vals[2]
    b = rng.uniform(-1, 1, (B, n)).astype(np.float32)
    b[1] = 0
    b[4, 17] = np.nan
    A = m.SparseMatrix(m.SparsityPattern.csr(n, n, p1.row_ptr, p1.col), batches=B).setData(vals)
    out = []
    for onchip in (True, False):
        def make():
            cg = m.ConjugateGradient(A).setTolerance(1e-6)
            return cg.solve(torch.from_numpy(b).to(cuda)).cpu().numpy(), cg.system_stats()
        out.append(_solve(monkeypatch, onchip, make))
    assert out[0][1]["status"].tolist() == out[1][1]["status"].tolist() == [0, 2, 3, 0, 4, 0]
    assert np.array_equal(out[0][0], out[1][0], equal_nan=True)


@pytest.mark.parametrize("values", [torch.float32, torch.float64])
@pytest.mark.parametrize("name", sorted(BATCHES))
def test_fp64_against_persistent(cuda, monkeypatch, name, values):
    m = cm()
    dims, sides = BATCHES[name]
    off, row_ptr, col, val, b = _packed(sides, dims, 7)
    n = b.size
    p = m.SparsityPattern.csr(n, n, row_ptr, col)
    p.set_systems(off)
    A = m.SparseMatrix(p, dtype=values).setData(val)
    bt = torch.from_numpy(b.astype(np.float64)).to(cuda)
    out = []
    for onchip in (True, False):
        def make():
            cg = m.ConjugateGradient(A).setTolerance(1e-12).set_path(1)
            return cg.solve(bt).cpu().numpy(), cg.system_stats()
        out.append(_solve(monkeypatch, onchip, make))
    assert np.all(out[0][1]["status"] == 0)
    assert np.all(np.abs(out[0][1]["iterations"] - out[1][1]["iterations"]) <= 2)
    # both residuals below 1e-12 |b|; |A^-1| |b| / |x| of these systems is below 1e3
    assert np.linalg.norm(out[0][0] - out[1][0]) <= 2e-9 * np.linalg.norm(out[1][0])


@pytest.mark.parametrize("inner,outer", [(torch.float32, None), (torch.float32, torch.float64),
                                         (torch.bfloat16, torch.float32), (torch.bfloat16, torch.float64)])
@pytest.mark.parametrize("name", sorted(BATCHES))
def test_mixed_equals_persistent(cuda, monkeypatch, name, inner, outer):
    m = cm()
    dims, sides = BATCHES[name]
    off, row_ptr, col, val, b = _packed(sides, dims, 9)
    n = b.size
    p = m.SparsityPattern.csr(n, n, row_ptr, col)
    p.set_systems(off)
    A = m.SparseMatrix(p, dtype=inner).setData(val)
    Ao = m.SparseMatrix(p, dtype=outer).setData(val) if outer else None
    bt = torch.from_numpy(b.astype(np.float64)).to(cuda)
    monkeypatch.setenv("CUMAT_CG_BF16_FALLBACK", "0")
    out = []
    for onchip in (True, False):
        def make():
            cg = m.ConjugateGradient(A).set_path(1)
            return cg.solve_refined(bt, outer=Ao, outer_tol=1e-11, max_outer=200).cpu().numpy(), cg.system_stats()
        out.append(_solve(monkeypatch, onchip, make))
    assert np.array_equal(out[0][0], out[1][0])
    for k in ("iterations", "status", "outer", "error"):
        assert np.array_equal(out[0][1][k], out[1][1][k]), k
    if inner == torch.float32:
        assert np.all(out[0][1]["status"] == 0)


def test_mixed_iteration_limit_reports_the_true_residual(cuda):
    m = cm()
    p1 = P.fv2d_batch(1, 100, 100, 0.5, 4)
    A = m.SparseMatrix(m.SparsityPattern.csr(p1.n, p1.n, p1.row_ptr, p1.col)).setData(p1.val)
    b = p1.b.astype(np.float64)
    cg = m.ConjugateGradient(A).setMaxIterations(20)
    x = cg.solve_refined(torch.from_numpy(b).to(cuda), outer_tol=1e-10).cpu().numpy()
    st = cg.system_stats()
    assert st["status"][0] == 1 and st["iterations"][0] == 20
    r = b - np.add.reduceat(p1.val.astype(np.float64) * x[p1.col], p1.row_ptr[:-1])
    assert abs(np.linalg.norm(r) / np.linalg.norm(b) - cg.error()) <= 1e-12


@pytest.mark.parametrize("offsets", [(1, 7000), (3, 4099)])
def test_wide_halo_keeps_the_other_kernels(cuda, monkeypatch, offsets):
    # a halo that fits no launch form: the solve still runs, with the same result
    m = cm()
    n = 15000
    row_ptr, col, val = _banded(n, offsets, 1)
    b = P.uniform(2, n)
    A = m.SparseMatrix(m.SparsityPattern.csr(n, n, row_ptr, col)).setData(val)
    for dt in (torch.float32, torch.float64):
        out = []
        for onchip in (True, False):
            def make():
                cg = m.ConjugateGradient(A).setTolerance(1e-5).set_path(1)
                return cg.solve(torch.from_numpy(b).to(cuda).to(dt)).cpu().numpy(), cg.system_stats()
            out.append(_solve(monkeypatch, onchip, make))
        assert out[0][1]["status"][0] == 0
        assert np.linalg.norm(out[0][0] - out[1][0]) <= 1e-4 * np.linalg.norm(out[1][0])
