"""Sampled outer products and value uploads of many batches. Both are elementwise
(one product of two roundings, one conversion), so they are compared with NumPy
and torch bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def cm():
    import cumat_b200
    return cumat_b200


def _ragged(rows, cols, seed, longest=70):
    """Rows of 0 .. 6 entries, some empty runs, two long rows."""
    rng = np.random.RandomState(seed)
    length = rng.randint(0, 7, rows)
    length[rows // 3:rows // 3 + 5] = 0
    length[rows // 2] = longest
    length[-1] = 0 if seed % 2 else longest
    row_ptr = np.concatenate([[0], np.cumsum(length)]).astype(np.int32)
    col = rng.randint(0, cols, row_ptr[-1]).astype(np.int32)
    return row_ptr, col


# rows at the edges of a warp's 32, and either side of the rule's 303,104 rows
@pytest.mark.parametrize("rows", [12, 31, 32, 33, 64, 1000, 302_593, 303_105])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_sddmm_batches(cuda, rows, dtype):
    m = cm()
    np_dt = np.float32 if dtype == torch.float32 else np.float64
    for cols, ub, vb in ((rows, 1, 1), (rows + 3, 2, 2), (rows, 9, 1), (5, 1, 8), (rows, 17, 17)):
        if rows > 100_000 and max(ub, vb) > 9:
            continue
        row_ptr, col = _ragged(rows, cols, rows + ub)
        if row_ptr[-1] == 0:
            row_ptr[-1] = 1
            col = np.zeros(1, np.int32)
        A = m.SparseMatrix(m.SparsityPattern.csr(rows, cols, row_ptr, col), dtype=dtype)
        rng = np.random.RandomState(7)
        u = rng.uniform(-1, 1, (ub, rows)).astype(np_dt)
        v = rng.uniform(-1, 1, (vb, cols)).astype(np_dt)
        got = m.sddmm(A, torch.from_numpy(u).to(cuda), torch.from_numpy(v).to(cuda), alpha=-0.7).cpu().numpy()
        row = np.repeat(np.arange(rows), np.diff(row_ptr))
        want = (np_dt(-0.7) * u)[:, row] * v[:, col]
        assert got.shape == want.shape and np.array_equal(got, want), (cols, ub, vb)


@pytest.mark.parametrize("stored", [torch.float32, torch.float64, torch.bfloat16])
@pytest.mark.parametrize("given", [torch.float32, torch.float64, torch.bfloat16])
@pytest.mark.parametrize("batches", [1, 3, 300])
def test_value_upload_batches(cuda, stored, given, batches):
    m = cm()
    rows = 37
    row_ptr, col = _ragged(rows, rows, 3)
    ind = np.random.RandomState(1).randint(0, rows, (rows, 3))
    for p, shape in ((m.SparsityPattern.csr(rows, rows, row_ptr, col), (batches, int(row_ptr[-1]))),
                     (m.SparsityPattern.ell(rows, rows, ind), (batches, rows, 3))):
        val = torch.from_numpy(np.random.RandomState(2).uniform(-3, 3, shape)).to(given)
        want = val.to(stored).to(torch.float64).numpy()
        for src in (val, val.to(cuda)):
            got = m.SparseMatrix(p, dtype=stored, batches=batches).setData(src).getData()
            assert np.array_equal(np.asarray(got, np.float64).reshape(shape), want), (p.format, src.device)
