"""Timed cases of the sparse solver path: what a user of the package calls, at
the sizes it meets.

A case names a kind of call and its sizes:

  solve      ConjugateGradient.solve: one system, or a packed batch of uneven
             systems, FP32 or FP64, with or without an initial guess
  refined    ConjugateGradient.solve_refined: FP32 CG with FP64 residuals
  adjoint    sparse_solve forward and backward through torch.autograd
  product    A x or A^T x in CSR, CSC or ELLPACK storage
  blocked    ConjugateGradient on a matrix of 3 x 3 blocks (block CSR)
  vectors    dot, linear_combination and reduce on batched vectors

The matrices are finite-volume diffusion operators on square or cubic grids
with Dirichlet boundaries (face coefficients exp(N(0, sigma^2)); sigma 0 is the
Poisson matrix), the right-hand sides uniform on [-1, 1].
"""
import math

import numpy as np
import torch

import cumat_b200 as cm
from cumat_b200.autograd import SparseSolveOp, sparse_solve

_F = {"f32": torch.float32, "f64": torch.float64}


def listed():
    return [
        # one small system solved to single precision, the latency of a whole
        # solve: the 64 x 64 Poisson problem, no preconditioner
        {"name": "solve_one_64", "kind": "solve", "dims": 2, "side": 64, "side_lo": 64, "count": 1, "sigma": 0.0,
         "dtype": "f32", "jacobi": False, "tol": 1e-6, "guess": False},
        # one system of ordinary size at the tolerance of the solver benchmark
        {"name": "solve_one_300", "kind": "solve", "dims": 2, "side": 300, "side_lo": 300, "count": 1, "sigma": 0.0,
         "dtype": "f32", "jacobi": True, "tol": 1e-4, "guess": False},
        # the large single system: 1024 x 1024 Poisson, Jacobi, to 1e-6
        {"name": "solve_one_1024", "kind": "solve", "dims": 2, "side": 1024, "side_lo": 1024, "count": 1, "sigma": 0.0,
         "dtype": "f32", "jacobi": True, "tol": 1e-6, "guess": False},
        # many uneven systems in one call, single precision throughout
        {"name": "solve_batch_f32", "kind": "solve", "dims": 2, "side": 128, "side_lo": 16, "count": 1024, "sigma": 0.5,
         "dtype": "f32", "jacobi": True, "tol": 1e-6, "guess": False},
        # the same family in double precision
        {"name": "solve_batch_f64", "kind": "solve", "dims": 2, "side": 128, "side_lo": 16, "count": 512, "sigma": 0.5,
         "dtype": "f64", "jacobi": True, "tol": 1e-12, "guess": False},
        # many uneven systems to FP64 accuracy with FP32 iterations (the
        # package's headline workload; the adjoint's default tolerance)
        {"name": "refined_batch", "kind": "refined", "dims": 2, "side": 128, "side_lo": 16, "count": 2048, "sigma": 0.5,
         "tol": 1e-12},
        # one ill-conditioned 3-D system to FP64 accuracy
        {"name": "refined_3d_64", "kind": "refined", "dims": 3, "side": 64, "side_lo": 64, "count": 1, "sigma": 1.0,
         "tol": 1e-12},
        # training through the solver: 256 value sets on one 128 x 128 pattern,
        # gradients with respect to matrix values and right-hand sides
        {"name": "adjoint_256x128", "kind": "adjoint", "side": 128, "batches": 256, "sigma": 0.5, "tol": 1e-11},
        # products with vectors, forward and transposed
        {"name": "product_csr_1024", "kind": "product", "side": 1024, "format": "csr", "transposed": False,
         "dtype": "f32", "batches": 1},
        {"name": "product_csr_t_2048", "kind": "product", "side": 2048, "format": "csr", "transposed": True,
         "dtype": "f32", "batches": 1},
        # vector-valued unknowns: 3 x 3 blocks on a 512 x 512 grid
        {"name": "blocked_512", "kind": "blocked", "side": 512, "tol": 1e-6},
        # the vector operations of a user's own iteration
        {"name": "vectors_1000003", "kind": "vectors", "n": 1000003, "batches": 4, "dtype": "f32"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["one", "one", "one", "batch", "batch", "refined", "refined", "cube", "adjoint", "product",
                       "product", "blocked", "vectors"])
    if kind == "one":
        f64 = rng.random() < 0.25
        side = _log_int(rng, 16, 512 if f64 else 1000)
        return {"kind": "solve", "dims": 2, "side": side, "side_lo": side, "count": 1,
                "sigma": rng.choice([0.0, 0.5]), "dtype": "f64" if f64 else "f32", "jacobi": rng.random() < 0.75,
                "tol": 1e-12 if f64 else rng.choice([1e-4, 1e-6]), "guess": rng.random() < 0.25}
    if kind == "batch":
        f64 = rng.random() < 0.4
        lo = _log_int(rng, 8, 64)
        return {"kind": "solve", "dims": 2, "side": _log_int(rng, lo + 1, 128), "side_lo": lo,
                "count": _log_int(rng, 16, 512 if f64 else 1500), "sigma": 0.5, "dtype": "f64" if f64 else "f32",
                "jacobi": True, "tol": 1e-12 if f64 else 1e-6, "guess": False}
    if kind == "refined":
        lo = _log_int(rng, 8, 64)
        return {"kind": "refined", "dims": 2, "side": _log_int(rng, lo + 1, 128), "side_lo": lo,
                "count": _log_int(rng, 16, 2500), "sigma": 0.5, "tol": 1e-12}
    if kind == "cube":
        side = _log_int(rng, 27, 96)
        return {"kind": "refined", "dims": 3, "side": side, "side_lo": side, "count": 1,
                "sigma": rng.choice([0.5, 1.0]), "tol": 1e-12}
    if kind == "adjoint":
        return {"kind": "adjoint", "side": _log_int(rng, 32, 128), "batches": _log_int(rng, 16, 256), "sigma": 0.5,
                "tol": 1e-11}
    if kind == "product":
        fmt = rng.choice(["csr", "csr", "csc", "ell"])
        return {"kind": "product", "side": _log_int(rng, 64, 2048), "format": fmt,
                "transposed": fmt != "ell" and rng.random() < 0.5, "dtype": rng.choice(["f32", "f32", "f64"]),
                "batches": rng.choice([1, 1, 3])}
    if kind == "blocked":
        return {"kind": "blocked", "side": _log_int(rng, 64, 512), "tol": 1e-6}
    return {"kind": "vectors", "n": _log_int(rng, 1000, 20000000), "batches": rng.choice([1, 2, 4, 7]),
            "dtype": rng.choice(["f32", "f32", "f64"])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

class _Grid:
    """Packed finite-volume systems: `idx` / `coef` (n, 2 dims + 1) hold the
    columns of every row in ascending order and their values rounded to FP32
    (0 where there is no neighbour, whose column is then the row's own),
    `mask` the entries that exist, `off` the first row of each system."""

    def __init__(self, dims, sides, sigma, seed, sets=1):
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        self.gen, self.dims = g, dims
        s = torch.tensor(sides, device="cuda", dtype=torch.int64)
        length = s ** dims
        self.off = torch.cat([length.new_zeros(1), length.cumsum(0)])
        n = self.n = int(self.off[-1])
        sys = torch.repeat_interleave(torch.arange(len(sides), device="cuda"), length, output_size=n)
        side, row = s[sys], torch.arange(n, device="cuda")
        local = row - self.off[sys]
        idx, mask, step = [row], [torch.ones(n, dtype=torch.bool, device="cuda")], torch.ones_like(side)
        faces, diag = [], 0.0
        for _ in range(dims):
            c = (local // step) % side
            up = torch.exp(sigma * torch.randn(sets, n, device="cuda", generator=g, dtype=torch.float64))
            edge = torch.exp(sigma * torch.randn(sets, n, device="cuda", generator=g, dtype=torch.float64))
            has_lo, has_hi = c > 0, c < side - 1
            lo, hi = torch.where(has_lo, row - step, row), torch.where(has_hi, row + step, row)
            down = torch.where(has_lo, up[:, lo], edge)
            diag = diag + up + down
            idx, mask = [lo] + idx + [hi], [has_lo] + mask + [has_hi]
            faces = [-down * has_lo] + faces + [-up * has_hi]
            step = step * side
        # (axes were added innermost first, so the columns are in ascending order)
        self.idx, self.mask = torch.stack(idx, 1), torch.stack(mask, 1)
        coef = faces[:dims] + [diag] + faces[dims:]
        self.coef = torch.stack(coef, 2).float()   # (sets, n, 2 dims + 1)
        self.row_ptr = torch.cat([self.off.new_zeros(1), self.mask.sum(1).cumsum(0)])

    def csr(self):
        return (self.row_ptr.to(torch.int32).cpu().numpy(), self.idx[self.mask].to(torch.int32).cpu().numpy())

    def values(self):
        """(sets, nnz) FP32 in CSR order."""
        return self.coef[:, self.mask]

    def uniform(self, *shape, dtype=torch.float32):
        return torch.rand(*shape, device="cuda", generator=self.gen, dtype=dtype) * 2 - 1

    # -- 64-bit arithmetic on the same numbers, without the package --

    def apply(self, x, coef=None):
        """A x in FP64; x (sets, n)."""
        c = self.coef if coef is None else coef
        return sum(c[:, :, k].double() * x[:, self.idx[:, k]] for k in range(self.idx.shape[1]))

    def solve(self, b):
        """A^-1 b in FP64: Jacobi-CG per system, restarted on the true residual."""
        lengths = self.off[1:] - self.off[:-1]

        def total(v):   # per-system sums, spread over the rows
            if lengths.numel() == 1:
                return v.sum(1, keepdim=True)
            t = torch.stack([torch.segment_reduce(u, "sum", lengths=lengths) for u in v])
            return torch.repeat_interleave(t, lengths, dim=1, output_size=self.n)

        b = b.double()
        inv = 1.0 / self.coef[:, :, self.dims].double()
        x, goal = torch.zeros_like(b), 1e-30 * total(b * b)
        for _ in range(3):
            r = b - self.apply(x)
            z = inv * r
            p, rz = z.clone(), total(r * z)
            for it in range(20000):
                q = self.apply(p)
                pq = total(p * q)
                alpha = torch.where(pq > 0, rz / pq, torch.zeros_like(pq))
                x += alpha * p
                r -= alpha * q
                z = inv * r
                new = total(r * z)
                p = z + torch.where(rz > 0, new / rz, torch.zeros_like(rz)) * p
                rz = new
                if it % 50 == 49 and bool((total(r * r) <= goal).all()):
                    break
        return x


def _sides(case):
    """Grid sides of the systems, a fixed uneven mix for a case (its values and
    right-hand sides come from the seed)."""
    if case["count"] == 1:
        return [case["side"]]
    rng = np.random.RandomState(case["side"] * 1009 + case["side_lo"])
    return [int(v) for v in rng.randint(case["side_lo"], case["side"] + 1, case["count"])]


def _system(case, seed):
    grid = _Grid(case["dims"], _sides(case), case["sigma"], seed)
    b = grid.uniform(grid.n, dtype=torch.float64)
    guess = grid.uniform(grid.n, dtype=torch.float64)
    return grid, b, guess


def _pattern(grid):
    row_ptr, col = grid.csr()
    pattern = cm.SparsityPattern.csr(grid.n, grid.n, row_ptr, col)
    if grid.off.numel() > 2:
        pattern.set_systems(grid.off.cpu().numpy())
    return pattern


_BLOCK = np.array([[4.0, 1.0, 0.5], [1.0, 5.0, 1.0], [0.5, 1.0, 6.0]], np.float32)   # a cell's own coupling


def _blocked(case, seed):
    grid = _Grid(2, [case["side"]], 0.5, seed)
    # block of entry (i, j): a_ij times the identity, plus the cell's coupling on the diagonal
    vals = grid.values()[0][:, None, None] * torch.eye(3, device="cuda")
    row = torch.repeat_interleave(torch.arange(grid.n, device="cuda"), grid.mask.sum(1))
    on_diagonal = grid.idx[grid.mask] == row
    vals = vals + on_diagonal[:, None, None] * torch.from_numpy(_BLOCK).cuda()
    return grid, vals.contiguous(), grid.uniform(3 * grid.n)


def _vectors(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    shape = (case["batches"], case["n"])
    return [torch.randn(shape, device="cuda", generator=g, dtype=_F[case["dtype"]]) for _ in range(3)]


def _product(case, seed):
    grid = _Grid(2, [case["side"]], 0.5, seed, sets=case["batches"])
    x = grid.uniform(case["batches"], grid.n, dtype=_F[case["dtype"]])
    return grid, x


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        grid, b, guess = _system(case, seed)
        dtype = _F[case["dtype"]]
        A = cm.SparseMatrix(_pattern(grid), dtype=dtype).setData(grid.values())
        cg = cm.ConjugateGradient(A, cm.DiagonalPreconditioner if case["jacobi"] else cm.IdentityPreconditioner)
        cg.setTolerance(case["tol"])
        return {"kind": kind, "cg": cg, "b": b.to(dtype), "guess": guess.to(dtype) if case["guess"] else None}
    if kind == "refined":
        grid, b, _ = _system(case, seed)
        A = cm.SparseMatrix(_pattern(grid)).setData(grid.values())
        return {"kind": kind, "cg": cm.ConjugateGradient(A), "b": b, "tol": case["tol"]}
    if kind == "adjoint":
        grid = _Grid(2, [case["side"]], case["sigma"], seed, sets=case["batches"])
        row_ptr, col = grid.csr()
        shape = (case["batches"], grid.n)
        return {"kind": kind, "op": SparseSolveOp(grid.n, row_ptr, col, tol=case["tol"]),
                "values": grid.values().double().requires_grad_(),
                "b": grid.uniform(*shape, dtype=torch.float64).requires_grad_(),
                "target": torch.randn(shape, device="cuda", generator=grid.gen, dtype=torch.float64)}
    if kind == "product":
        grid, x = _product(case, seed)
        row_ptr, col = grid.csr()
        values = grid.values()
        if case["format"] == "ell":
            ind = torch.where(grid.mask, grid.idx, -torch.ones_like(grid.idx)).cpu().numpy()
            pattern, values = cm.SparsityPattern.ell(grid.n, grid.n, ind), grid.coef
        elif case["format"] == "csc":   # the operator is symmetric: its CSR arrays are its CSC arrays
            pattern = cm.SparsityPattern.csc(grid.n, grid.n, row_ptr, col)
        else:
            pattern = cm.SparsityPattern.csr(grid.n, grid.n, row_ptr, col)
        A = cm.SparseMatrix(pattern, dtype=_F[case["dtype"]], batches=case["batches"]).setData(values)
        return {"kind": kind, "A": A, "x": x, "transposed": case["transposed"]}
    if kind == "blocked":
        grid, vals, b = _blocked(case, seed)
        row_ptr, col = grid.csr()
        A = cm.SparseMatrix(cm.SparsityPattern.bsr(grid.n, grid.n, 3, row_ptr, col)).setData(vals)
        return {"kind": kind, "cg": cm.ConjugateGradient(A).setTolerance(case["tol"]), "b": b}
    return {"kind": kind, "v": _vectors(case, seed)}


def run(state):
    kind = state["kind"]
    if kind == "solve":
        return state["cg"].solveWithGuess(state["b"], state["guess"])
    if kind == "refined":
        return state["cg"].solve_refined(state["b"], outer_tol=state["tol"], max_outer=100)
    if kind == "adjoint":
        x = sparse_solve(state["values"], state["b"], state["op"])
        d_values, d_b = torch.autograd.grad(x, (state["values"], state["b"]), x.detach() - state["target"])
        return {"x": x.detach(), "d_values": d_values, "d_b": d_b}
    if kind == "product":
        return state["A"].transposed_product(state["x"]) if state["transposed"] else state["A"] * state["x"]
    if kind == "blocked":
        return state["cg"].solve(state["b"])
    u, v, w = state["v"]
    return {"dot": cm.dot(u, v), "sum": cm.linear_combination([0.5, -1.25, 2.0], [u, v, w]),
            "over_batches": cm.reduce(u.unsqueeze(0), "sum", ("cols",))}


def _rows(case):
    side, lo = case["side"], case["side_lo"]
    return case["count"] * sum(s ** case["dims"] for s in range(lo, side + 1)) / (side - lo + 1)


def work(case):
    """Inputs read once and outputs written once; the multiplications and
    additions of one product with the matrix (a solve's iteration count is not
    known beforehand)."""
    kind = case["kind"]
    if kind in ("solve", "refined"):
        n = _rows(case)
        nnz = (2 * case["dims"] + 1) * n
        es = 4 if case.get("dtype") == "f32" else 8
        value = 8 if case.get("dtype") == "f64" else 4
        return {"bytes": nnz * (value + 4) + n * (4 + (3 if case.get("guess") else 2) * es), "flops": 2 * nnz}
    if kind == "adjoint":
        n = case["side"] ** 2
        return {"bytes": case["batches"] * (2 * 5 * n * 8 + 4 * n * 8) + n * 24, "flops": case["batches"] * 2 * 2 * 5 * n}
    if kind == "product":
        n, es = case["side"] ** 2, 8 if case["dtype"] == "f64" else 4
        nnz = 5 * n - 4 * case["side"]
        index = 4 * (5 * n if case["format"] == "ell" else nnz + n)
        return {"bytes": index + case["batches"] * es * (nnz + 2 * n), "flops": case["batches"] * 2 * nnz}
    if kind == "blocked":
        n = case["side"] ** 2
        return {"bytes": 5 * n * (36 + 4) + n * (4 + 24), "flops": 2 * 45 * n}
    es, n = 8 if case["dtype"] == "f64" else 4, case["batches"] * case["n"]
    return {"bytes": es * (4 * n + case["n"]), "flops": 8 * n}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------

def _poisson(b, side):
    """Solution of the 2-D Poisson system by its eigenvectors (sine transform)."""
    k = torch.arange(1, side + 1, device=b.device, dtype=torch.float64)
    s = math.sqrt(2.0 / (side + 1)) * torch.sin(math.pi / (side + 1) * k[:, None] * k[None, :])
    lam = 2 - 2 * torch.cos(math.pi * k / (side + 1))
    return (s @ ((s @ b.view(side, side) @ s) / (lam[:, None] + lam[None, :])) @ s).reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "refined"):
        grid, b, _ = _system(case, seed)
        b = b.to(_F[case.get("dtype", "f64")]).double()
        if case["count"] == 1 and case["sigma"] == 0.0:
            return _poisson(b, case["side"])
        return grid.solve(b[None])[0]
    if kind == "adjoint":
        grid = _Grid(2, [case["side"]], case["sigma"], seed, sets=case["batches"])
        shape = (case["batches"], grid.n)
        b = grid.uniform(*shape, dtype=torch.float64)
        target = torch.randn(shape, device="cuda", generator=grid.gen, dtype=torch.float64)
        x = grid.solve(b)
        lam = grid.solve(x - target)
        row = torch.repeat_interleave(torch.arange(grid.n, device="cuda"), grid.mask.sum(1))
        return {"x": x, "d_values": -lam[:, row] * x[:, grid.idx[grid.mask]], "d_b": lam}
    if kind == "product":
        grid, x = _product(case, seed)   # (a symmetric operator: A^T = A)
        return grid.apply(x.double())
    if kind == "blocked":
        grid, vals, b = _blocked(case, seed)
        # the operator is I (x) L + blkdiag(C): solved as its own CG in FP64
        own = vals.double()[grid.idx[grid.mask] == torch.repeat_interleave(
            torch.arange(grid.n, device="cuda"), grid.mask.sum(1))]   # (n, 3, 3) diagonal blocks
        coef = grid.coef.clone()
        coef[:, :, 2] = 0.0

        def apply(v):
            return grid.apply(v.T.contiguous(), coef.expand(3, -1, -1)).T + torch.einsum("nij,nj->ni", own, v)

        b = b.double().view(-1, 3)
        inv = 1.0 / torch.diagonal(own, dim1=1, dim2=2)
        x, goal = torch.zeros_like(b), 1e-30 * (b * b).sum()
        r = b.clone()
        p = inv * r
        rz = (r * p).sum()
        for _ in range(500):
            q = apply(p)
            alpha = rz / (p * q).sum()
            x += alpha * p
            r -= alpha * q
            if (r * r).sum() <= goal:
                break
            z = inv * r
            new = (r * z).sum()
            p = z + new / rz * p
            rz = new
        return x.reshape(-1)
    u, v, w = (t.double() for t in _vectors(case, seed))
    return {"dot": (u * v).sum(1), "sum": 0.5 * u - 1.25 * v + 2.0 * w, "over_batches": u.sum(0).view(1, 1, -1)}
