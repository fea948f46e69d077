"""Single-CTA fronts at the edges of their blocks (16 columns), panels (64),
thread counts (fronts of 112 and fewer) and limits (160 float64, 224 float32,
112 complex128), against dense solves in float64.

Tolerances: Cholesky and the products with its inverses are backward stable
up to a modest multiple of n u, and the matrices have a condition number
below 4, so the relative error of a solution stays below 4 * 8 n u (u the unit
roundoff; twice that for complex arithmetic)."""
import numpy as np
import pytest
import torch

from simpeg_dc_torch_b200 import make_solver

pytestmark = pytest.mark.gpu

U = {torch.float64: 2.0 ** -53, torch.float32: 2.0 ** -24, torch.complex128: 2.0 ** -52}
LIMIT = {torch.float64: 160, torch.float32: 224, torch.complex128: 112}
SIZES = (1, 2, 7, 15, 16, 17, 31, 33, 48, 63, 64, 65, 80, 111, 112, 113, 128, 129, 159, 160,
         191, 193, 223, 224)


def dense_system(n, dtype, seed):
    """A symmetric matrix with its spectrum within [0.5, 2] times n (complex: plus a small
    symmetric imaginary part)."""
    rng = np.random.default_rng(seed)
    G = rng.standard_normal((n, n))
    G = (G + G.T) / 2
    A = n * np.eye(n) + 0.5 * n * G / max(1e-30, np.linalg.norm(G, 2))
    if dtype.is_complex:
        A = A + 0.1j * np.diag(np.diag(A)) + 0.1j * (A - np.diag(np.diag(A)))
    return A


def solver_for(pattern, dtype, k, cuda, leaf):
    n = pattern.shape[0]
    crow = np.concatenate([[0], np.cumsum(pattern.sum(1))]).astype(np.int32)
    col = np.nonzero(pattern)[1].astype(np.int32)
    return make_solver(torch.tensor(crow), torch.tensor(col), n, k, device=cuda, dtype=dtype,
                       refine=0, leaf_size=leaf)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32, torch.complex128])
def test_one_front_of_every_edge_size(cuda, dtype):
    for n in (m for m in SIZES if m <= LIMIT[dtype]):
        A = dense_system(n, dtype, n)
        b = np.random.default_rng(n + 1).standard_normal((n, 3)).astype(A.dtype)
        slv = solver_for(np.ones((n, n), bool), dtype, 3, cuda, max(n, 1))
        assert slv.analysis()["max_front"] == n
        At, bt = torch.tensor(A).to(dtype), torch.tensor(b).to(dtype)
        slv.factorize(At.reshape(-1).to(cuda))
        x = slv.solve(bt.to(cuda)).cpu()
        slv.check()
        wide = torch.complex128 if dtype.is_complex else torch.float64
        ref = torch.linalg.solve(At.to(wide), bt.to(wide))
        err = float(torch.linalg.norm(x.to(wide) - ref) / torch.linalg.norm(ref))
        assert err <= 4 * 8 * max(n, 4) * U[dtype], (n, err)


@pytest.mark.parametrize("shape", [(7, 5), (19, 17), (40, 23), (61, 33)])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32, torch.complex128])
def test_fronts_with_children(cuda, dtype, shape):
    """A grid's tree of fronts: assembly of the children and the Schur complements."""
    idx = np.arange(shape[0] * shape[1]).reshape(shape)
    n = idx.size
    P = np.eye(n, dtype=bool)
    for a, c in ((idx[1:], idx[:-1]), (idx[:, 1:], idx[:, :-1])):
        P[a.ravel(), c.ravel()] = P[c.ravel(), a.ravel()] = True
    rng = np.random.default_rng(n)
    A = np.where(P, rng.uniform(-0.25, 0.25, (n, n)), 0.0)
    A = (A + A.T) / 2
    np.fill_diagonal(A, 2.0)            # rows sum to at most 1 off the diagonal: condition < 4
    if dtype.is_complex:
        A = A + 0.1j * A
    b = rng.standard_normal((n, 5)).astype(A.dtype)
    At, bt = torch.tensor(A).to(dtype), torch.tensor(b).to(dtype)
    for leaf in (8, 64):
        slv = solver_for(P, dtype, 5, cuda, leaf)
        slv.factorize(At[torch.tensor(P)].to(cuda))
        x = slv.solve(bt.to(cuda)).cpu()
        slv.check()
        wide = torch.complex128 if dtype.is_complex else torch.float64
        ref = torch.linalg.solve(At.to(wide), bt.to(wide))
        err = float(torch.linalg.norm(x.to(wide) - ref) / torch.linalg.norm(ref))
        assert err <= 4 * 8 * max(shape) * 4 * U[dtype], (leaf, err)


@pytest.mark.parametrize("at", [0, 5, 15, 16, 40, 63, 64, 89])
def test_bad_pivot_is_reported_and_the_rest_is_solved(cuda, at):
    """A pivot that is not positive counts as 1: an unknown without couplings then returns its
    right-hand side, and the others are those of the remaining system."""
    n = 90
    A = dense_system(n, torch.float64, 3)
    A[at, :] = A[:, at] = 0.0
    A[at, at] = -2.0
    slv = solver_for(np.ones((n, n), bool), torch.float64, 1, cuda, n)
    b = np.random.default_rng(4).standard_normal(n)
    slv.factorize(torch.tensor(A.reshape(-1), device=cuda))
    x = slv.solve(torch.tensor(b, device=cuda)).cpu().numpy()
    with pytest.raises(Exception, match="factorization"):
        slv.check()
    A[at, at] = 1.0
    ref = np.linalg.solve(A, b)
    assert np.linalg.norm(x - ref) <= 4 * n * 8 * n * 2.0 ** -53 * np.linalg.norm(ref)


def test_general_front_of_every_edge_size(cuda):
    """L U of one front (float64, rows and columns dominated by the diagonal: pivots grow by less
    than 2 and the condition number stays below 4), A x = b and A^T x = b.  Tolerance as above,
    doubled for the two factors."""
    from simpeg_dc_torch_b200 import make_solver as make
    for n in (m for m in SIZES if m <= 160):
        rng = np.random.default_rng(n)
        A = rng.uniform(-1, 1, (n, n))
        np.fill_diagonal(A, 0.0)
        A = A / max(1e-30, np.abs(A).sum(0).max(), np.abs(A).sum(1).max()) + 2.0 * np.eye(n)
        b = rng.standard_normal((n, 3))
        crow = np.arange(0, n * n + 1, n).astype(np.int32)
        col = np.tile(np.arange(n), n).astype(np.int32)
        slv = make(torch.tensor(crow), torch.tensor(col), n, 3, device=cuda,
                   dtype=torch.float64, matrix_type="general", leaf_size=max(n, 1))
        slv.factorize(torch.tensor(A.reshape(-1), device=cuda))
        assert slv.static_pivots() == 0
        for t in (False, True):
            x = slv.solve(torch.tensor(b, device=cuda), transposed=t).cpu().numpy()
            ref = np.linalg.solve(A.T if t else A, b)
            err = np.linalg.norm(x - ref) / np.linalg.norm(ref)
            assert err <= 4 * 16 * max(n, 4) * 2.0 ** -53, (n, t, err)
        slv.check()
