"""Substitution of the single-panel supernodes at the edges of their tiles: right-hand-side
counts around 8, 16, 32 and 64 (and odd ones, whose rows are not 16-byte aligned), supernodes
narrower and wider than a fragment, and right-hand sides that are zero on whole subtrees.

Tolerance: the condition number of the matrices is below 4 and the substitution with
explicit inverses is backward stable up to a modest multiple of the front order, so the relative
error stays below 4 * 8 n_front u (u the unit roundoff; doubled for complex arithmetic)."""
import numpy as np
import pytest
import torch

from simpeg_dc_torch_b200 import make_batch_solver

pytestmark = pytest.mark.gpu

U = {torch.float64: 2.0 ** -53, torch.float32: 2.0 ** -24, torch.complex128: 2.0 ** -52}


def grid_system(shape, dtype, nbatch, seed):
    idx = np.arange(shape[0] * shape[1]).reshape(shape)
    n = idx.size
    P = np.eye(n, dtype=bool)
    for a, c in ((idx[1:], idx[:-1]), (idx[:, 1:], idx[:, :-1])):
        P[a.ravel(), c.ravel()] = P[c.ravel(), a.ravel()] = True
    rng = np.random.default_rng(seed)
    A = np.where(P, rng.uniform(-0.25, 0.25, (nbatch, n, n)), 0.0)
    A = (A + A.transpose(0, 2, 1)) / 2
    A[:, np.arange(n), np.arange(n)] = 2.0   # condition number below 4
    if dtype.is_complex:
        A = A + 0.1j * A
    crow = np.concatenate([[0], np.cumsum(P.sum(1))]).astype(np.int32)
    col = np.nonzero(P)[1].astype(np.int32)
    return P, crow, col, torch.tensor(A).to(dtype)


def check(slv, A, P, b, cuda, bound):
    wide = torch.complex128 if A.dtype.is_complex else torch.float64
    x = slv.solve(b.to(cuda)).cpu().to(wide)
    slv.check()
    ref = torch.linalg.solve(A.to(wide), b.to(wide) if b.dim() == 3 else
                             b.to(wide).expand(A.shape[0], *b.shape))
    scale = torch.linalg.norm(ref)
    assert float(torch.linalg.norm(x - ref)) <= bound * float(scale), tuple(b.shape)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32, torch.complex128])
@pytest.mark.parametrize("leaf", [4, 30, 64])
def test_right_hand_side_counts(cuda, dtype, leaf):
    P, crow, col, A = grid_system((23, 14), dtype, 2, leaf)
    slv = make_batch_solver(torch.tensor(crow), torch.tensor(col), P.shape[0], 140, 2,
                            device=cuda, dtype=dtype, refine=0, leaf_size=leaf)
    slv.factorize(A[:, torch.tensor(P)].to(cuda))
    bound = 4 * 8 * slv.analysis()["max_front"] * U[dtype]
    gen = torch.Generator().manual_seed(7)
    for k in (1, 2, 7, 8, 9, 15, 16, 17, 24, 31, 32, 33, 48, 63, 64, 65, 68, 96, 97, 130, 140):
        b = torch.randn(2, P.shape[0], k, dtype=dtype, generator=gen)
        check(slv, A, P, b, cuda, bound)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32, torch.complex128])
def test_right_hand_sides_that_are_zero_on_subtrees(cuda, dtype):
    P, crow, col, A = grid_system((40, 23), dtype, 2, 5)
    n = P.shape[0]
    slv = make_batch_solver(torch.tensor(crow), torch.tensor(col), n, 70, 2, device=cuda,
                            dtype=dtype, refine=0, leaf_size=16)
    slv.factorize(A[:, torch.tensor(P)].to(cuda))
    bound = 4 * 8 * slv.analysis()["max_front"] * U[dtype]
    for k in (5, 70):
        b = torch.zeros(n, k, dtype=dtype)
        b[torch.arange(k) * 11 % n, torch.arange(k)] = 1.0     # one source per column
        b[(torch.arange(k) * 17 + 3) % n, torch.arange(k)] -= 1.0
        check(slv, A, P, b, cuda, bound)
    b = torch.zeros(n, 5, dtype=dtype)
    b[n // 2, 3] = -0.0                                         # nothing at all
    assert float(slv.solve(b.to(cuda)).abs().max()) == 0.0
    b[3, 1] = float("nan")                                      # a NaN is not a zero
    x = slv.solve(b.to(cuda)).cpu()
    assert bool(torch.isnan(x[:, 3, 1]).all()) and float(x[:, :, [0, 2, 3, 4]].abs().max()) == 0.0


def test_long_boundary(cuda):
    """A panel with more boundary rows than the row indices kept at a time: two blocks of 40
    unknowns that only a dense block of 1,300 connects."""
    m, q = 40, 1300
    n = 2 * m + q
    P = np.zeros((n, n), bool)
    P[:m, :m] = P[m:2 * m, m:2 * m] = P[2 * m:, :] = P[:, 2 * m:] = True
    rng = np.random.default_rng(1)
    A = np.where(P, 0.25 * rng.uniform(-1, 1, (n, n)) / np.sqrt(n), 0.0)
    A = (A + A.T) / 2 + 2.0 * np.eye(n)
    crow = np.concatenate([[0], np.cumsum(P.sum(1))]).astype(np.int32)
    col = np.nonzero(P)[1].astype(np.int32)
    slv = make_batch_solver(torch.tensor(crow), torch.tensor(col), n, 9, 1, device=cuda,
                            dtype=torch.float64)
    ns = np.diff(slv._sym.array("sn_first"))
    assert (slv._sym.array("front_n") - ns)[ns <= 64].max() > 1024
    At = torch.tensor(A)[None]
    slv.factorize(At[:, torch.tensor(P)].to(cuda))
    gen = torch.Generator().manual_seed(3)
    check(slv, At, P, torch.randn(1, n, 9, dtype=torch.float64, generator=gen), cuda,
          4 * 8 * n * U[torch.float64])


@pytest.mark.parametrize("shape", [(23, 14), (34, 33)])
def test_refined_right_hand_side_counts(cuda, shape):
    """Float32 plans with two corrections: rows of k right-hand sides that are and are not a
    multiple of four (the work buffers pad them) and of two (16-byte rows).  With a condition
    number below 4 the first correction already leaves less than (30 n_front u)^2, so what
    remains is the rounding of the result: 2^-24, bounded here by twice that."""
    P, crow, col, A = grid_system(shape, torch.float32, 2, 11)
    n = P.shape[0]
    slv = make_batch_solver(torch.tensor(crow), torch.tensor(col), n, 70, 2, device=cuda,
                            dtype=torch.float32)
    slv.factorize(A[:, torch.tensor(P)].to(cuda))
    gen = torch.Generator().manual_seed(5)
    for k in (1, 2, 3, 4, 5, 6, 7, 65, 66, 67, 68, 70):
        check(slv, A, P, torch.randn(2, n, k, generator=gen), cuda, 2.0 ** -23)
        check(slv, A, P, torch.randn(n, k, generator=gen), cuda, 2.0 ** -23)
