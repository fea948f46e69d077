"""Fronts of several CTAs and supernodes of several panels (float64, complex and general
plans) at the edges of their tiles: right-hand-side counts around the tile widths, panels and
boundaries that are not multiples of 16 or 64, blocks of four panels and remainders.

Tolerance: the condition number of the matrices is below 4, and factorization and
substitution are backward stable up to a modest multiple of the front order, so the relative
error stays below 4 * 8 n_front u (doubled for complex arithmetic, and for the two factors of a
general plan, whose pivots grow by less than 2 on these diagonally dominant matrices)."""
import numpy as np
import pytest
import torch

from simpeg_dc_torch_b200 import make_batch_solver

pytestmark = pytest.mark.gpu

KINDS = {"spd": (torch.float64, 2.0 ** -53), "symmetric": (torch.complex128, 2.0 ** -52),
         "general": (torch.float64, 2.0 ** -51)}


def system(P, kind, nbatch, seed):
    """Diagonally dominant systems on the pattern P: every row sums to half its diagonal."""
    n = P.shape[0]
    rng = np.random.default_rng(seed)
    A = np.where(P, rng.uniform(-1, 1, (nbatch, n, n)), 0.0)
    if kind != "general":
        A = A + A.transpose(0, 2, 1)
    d = np.arange(n)
    A[:, d, d] = 0.0
    scale = max(np.abs(A).sum(1).max(), np.abs(A).sum(2).max())
    A = A / scale
    A[:, d, d] = 2.0
    return A * (1.0 + 0.1j) if kind == "symmetric" else A


def run(P, kind, cuda, counts, seed, nbatch=2, leaf=64):
    dtype, u = KINDS[kind]
    A = torch.tensor(system(P, kind, nbatch, seed))
    n = P.shape[0]
    crow = np.concatenate([[0], np.cumsum(P.sum(1))]).astype(np.int32)
    col = np.nonzero(P)[1].astype(np.int32)
    slv = make_batch_solver(torch.tensor(crow), torch.tensor(col), n, max(counts), nbatch,
                            device=cuda, dtype=dtype, matrix_type=kind, leaf_size=leaf)
    slv.factorize(A[:, torch.tensor(P)].to(cuda))
    info = slv.analysis()
    bound = 4 * 8 * info["max_front"] * u
    gen = torch.Generator().manual_seed(seed)
    for k in counts:
        b = torch.randn(nbatch, n, k, dtype=dtype, generator=gen)
        for transposed in ((False, True) if kind == "general" else (False,)):
            x = slv.solve(b.to(cuda), transposed=transposed).cpu()
            ref = torch.linalg.solve(A.transpose(1, 2) if transposed else A, b)
            err = float(torch.linalg.norm(x - ref) / torch.linalg.norm(ref))
            assert err <= bound, (k, transposed, err)
    slv.check()
    return info


@pytest.mark.parametrize("kind", list(KINDS))
def test_grid(cuda, kind):
    idx = np.arange(14 * 13 * 13).reshape(14, 13, 13)
    P = np.eye(idx.size, dtype=bool)
    for a, c in ((idx[1:], idx[:-1]), (idx[:, 1:], idx[:, :-1]), (idx[:, :, 1:], idx[:, :, :-1])):
        P[a.ravel(), c.ravel()] = P[c.ravel(), a.ravel()] = True
    info = run(P, kind, cuda, (1, 3, 8, 9, 16, 17, 31, 32, 33, 63, 64, 65, 72, 100, 129, 130), 1)
    assert info["max_front"] > 160 and info["max_ns"] > 64


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("nd", [225, 257, 319, 513, 650])
def test_one_wide_supernode(cuda, kind, nd):
    """A dense block: one front of nd columns and no boundary, plus a few rows above it."""
    n = nd + 6
    P = np.ones((n, n), bool)
    P[:3, 3:6] = P[3:6, :3] = False          # two small blocks only the dense one connects
    info = run(P, kind, cuda, (1, 7, 40, 66), nd, nbatch=1, leaf=4)
    assert info["max_ns"] > 160


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("blocks,m,core", [(2, 30, 200), (3, 33, 230), (5, 20, 200), (7, 9, 300)])
def test_front_with_many_children(cuda, kind, blocks, m, core):
    """Dense blocks that only a dense core connects: one large front assembled from one, two or
    more children (the first two in one pass, the others one by one)."""
    n = blocks * m + core
    P = np.zeros((n, n), bool)
    for i in range(blocks):
        P[i * m:(i + 1) * m, i * m:(i + 1) * m] = True
    P[blocks * m:, :] = P[:, blocks * m:] = True
    run(P, kind, cuda, (1, 20), blocks, nbatch=2, leaf=8)
