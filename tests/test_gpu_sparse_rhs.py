"""Right-hand sides that reach only some supernodes (dct_solve_permuted): one electrode, one
corner, none at all, and dense ones, shared by the systems or one set per system, in place where
that is allowed.

Tolerance: as for the fronts of several CTAs, the condition number is below 4 and the relative
error of a float64 solve below 4 * 8 n_front u; a float32 plan refines to 1e-10."""
import numpy as np
import pytest
import torch

from simpeg_dc_torch_b200 import make_batch_solver

pytestmark = pytest.mark.gpu


def grid_systems(shape, nbatch, seed):
    idx = np.arange(int(np.prod(shape))).reshape(shape)
    n = idx.size
    P = np.eye(n, dtype=bool)
    for a, c in ((idx[1:], idx[:-1]), (idx[:, 1:], idx[:, :-1]), (idx[:, :, 1:], idx[:, :, :-1])):
        P[a.ravel(), c.ravel()] = P[c.ravel(), a.ravel()] = True
    A = np.where(P, np.random.default_rng(seed).uniform(-1, 1, (nbatch, n, n)), 0.0)
    A = A + A.transpose(0, 2, 1)
    A[:, np.arange(n), np.arange(n)] = 0.0
    A /= np.abs(A).sum(1).max()
    A[:, np.arange(n), np.arange(n)] = 2.0
    return P, torch.tensor(A)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("k", [1, 7, 66])
def test_reached_supernodes(cuda, dtype, k):
    nbatch = 2
    P, A = grid_systems((14, 13, 13), nbatch, k)
    n = P.shape[0]
    crow = np.concatenate([[0], np.cumsum(P.sum(1))]).astype(np.int32)
    slv = make_batch_solver(torch.tensor(crow), torch.tensor(np.nonzero(P)[1].astype(np.int32)),
                            n, k, nbatch, device=cuda, dtype=dtype, leaf_size=64)
    slv.factorize(A[:, torch.tensor(P)].to(cuda))
    info = slv.analysis()
    assert info["max_ns"] > 64
    bound = 1e-10 if dtype == torch.float32 else 4 * 8 * info["max_front"] * 2.0 ** -53
    iperm = torch.empty(n, dtype=torch.int64)
    perm = torch.as_tensor(slv._sym.array("perm").astype(np.int64))
    iperm[perm] = torch.arange(n)
    gen = torch.Generator().manual_seed(k)
    stream = torch.cuda.current_stream().cuda_stream
    dense = torch.randn(nbatch, n, k, dtype=torch.float64, generator=gen)
    sparse = {"none": [], "first": [0], "last": [n - 1], "corner": [0, 1, 13, 169],
              "three": [5, n // 2, n - 7]}
    cases = [torch.zeros_like(dense).index_copy(1, torch.tensor(r, dtype=torch.int64), dense[:, r])
             for r in sparse.values()]
    for q, b in enumerate([dense] + cases + [dense]):
        if b is cases[-1]:
            b[1] = 0.0                      # the systems reach different supernodes
        for shared in (False, True):
            bb = b[:1].expand(nbatch, n, k) if shared else b
            ref = torch.linalg.solve(A, bb)
            bp = torch.empty_like(b).to(cuda)
            bp[:, iperm.to(cuda)] = bb.to(cuda)
            src = bp[0].contiguous() if shared else bp
            for in_place in ((False, True) if not shared and dtype == torch.float64 else (False,)):
                xp = src if in_place else torch.full_like(bp, float("nan"))
                slv.plan.solve_permuted(src.data_ptr(), int(not shared), k, xp.data_ptr(), stream)
                x = xp[:, iperm.to(cuda)].cpu()
                err = float(torch.linalg.norm(x - ref))
                assert err <= bound * float(torch.linalg.norm(ref)), (q, shared, in_place, err)
    slv.check()
