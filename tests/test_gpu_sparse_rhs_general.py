"""General plans whose forward pass is mostly large products: right-hand sides that reach only some
supernodes (dct_solve_permuted).

Tolerance: as in test_gpu_sparse_rhs, times four: two factors, pivots that grow by less than 2."""
import numpy as np
import pytest
import torch

from simpeg_dc_torch_b200 import make_batch_solver
from test_gpu_sparse_rhs import grid_systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 7, 66])
def test_reached_supernodes(cuda, k):
    nbatch = 2
    P, _ = grid_systems((14, 13, 13), 1, k)
    n = P.shape[0]
    A = np.where(P, np.random.default_rng(k).uniform(-1, 1, (nbatch, n, n)), 0.0)
    A[:, np.arange(n), np.arange(n)] = 0.0
    A /= max(np.abs(A).sum(1).max(), np.abs(A).sum(2).max())
    A[:, np.arange(n), np.arange(n)] = 2.0
    A = torch.tensor(A)
    crow = np.concatenate([[0], np.cumsum(P.sum(1))]).astype(np.int32)
    slv = make_batch_solver(torch.tensor(crow), torch.tensor(np.nonzero(P)[1].astype(np.int32)),
                            n, k, nbatch, device=cuda, dtype=torch.float64,
                            matrix_type="general", leaf_size=64)
    slv.factorize(A[:, torch.tensor(P)].to(cuda))
    info = slv.analysis()
    assert info["max_ns"] > 64
    bound = 4 * 4 * 8 * info["max_front"] * 2.0 ** -53
    perm = torch.as_tensor(slv._sym.array("perm").astype(np.int64))
    stream = torch.cuda.current_stream().cuda_stream
    dense = torch.randn(nbatch, n, k, dtype=torch.float64,
                        generator=torch.Generator().manual_seed(k))
    for rows in ([], [0], [n - 1], [0, 1, 13, 169], [5, n // 2, n - 7], list(range(n)), [0]):
        at = torch.tensor(rows, dtype=torch.int64)
        b = torch.zeros_like(dense).index_copy(1, at, dense[:, at])
        if rows == [0]:
            b[1] = 0.0                      # the systems reach different supernodes
        for shared in (False, True):
            bb = b[:1].expand(nbatch, n, k) if shared else b
            src = (bb[0] if shared else bb)[..., perm, :].contiguous().to(cuda)
            xp = torch.full((nbatch, n, k), float("nan"), dtype=torch.float64, device=cuda)
            slv.plan.solve_permuted(src.data_ptr(), int(not shared), k, xp.data_ptr(), stream)
            x = torch.empty_like(dense)
            x[:, perm] = xp.cpu()
            ref = torch.linalg.solve(A, bb)
            err = float(torch.linalg.norm(x - ref))
            assert err <= bound * float(torch.linalg.norm(ref)), (rows[:4], shared, err)
    slv.check()
