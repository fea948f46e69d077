"""Leaves that take their right-hand sides from the caller's array (float64 plans of 2-D grids,
dct_solve_permuted): one array for all systems or one per system, in place, with the array at an
odd multiple of eight bytes, for odd and even counts; the array is unchanged unless it is the
solution.

Tolerance: the condition number is below 4 and the relative error below 4 * 8 n_front u (general
plans four times that: two factors, pivots that grow by less than 2)."""
import numpy as np
import pytest
import torch

from simpeg_dc_torch_b200 import make_batch_solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["spd", "general"])
@pytest.mark.parametrize("shape,leaf", [((31, 22), 48), ((9, 5), 64), ((1, 40), 6)])
def test_leaf_rows(cuda, kind, shape, leaf):
    nbatch = 3
    idx = np.arange(shape[0] * shape[1]).reshape(shape)
    n = idx.size
    P = np.eye(n, dtype=bool)
    for a, c in ((idx[1:], idx[:-1]), (idx[:, 1:], idx[:, :-1])):
        P[a.ravel(), c.ravel()] = P[c.ravel(), a.ravel()] = True
    A = np.where(P, np.random.default_rng(n).uniform(-1, 1, (nbatch, n, n)), 0.0)
    if kind == "spd":
        A = A + A.transpose(0, 2, 1)
    A[:, np.arange(n), np.arange(n)] = 0.0
    A /= max(np.abs(A).sum(1).max(), np.abs(A).sum(2).max())
    A[:, np.arange(n), np.arange(n)] = 2.0
    A = torch.tensor(A).to(cuda)
    counts = (1, 6, 33, 66)
    crow = np.concatenate([[0], np.cumsum(P.sum(1))]).astype(np.int32)
    slv = make_batch_solver(torch.tensor(crow), torch.tensor(np.nonzero(P)[1].astype(np.int32)),
                            n, max(counts), nbatch, device=cuda, dtype=torch.float64,
                            matrix_type=kind, leaf_size=leaf)
    slv.factorize(A[:, torch.tensor(P).to(cuda)])
    bound = 4 * 8 * slv.analysis()["max_front"] * 2.0 ** -53 * (4 if kind == "general" else 1)
    perm = torch.as_tensor(slv._sym.array("perm").astype(np.int64), device=cuda)
    gen = torch.Generator(device=cuda).manual_seed(n)
    st = torch.cuda.current_stream().cuda_stream
    for k in counts:
        dense = torch.randn(nbatch, n, k, dtype=torch.float64, generator=gen, device=cuda)
        few = torch.zeros_like(dense)
        few[:, [0, n // 3, n - 1]] = dense[:, [0, n // 3, n - 1]]
        for b in (dense, few):
            for shared in (False, True):
                bb = b[:1].expand_as(b) if shared else b
                ref = torch.linalg.solve(A, bb)
                rows = (bb[0] if shared else bb)[..., perm, :].contiguous()
                for shift in (0, 1):
                    src = torch.zeros(rows.numel() + shift, dtype=torch.float64, device=cuda)
                    src[shift:] = rows.ravel()
                    for in_place in ((False,) if shared else (False, True)):
                        x = src if in_place else torch.full((nbatch * n * k + shift,), float("nan"),
                                                            dtype=torch.float64, device=cuda)
                        slv.plan.solve_permuted(src.data_ptr() + 8 * shift, int(not shared), k,
                                                x.data_ptr() + 8 * shift, st)
                        if not in_place:
                            assert torch.equal(src[shift:], rows.ravel())
                        got = torch.empty_like(ref)
                        got[:, perm] = x[shift:].view(nbatch, n, k)
                        err = float(torch.linalg.norm(got - ref) / torch.linalg.norm(ref))
                        assert err <= bound, (k, shared, shift, in_place, err)
    slv.check()
