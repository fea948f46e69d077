"""Single-panel supernodes whose thread blocks go through several chunks of right-hand sides:
many small systems, so that the launches are large enough, with dense right-hand sides and with
chunks that are zero before, between and after others.

Tolerance: the condition number is below 4 and the relative error of a float64 solve below
4 * 8 n_front u (complex: twice); a float32 plan refines to 1e-10."""
import numpy as np
import pytest
import torch

from simpeg_dc_torch_b200 import make_batch_solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,kind", [(torch.float64, "spd"), (torch.float32, "spd"),
                                        (torch.float64, "general"),
                                        (torch.complex128, "symmetric")])
@pytest.mark.parametrize("nbatch", [180, 700])
def test_chunks(cuda, dtype, kind, nbatch):
    idx = np.arange(8 * 7).reshape(8, 7)
    n = idx.size
    P = np.eye(n, dtype=bool)
    for a, c in ((idx[1:], idx[:-1]), (idx[:, 1:], idx[:, :-1])):
        P[a.ravel(), c.ravel()] = P[c.ravel(), a.ravel()] = True
    A = np.where(P, np.random.default_rng(nbatch).uniform(-1, 1, (nbatch, n, n)), 0.0)
    if kind != "general":
        A = A + A.transpose(0, 2, 1)
    A[:, np.arange(n), np.arange(n)] = 0.0
    A /= max(np.abs(A).sum(1).max(), np.abs(A).sum(2).max())
    A[:, np.arange(n), np.arange(n)] = 2.0
    wide = torch.complex128 if dtype == torch.complex128 else torch.float64
    A = torch.tensor(A).to(wide) * (1 + 0.1j if dtype == torch.complex128 else 1)
    A = A.to(cuda)
    counts = (33, 64, 65, 97, 187)
    crow = np.concatenate([[0], np.cumsum(P.sum(1))]).astype(np.int32)
    slv = make_batch_solver(torch.tensor(crow), torch.tensor(np.nonzero(P)[1].astype(np.int32)),
                            n, max(counts), nbatch, device=cuda, dtype=dtype, matrix_type=kind,
                            leaf_size=14)
    slv.factorize(A[:, torch.tensor(P).to(cuda)])
    bound = 4 * 8 * slv.analysis()["max_front"] * 2.0 ** -53 * (1 if wide == torch.float64 else 2)
    if kind == "general":
        bound *= 4                       # the two factors, pivots that grow by less than 2
    if dtype == torch.float32:
        bound = 1e-10
    iperm = torch.empty(n, dtype=torch.int64, device=cuda)
    iperm[torch.as_tensor(slv._sym.array("perm").astype(np.int64), device=cuda)] = \
        torch.arange(n, device=cuda)

    def solve(rhs):
        if kind != "spd":
            return slv.solve(rhs)
        # float64 on both sides, also for a float32 plan (whose solve takes and returns float32)
        bp, xp = torch.empty_like(rhs), torch.empty_like(rhs)
        bp[:, iperm] = rhs
        slv.plan.solve_permuted(bp.data_ptr(), 1, rhs.shape[-1], xp.data_ptr(),
                                torch.cuda.current_stream().cuda_stream)
        return xp[:, iperm]

    gen = torch.Generator(device=cuda).manual_seed(nbatch)
    for k in counts:
        b = torch.randn(nbatch, n, k, dtype=wide, generator=gen, device=cuda)
        sparse = torch.zeros_like(b)
        sparse[:, 3, 32:34] = 1.0
        sparse[:, n - 1, k - 1] = -2.0
        sparse[::2, n // 2, 0] = 0.5
        for rhs in (b, sparse):
            x = solve(rhs)
            ref = torch.linalg.solve(A, rhs)
            err = float(torch.linalg.norm(x - ref) / torch.linalg.norm(ref))
            assert err <= bound, (k, err)
    slv.check()
