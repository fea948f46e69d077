"""The factorization's profile (dct_plan_profile): every interval that is timed holds a launch, and
the assembly of large fronts is credited where it runs."""
import pytest
import scipy.sparse as sp
import torch

import schedule_replay as R
from simpeg_dc_torch_b200 import make_solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32, torch.complex128])
def test_assembly_is_counted_where_it_runs(cuda, dtype):
    T = [sp.diags([-1.0, 2.2, -1.0], [-1, 0, 1], shape=(m, m)) for m in (21, 19, 18)]
    E = [sp.eye(t.shape[0]) for t in T]
    A = (sp.kron(sp.kron(T[0], E[1]), E[2]) + sp.kron(sp.kron(E[0], T[1]), E[2])
         + sp.kron(sp.kron(E[0], E[1]), T[2])).tocsr()
    A.sort_indices()
    slv = make_solver(torch.tensor(A.indptr), torch.tensor(A.indices), A.shape[0], 1,
                      device=cuda, dtype=dtype, leaf_size=64)
    vals = torch.tensor(A.data).to(dtype).to(cuda)
    slv.factorize(vals)
    slv.plan.profile(True)
    slv.factorize(vals)
    got = slv.plan.profile_read()
    slv.plan.profile(False)
    slv.check()
    S = R.Struct(slv._sym)
    code = {torch.float64: 0, torch.float32: 1, torch.complex128: 2}[dtype]
    size = {0: 8, 1: 4, 2: 16}[code]
    tasks, launches = slv._sym.schedule(code, 0 if code == 1 else 5)
    third = [L for L in launches if L[0] == R.LEXTEND and L[4] >= 2 and L[3] > 0]
    assert got["extend_add"][1] == len(third)
    want = 0.0
    fronts = [tasks[L[2] + q][0] for L in launches if L[0] == R.LSCATTER for q in range(L[3])]
    assert fronts
    for s in fronts:
        N = float(S.front_n[s])
        want += float(S.amap_ptr[s + 1] - S.amap_ptr[s]) * (3 * size + 8) + size * N * (N + 1) / 2
        for c in S.child[S.child_ptr[s]:S.child_ptr[s + 1]][:2]:
            nb = float(S.front_n[c]) - S.ns(c)
            want += size * nb * (nb + 1) / 2
    assert got["large_scatter"][3] == pytest.approx(want, rel=1e-12)
