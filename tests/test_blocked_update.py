"""The float64 plans' factorization schedule, whose trailing updates come in blocks of four
panels, replayed task by task on the CPU (forward and in reverse order)."""
import numpy as np
import pytest
import scipy.sparse as sp

import schedule_replay as R
from simpeg_dc_torch_b200 import _native as nat


def wide_matrix(nd, ng, seed):
    """A dense nd x nd block coupled to a small grid: one supernode of several panels."""
    rng = np.random.default_rng(seed)
    G = rng.standard_normal((nd, nd))
    T = sp.diags([-1.0, 2.0, -1.0], [-1, 0, 1], shape=(ng, ng))
    L = sp.kron(sp.eye(ng), T) + sp.kron(T, sp.eye(ng)) + 2.1 * sp.eye(ng * ng)
    C = sp.random(ng * ng, nd, density=0.02, random_state=seed) * 0.05
    A = sp.bmat([[L, C], [C.T, sp.csr_matrix(G @ G.T / nd + 4 * np.eye(nd))]]).tocsr()
    A = ((A + A.T) * 0.5).tocsr()
    A.sort_indices()
    return A


@pytest.mark.parametrize("nd", [200, 256, 321, 330, 513])
def test_blocked_schedule(nd):
    A = wide_matrix(nd, 9, nd)
    sym = nat.Symbolic(A.indptr, A.indices, None, 64)
    S = R.Struct(sym)
    tasks, launches = sym.schedule(0, 5)
    base, _ = sym.schedule(0, 0)
    assert len(tasks) <= len(base)
    fronts, dinv = np.zeros(S.front_total), {}
    for kind, lv, first, count, arg in launches:
        chunk = tasks[first:first + count]
        before, dbefore = fronts.copy(), dict(dinv)
        for order in (chunk, chunk[::-1]):
            fronts[:], d = before, {k: v.copy() for k, v in dbefore.items()}
            for tk in order:
                R._task_factor(S, kind, tk, fronts, A.data, arg, d, R.UTILE, 4)
            if order is chunk:
                first_result = fronts.copy()
        assert np.abs(fronts - first_result).max() <= 1e-9 * max(1.0, np.abs(fronts).max())
        dinv = d
    # L L^T of the widest supernode's pivot block against a dense factorization
    ref, _ = R.replay_factor(sym, S, A.data, 0)
    for s in range(S.nsuper):
        ns = S.ns(s)
        got, want = (np.tril(S.front(f, s)[:, :ns]) for f in (fronts, ref))
        assert np.abs(got - want).max() <= 1e-10 * np.abs(want).max()
