"""dct_tuning_default's panels per update block are those of the factorization schedule that a plan
of the type runs: with that block size its trailing updates have the schedule's tiles."""
import pytest

import schedule_replay as R
from simpeg_dc_torch_b200 import _native as nat
from test_blocked_update import wide_matrix


@pytest.mark.parametrize("dtype,which", [(0, 5), (1, 0), (2, 5)])
def test_update_block_is_the_schedules(dtype, which):
    A = wide_matrix(513, 9, 1)
    sym = nat.Symbolic(A.indptr, A.indices, None, 64)
    S = R.Struct(sym)
    tasks, launches = sym.schedule(dtype, which)
    block = nat.default_tuning(dtype)["update_block"]
    wide = max(range(S.nsuper), key=S.ns)
    ns, N = S.ns(wide), int(S.front_n[wide])
    assert ns > 4 * R.PANEL
    tile = R.TCTILE if dtype == 1 else R.UTILE
    for kind, _, first, count, p in launches:
        if kind != R.LUPDATE:
            continue
        got = max((t[3] for t in tasks[first:first + count] if t[0] == wide and t[2] >= 0),
                  default=-1) + 1
        if got == 0:
            continue
        base, (_, end) = min(ns, (p + 1) * R.PANEL), R.update_range(p, ns, N, block)
        origin = base & ~7 if dtype == 1 else base
        assert got == -(-(end - origin) // tile), (p, block)
