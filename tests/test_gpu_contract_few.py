"""The value-gradient contraction for few right-hand sides, at the edges of its lane groups (1 to
65 right-hand sides, odd and even; arrays at odd multiples of eight bytes) and of its runs of 32
entries (rows of 1 to 70 entries, fewer entries than a run), without scales.

Tolerance: both sides sum k products in double, so they differ by at most
2 k u sum |Y X| in every entry."""
import numpy as np
import pytest
import torch

from simpeg_dc_torch_b200 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 7, 8, 9, 16, 17, 18, 31, 32, 33, 34, 47, 48, 63, 64, 65])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("lengths", [(3,), (1, 2, 3, 4, 5, 6, 7, 8, 9, 31, 32, 33, 70),
                                     (9,) * 40])
def test_few(cuda, k, shift, lengths):
    rng = np.random.default_rng(k + len(lengths))
    nbatch, n = 2, max(len(lengths), 5)
    row = np.repeat(np.arange(len(lengths)), lengths).astype(np.int32)
    nnz = row.size
    t = lambda a: torch.as_tensor(a, device=cuda).contiguous()  # noqa: E731
    d_row, d_iperm = t(row), t(rng.permutation(n).astype(np.int32))
    d_col = t(rng.integers(0, n, nnz).astype(np.int32))
    Y, X = (t(rng.standard_normal(nbatch * n * k + 1))[shift:][:nbatch * n * k].view(nbatch, n, k)
            for _ in range(2))
    gv = torch.full((nbatch * nnz,), float("nan"), dtype=torch.float64, device=cuda)
    nat.check(nat.lib().dct_gather_contract(
        nbatch, n, nnz, k, d_row.data_ptr(), d_col.data_ptr(), d_iperm.data_ptr(), None,
        Y.data_ptr(), X.data_ptr(), gv.data_ptr(),
        torch.cuda.current_stream(cuda).cuda_stream), "dct_gather_contract")
    prod = Y[:, d_iperm[d_row.long()].long()] * X[:, d_iperm[d_col.long()].long()]
    err = (gv.view(nbatch, nnz) + prod.sum(-1)).abs()
    assert bool((err <= 2 * k * 2.0 ** -53 * prod.abs().sum(-1)).all())
