"""Pivots over the exponent range of a double.

Diagonal systems are exact: with d = sqrt(p) and r = 1 / d correctly rounded, a solve is r (r b),
each product rounded once, and every other term is a zero; so the solution has numpy's bits, also
for subnormal pivots.  Scaled systems: A and 2^e A have the same condition number, so the bound of
the unscaled ones (condition below 4: 4 * 8 n_front u) holds for both parities of e."""
import numpy as np
import pytest
import torch

from simpeg_dc_torch_b200 import make_solver
from test_gpu_sparse_rhs import grid_systems

pytestmark = pytest.mark.gpu


# unconnected unknowns, one single-CTA front of one and of several panels, and a front of several
# CTAs (values off the diagonal are zeros)
@pytest.mark.parametrize("n,dense", [(2000, False), (16, True), (100, True), (160, True),
                                     (500, True)])
@pytest.mark.parametrize("span", [(-1000, 1000), (-1060, -900), (-1, 1)])
def test_diagonal_systems_are_exact(cuda, n, dense, span):
    rng = np.random.default_rng(n + abs(span[1]))
    p = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(*span, size=n, endpoint=True))
    p[:3] = np.ldexp([1.0, 1.0, np.nextafter(4.0, 0.0)], [0, 1, 0])
    b = np.ldexp(rng.uniform(1.0, 2.0, n), -200)
    if dense:
        crow, col = np.arange(0, n * n + 1, n), np.tile(np.arange(n), n)
        vals = np.diag(p).ravel()
    else:
        crow, col, vals = np.arange(n + 1), np.arange(n), p
    slv = make_solver(torch.tensor(crow.astype(np.int32)), torch.tensor(col.astype(np.int32)), n, 1,
                      device=cuda, dtype=torch.float64, leaf_size=n if dense else 64)
    slv.factorize(torch.tensor(vals, device=cuda))
    x = slv.solve(torch.tensor(b, device=cuda)).cpu().numpy()
    slv.check()
    r = 1.0 / np.sqrt(p)
    np.testing.assert_array_equal(x, r * (r * b))


@pytest.mark.parametrize("e", [-400, -399, -1, 0, 1, 399, 400])
def test_scaled_systems(cuda, e):
    P, A = grid_systems((11, 10, 9), 1, 5)
    n = P.shape[0]
    crow = np.concatenate([[0], np.cumsum(P.sum(1))]).astype(np.int32)
    col = np.nonzero(P)[1].astype(np.int32)
    b = torch.randn(n, 3, dtype=torch.float64, generator=torch.Generator().manual_seed(3))
    slv = make_solver(torch.tensor(crow), torch.tensor(col), n, 3, device=cuda,
                      dtype=torch.float64, leaf_size=64)
    slv.factorize((A[0][torch.tensor(P)] * 2.0 ** e).to(cuda))
    x = slv.solve(b.to(cuda)).cpu() * 2.0 ** e
    slv.check()
    ref = torch.linalg.solve(A[0], b)
    bound = 4 * 8 * slv.analysis()["max_front"] * 2.0 ** -53
    assert float(torch.linalg.norm(x - ref) / torch.linalg.norm(ref)) <= bound
