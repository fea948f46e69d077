"""TorchCR2D.voltages and dpred_from_fields on models of a wrong length (refused, as the sparse
products refuse them), and a single chargeability for all cells (taken for every cell)."""
import pytest
import torch

from simpeg_dc_torch_b200 import TorchCR2D
from simpeg_dc_torch_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine(cuda):
    mesh, survey, m = syn.tiny_2d()
    return TorchCR2D(mesh, survey, nky=7, device=cuda), torch.tensor(m, device=cuda)


@pytest.mark.parametrize("call", ["voltages", "dpred_from_fields"])
def test_wrong_lengths(engine, call):
    eng, m = engine
    chg = torch.full_like(m, 0.1)
    longer = lambda x: torch.cat([x, x[:1]])  # noqa: E731
    for mr, mi in ((m[:-1], chg[:-1]), (longer(m), longer(chg)), (m[:1], chg[:1]), (m[:1], chg)):
        with pytest.raises((ValueError, RuntimeError)):
            getattr(eng, call)(mr, mi)


def test_one_chargeability_for_all_cells(engine):
    eng, m = engine
    one = torch.tensor(0.1)
    V = eng.voltages(m, one)
    ref = eng.voltages(m, torch.full_like(m, one.item()))   # (0.1 as a float32)
    eng.check()
    assert float((V - ref).abs().max()) <= 1e-12 * float(ref.abs().max())


def test_first_order_gradient_under_create_graph(engine):
    eng, m = engine
    x = torch.cat([m, torch.full_like(m, 0.1)]).requires_grad_(True)
    phi = lambda: sum((d ** 2).sum() for d in eng.dpred(x))  # noqa: E731
    (ref,) = torch.autograd.grad(phi(), x)
    (g,) = torch.autograd.grad(phi(), x, create_graph=True)
    eng.check()
    assert float((g - ref).detach().abs().max()) <= 1e-12 * float(ref.abs().max())
