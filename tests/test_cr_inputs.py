"""TorchCR2D's products with the assembly map, without a GPU: the two kernels are stood in for by
recorders, so what is checked is what reaches them."""
from contextlib import contextmanager
from types import SimpleNamespace

import pytest
import torch

from simpeg_dc_torch_b200 import cr2d

NC, NNZ, NKY = 6, 9, 2


class Kernels:
    """Records the calls and the device that was made current around each; every output stays as
    it was allocated."""

    def __init__(self):
        self.calls, self.current = [], None

    def dct_csr_spmv(self, *args):
        self.calls.append(("dct_csr_spmv", self.current))
        return 0

    def dct_values_vjp(self, *args):
        self.calls.append(("dct_values_vjp", self.current))
        return 0

    @contextmanager
    def device(self, device):
        before, self.current = self.current, device
        yield
        self.current = before


@pytest.fixture
def kernels(monkeypatch):
    k = Kernels()
    monkeypatch.setattr(torch.cuda, "device", k.device)
    monkeypatch.setattr(cr2d.nat, "lib", lambda: k)
    monkeypatch.setattr(cr2d, "_stream_ptr", lambda device: 0)
    return k


def path():
    t = torch.zeros(1)
    return SimpleNamespace(nC=NC, nnzA=NNZ, nbatch=NKY, L_ptr=t, L_col=t, L_val=t, Lt_ptr=t,
                           Lt_col=t, Lt_val=t)


@pytest.mark.parametrize("n", [0, 1, NC - 1, NC + 1, 2 * NC])
def test_wrong_length_is_refused_before_any_launch(kernels, n):
    with pytest.raises(ValueError, match=f"{NC} cells"):
        cr2d._Values.apply(torch.zeros(n, dtype=torch.float64), path())
    assert kernels.calls == []


def test_kernels_run_on_the_tensors_device(kernels):
    x = torch.zeros(NC, dtype=torch.float64, requires_grad=True)
    cr2d._Values.apply(x, path()).sum().backward()
    assert kernels.calls == [("dct_csr_spmv", x.device), ("dct_values_vjp", x.device)]
    assert kernels.current is None


def test_second_order_is_refused(kernels):
    x = torch.zeros(NC, dtype=torch.float64, requires_grad=True)
    gy = torch.ones(NKY * NNZ, dtype=torch.float64, requires_grad=True)
    (gx,) = torch.autograd.grad(cr2d._Values.apply(x, path()), x, gy, create_graph=True)
    with pytest.raises(RuntimeError, match="once_differentiable"):
        gx.sum().backward()
