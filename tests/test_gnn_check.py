"""A tensor-core kernel that gave up waiting is an error where its results are read: the
validation loss and the predicted field.  On the CPU, with the library's flag and the
network's passes replaced."""
from types import SimpleNamespace

import numpy as np
import pytest

from op2b import gnn as G
from op2b import lib as L
from op2b import mesh as M
from op2b import warmstart as S

torch = pytest.importorskip("torch")


class Net:
    torch = SimpleNamespace(from_numpy=torch.from_numpy, bfloat16=torch.bfloat16,
                            float64=torch.float64,
                            empty=lambda *s, dtype, device: torch.zeros(*s, dtype=dtype))
    norm, stream = np.ones(8), 0
    check = G.GraphNet.check

    def upload_graph(self, g):
        return g

    def forward(self, dg, ni, ei, train):
        return torch.zeros(len(ni), G.OUT)

    def release(self):
        pass


@pytest.fixture
def flag(monkeypatch):
    f = SimpleNamespace(value=0)
    monkeypatch.setattr(G, "_lib", lambda: SimpleNamespace(op2b_gemm_error=lambda reset: f.value))
    monkeypatch.setattr(G, "_call", lambda *a: None)
    monkeypatch.setattr(torch.Tensor, "cuda", lambda self: self)
    return f


def _predict():
    return S.predict_q(Net(), M.channel_bump(6, 4, seed=0), 0.5, 1.0, 0.05)


def _evaluate():
    m = M.channel_bump(6, 4, seed=0)
    data = SimpleNamespace(g=G.cell_graph(m), n=2,
                           batch=lambda s, b: (torch.zeros(b * m.ncell, G.NODE_IN), None,
                                               torch.ones(b * m.ncell, 4)))
    return S.evaluate(Net(), data, batch=2)


def test_results_without_a_failure(flag):
    assert _predict().shape == (24, 4) and _evaluate() == 1.0


@pytest.mark.parametrize("what", [_predict, _evaluate])
def test_a_kernel_that_gave_up_is_an_error(flag, what):
    flag.value = 1
    with pytest.raises(L.Op2Error, match="gave up"):
        what()
