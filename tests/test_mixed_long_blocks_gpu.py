"""Mixed precision at block sizes past the tensor-core products' longest
contraction (576): those products run on the FP64 pipe, none of them in place."""

import numpy as np
import pytest
import torch

import oracle
import serinv_gb300 as sg
from serinv_gb300.synthetic import generate

pytestmark = pytest.mark.gpu


def dev(arrays):
    return [torch.from_numpy(x.copy()).cuda() for x in arrays]


def close(x, y, tol):
    x = x.cpu().numpy()
    y = y if isinstance(y, np.ndarray) else y.cpu().numpy()
    return np.linalg.norm(x - y) <= tol * max(np.linalg.norm(y), 1e-300)


# 576: the last size with the tensor-core form (2.6e-12 off there)
@pytest.mark.parametrize("b,a", [(576, 3), (577, 0), (650, 5)])
def test_mixed(b, a):
    m = generate(3, b, a, 1, seed=b + a)
    d, ref = dev(m.arrays()), [x.copy() for x in m.arrays()]
    sg.pobtaf(*d, precision="mixed")
    oracle.pobtaf(*ref)
    assert all(close(x, y, 1e-10) for x, y in zip(d, ref))
    sg.pobtasi(*d, precision="mixed")
    oracle.pobtasi(*ref)
    assert all(close(x, y, 1e-9) for x, y in zip(d, ref))


def test_mixed_with_buffer():
    m = generate(4, 600, 7, 1, seed=3)
    out = []
    for precision in ("fp64", "mixed"):
        d = dev(m.arrays())
        buf = torch.zeros_like(d[0])
        sg.pobtaf(*d, buffer=buf, precision=precision)
        out.append([x[1:-1] if x.ndim == 3 else x for x in d])
    assert all(close(x, y, 1e-10) for x, y in zip(out[1], out[0]))
