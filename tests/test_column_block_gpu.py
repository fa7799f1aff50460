"""Column blocks whose trailing update takes several rounds of the workers, in
whole and in half tiles, with the rows dealt out evenly and unevenly, against
the oracle."""

import numpy as np
import pytest
import torch

import oracle
import serinv_gb300 as sg
from serinv_gb300.synthetic import generate

pytestmark = pytest.mark.gpu


# (152 SMs leave 142 workers: b = 256 stays within one round, b = 650 starts with five)
@pytest.mark.parametrize("b,a", [(256, 0), (289, 31), (416, 97), (512, 64), (650, 5)])
@pytest.mark.parametrize("dtype,precision,tol", [(np.float64, "fp64", 1e-12), (np.float64, "mixed", 1e-9), (np.float32, "fp64", 1e-5)])
def test_update_rounds(b, a, dtype, precision, tol):
    m = generate(2, b, a, 1, seed=b + a, dtype=dtype)
    d = [torch.from_numpy(x.copy()).cuda() for x in m.arrays()]
    ref = [x.astype(np.float64) for x in m.arrays()]
    sg.pobtaf(*d, precision=precision)
    oracle.pobtaf(*ref)
    for x, y in zip(d, ref):
        assert np.linalg.norm(x.cpu().numpy() - y) <= tol * max(np.linalg.norm(y), 1e-300)
