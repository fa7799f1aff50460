"""GPU: solves with many right-hand sides.  Small blocks take a CTA for every four
columns, others a cluster for every one to four columns, and products beyond what
a few rounds of clusters cover."""

import numpy as np
import pytest
import torch

import oracle
import serinv_gb300 as sg
from serinv_gb300.synthetic import generate

from _golden import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [4, 5, 33, 257, 1030, 4099])
@pytest.mark.parametrize("case", [(6, 5, 2, np.float64), (5, 16, 4, np.float64), (4, 32, 3, np.float32), (5, 24, 0, np.float64),
                                  (3, 70, 9, np.float64), (3, 64, 5, np.float32)])
def test_columns(case, nrhs):
    n, b, a, dt = case
    m = generate(n, b, a, nrhs, seed=nrhs + b, dtype=dt)
    oracle.pobtaf(*m.arrays())
    d = [torch.from_numpy(x).cuda() for x in m.arrays()]
    # well-conditioned factors: some hundred roundings of the type along a column
    tol = 1e-12 if dt == np.float64 else 1e-4
    for trans in ("N", "T"):
        ref = m.B.copy()
        oracle.pobtas(*m.arrays(), ref, trans=trans)
        wide = torch.full((m.B.shape[0], nrhs + 3), 7.0, dtype=d[0].dtype, device="cuda")
        B = torch.from_numpy(m.B).cuda()
        sg.pobtas(*d, B, trans=trans)
        assert rel_err(B.cpu().numpy(), ref) <= tol
        wide[:, :nrhs] = torch.from_numpy(m.B).cuda()
        view = wide[:, :nrhs]  # rows apart: columns past the right-hand sides stay
        sg.pobtas(*d, view, trans=trans)
        assert rel_err(view.cpu().numpy(), ref) <= tol
        assert bool((wide[:, nrhs:] == 7.0).all())
