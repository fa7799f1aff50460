"""GPU: pobtas in one cluster launch, after waits that gave up (poll limit 0, no
real hang) and launch after launch.  Every CTA takes in what its peers sent
before any of them leaves, so a sweep changes nothing that runs after it; when
the waits give up the whole right-hand side is NaN.
"""

import numpy as np
import pytest
import torch

import oracle
import serinv_gb300 as sg
from serinv_gb300.synthetic import generate

from _golden import rel_err
from test_failure_gpu import _SpinLimit

pytestmark = pytest.mark.gpu


def _factor(n, b, a, nrhs, dt, seed):
    m = generate(n, b, a, nrhs, seed=seed, dtype=dt)
    oracle.pobtaf(*m.arrays())
    return m


@pytest.mark.parametrize("case", [(5, 24, 3, 1, np.float64), (4, 64, 8, 2, np.float64), (3, 150, 40, 5, np.float64),
                                  (2, 300, 0, 1, np.float64), (4, 70, 5, 3, np.float32), (1, 40, 9, 4, np.float64)])
@pytest.mark.parametrize("trans", ["N", "T"])
def test_solve_that_gives_up_and_solves_after_it(case, trans):
    n, b, a, nrhs, dt = case
    m = _factor(n, b, a, nrhs, dt, seed=61)
    d = [torch.from_numpy(x).cuda() for x in m.arrays()]
    ref = m.B.copy()
    oracle.pobtas(*m.arrays(), ref, trans=trans)
    tol = 1e-12 if dt == np.float64 else 1e-4
    with _SpinLimit(0):
        B = torch.from_numpy(m.B).cuda()
        sg.pobtas(*d, B, trans=trans)
        torch.cuda.synchronize()
        assert bool(torch.isnan(B).all())
    first = None
    for _ in range(20):  # back to back: each launch's CTAs follow on the last one's SMs
        B = torch.from_numpy(m.B).cuda()
        sg.pobtas(*d, B, trans=trans)
        if first is None:
            first = B
            assert rel_err(B.cpu().numpy(), ref) <= tol
        assert torch.equal(B, first)
