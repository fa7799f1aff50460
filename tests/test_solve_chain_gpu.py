"""The one-launch solve at the edges of its sub-blocks, clusters and column groups,
against the oracle's sweeps."""

import numpy as np
import pytest
import torch

import oracle
import serinv_gb300 as sg
from serinv_gb300.synthetic import generate

pytestmark = pytest.mark.gpu

# b around the sub-block length (128) and the cluster sizes (1, 2, 4, 8, 16 CTAs of eight rows), tips around the same
# edges, columns around the groups of 1, 2 and 4 per cluster
SHAPES = [(1, 1, 0, 1), (3, 8, 1, 1), (4, 9, 8, 2), (3, 17, 9, 3), (5, 33, 32, 5), (3, 64, 65, 17), (4, 65, 3, 33),
          (3, 127, 127, 1), (2, 128, 128, 9), (3, 129, 130, 2), (3, 200, 33, 3), (2, 257, 300, 4), (3, 384, 0, 8),
          (1, 130, 5, 6), (2, 40, 4, 70)]


@pytest.mark.parametrize("dtype,tol", [(np.float64, 1e-12), (np.float32, 1e-5)])
@pytest.mark.parametrize("n,b,a,nrhs", SHAPES)
def test_solve_edges(n, b, a, nrhs, dtype, tol):
    m = generate(n, b, a, nrhs, seed=n * b + a, dtype=dtype)
    L = [x.astype(np.float64) for x in m.arrays()]
    oracle.pobtaf(*L)
    L = [x.astype(dtype) for x in L]
    d = [torch.from_numpy(x).cuda() for x in L]
    for trans in ("N", "C"):
        x = torch.from_numpy(m.B).cuda()
        sg.pobtas(*d, x, trans=trans)
        ref = m.B.astype(np.float64)
        oracle.pobtas(*[y.astype(np.float64) for y in L], ref, trans=trans)
        assert np.linalg.norm(x.cpu().numpy() - ref) <= tol * np.linalg.norm(ref)


def test_solve_keeps_a_bad_row_to_what_depends_on_it():
    """An Inf in the right-hand side reaches the rows below it, not those above."""
    n, b, a = 3, 150, 4
    m = generate(n, b, a, 2, seed=5)
    L = list(m.arrays())
    oracle.pobtaf(*L)
    d = [torch.from_numpy(x).cuda() for x in L]
    bad = b + 70
    B = m.B.copy()
    B[bad, 0] = np.inf
    x = torch.from_numpy(B).cuda()
    sg.pobtas(*d, x, trans="N")
    x = x.cpu().numpy()
    ref = m.B.copy()
    oracle.pobtas(*L, ref, trans="N")
    assert np.allclose(x[:bad, 0], ref[:bad, 0], rtol=1e-10) and not np.isfinite(x[bad, 0])
    assert np.allclose(x[:, 1], ref[:, 1], rtol=1e-10)
