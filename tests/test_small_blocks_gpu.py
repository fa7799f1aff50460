"""Blocks small enough for the one-launch kernels, around the sizes where they
and the two-tile column blocks begin and end, against the oracle."""

import numpy as np
import pytest
import torch

import oracle
import serinv_gb300 as sg
from serinv_gb300.synthetic import generate

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 0), (3, 1, 1), (2, 7, 31), (5, 8, 8), (12, 8, 32), (4, 9, 33), (9, 15, 2), (17, 16, 0), (3, 16, 32),
          (5, 17, 5), (9, 31, 1), (3, 32, 32), (4, 33, 3), (3, 64, 20), (1, 16, 4), (20, 12, 3)]


def rel(x, ref):
    n = np.linalg.norm(ref)
    return float(np.linalg.norm(x - ref) / n) if n else float(np.linalg.norm(x))


@pytest.mark.parametrize("dtype,tol", [(np.float64, 1e-12), (np.float32, 1e-5)])
@pytest.mark.parametrize("n,b,a", SHAPES)
def test_small(n, b, a, dtype, tol):
    m = generate(n, b, a, 5, seed=n + 7 * b + a, dtype=dtype)
    for last in (True, False):
        d = [torch.from_numpy(x.copy()).cuda() for x in m.arrays()]
        ref = [x.astype(np.float64) for x in m.arrays()]
        sg.pobtaf(*d, factorize_last_block=last)
        oracle.pobtaf(*ref, factorize_last_block=last)
        got = [x.cpu().numpy() for x in d]
        if not last:  # of what is left unfactored the lower triangles are defined
            got[0][-1], ref[0][-1] = np.tril(got[0][-1]), np.tril(ref[0][-1])
            got[3], ref[3] = np.tril(got[3]), np.tril(ref[3])
        assert max(rel(x, y) for x, y in zip(got, ref)) < tol
    d = [torch.from_numpy(x.copy()).cuda() for x in m.arrays()]
    sg.pobtaf(*d)
    L = [x.cpu().numpy().astype(np.float64) for x in d]
    for nrhs in (1, 5):
        for trans in ("N", "C"):
            x = torch.from_numpy(np.ascontiguousarray(m.B[:, :nrhs])).cuda()
            sg.pobtas(*d, x, trans=trans)
            y = m.B[:, :nrhs].astype(np.float64)
            oracle.pobtas(*L, y, trans=trans)
            assert rel(x.cpu().numpy(), y) < tol
    sg.pobtasi(*d)
    ref = [x.copy() for x in L]
    oracle.pobtasi(*ref)
    assert max(rel(x.cpu().numpy(), y) for x, y in zip(d, ref)) < tol


@pytest.mark.parametrize("n,b,a", [(4, 5, 3), (12, 16, 32), (6, 9, 0)])
def test_selected_inverse_from_a_given_last_block(n, b, a):
    m = generate(n, b, a, 1, seed=11)
    L = [x.copy() for x in m.arrays()]
    oracle.pobtaf(*L)
    full = [x.copy() for x in L]
    oracle.pobtasi(*full)
    given = [x.copy() for x in L]
    given[0][-1], given[3][:] = full[0][-1], full[3]
    if a:
        given[2][-1] = full[2][-1]
    d = [torch.from_numpy(x).cuda() for x in given]
    sg.pobtasi(*d, invert_last_block=False)
    assert max(rel(x.cpu().numpy(), y) for x, y in zip(d, full)) < 1e-12


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n,b,a,row", [(3, 6, 2, 8), (2, 16, 4, 33), (4, 3, 0, 12)])
def test_bad_pivot_row(n, b, a, row, dtype):
    """The 1-based row of the first bad pivot, in a block and in the tip."""
    m = generate(n, b, a, 1, seed=1, dtype=dtype)
    if row <= n * b:
        m.D[(row - 1) // b][(row - 1) % b, (row - 1) % b] = -1e6
    else:
        m.T[row - n * b - 1, row - n * b - 1] = -1e6
    d = [torch.from_numpy(x).cuda() for x in m.arrays()]
    with pytest.raises(np.linalg.LinAlgError, match=f"{row}-th"):
        sg.pobtaf(*d)
