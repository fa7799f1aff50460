"""Native FP64 sweeps on the exact slice products: around the block sizes where
they begin, at ragged tiles and at the longest contraction they take, and for
matrices whose rows and columns differ by many orders of magnitude."""

import numpy as np
import pytest
import torch

import oracle
import serinv_gb300 as sg
from serinv_gb300.synthetic import generate

pytestmark = pytest.mark.gpu

# 176: where the forms change over; 576: the longest contraction
SHAPES = [(5, 175, 8), (5, 176, 8), (4, 190, 0), (3, 223, 5), (3, 224, 0), (3, 240, 33), (4, 257, 64), (2, 300, 1), (3, 544, 32), (2, 576, 0), (2, 577, 3),
          (1, 320, 40)]


def rel(x, ref):
    n = np.linalg.norm(ref)
    return float(np.linalg.norm(x - ref) / n) if n else float(np.linalg.norm(x))


def both(m):
    d = [torch.from_numpy(x.copy()).cuda() for x in m]
    sg.pobtaf(*d)
    L = [x.cpu().numpy() for x in d]
    sg.pobtasi(*d)
    return L, [x.cpu().numpy() for x in d]


@pytest.mark.parametrize("n,b,a", SHAPES)
def test_against_the_oracle(n, b, a):
    m = generate(n, b, a, 1, seed=b + a)
    L, X = both(m.arrays())
    ref = [x.copy() for x in m.arrays()]
    oracle.pobtaf(*ref)
    assert max(rel(x, y) for x, y in zip(L, ref)) < 1e-12
    oracle.pobtasi(*ref)
    assert max(rel(x, y) for x, y in zip(X, ref)) < 1e-12


@pytest.mark.parametrize("n,b,a", [(3, 256, 20), (2, 512, 64)])
def test_scaled_rows_and_columns(n, b, a):
    """A = S A0 S with S over twelve orders of magnitude: the scaled-back factor
    and inverse keep the accuracy they have without S."""
    m = generate(n, b, a, 1, seed=3)
    ref = [x.copy() for x in m.arrays()]
    oracle.pobtaf(*ref)
    Lref = [x.copy() for x in ref]
    oracle.pobtasi(*ref)
    rng = np.random.default_rng(1)
    s, t = 2.0 ** rng.integers(-20, 21, (n, b)), 2.0 ** rng.integers(-20, 21, a)  # powers of two: nothing is rounded
    D, Lo, Ar, T = m.arrays()
    A = [D * s[:, :, None] * s[:, None, :], Lo * s[1:, :, None] * s[:-1, None, :], Ar * t[None, :, None] * s[:, None, :],
         T * t[:, None] * t[None, :]]
    L, X = both([np.ascontiguousarray(x) for x in A])
    L = [L[0] / s[:, :, None], L[1] / s[1:, :, None], L[2] / t[None, :, None], L[3] / t[:, None]]
    X = [X[0] * s[:, :, None] * s[:, None, :], X[1] * s[1:, :, None] * s[:-1, None, :],
         X[2] * t[None, :, None] * s[:, None, :], X[3] * t[:, None] * t[None, :]]
    assert max(rel(x, y) for x, y in zip(L, Lref)) < 1e-12
    assert max(rel(x, y) for x, y in zip(X, ref)) < 1e-12


def test_nan_reaches_the_pivots():
    m = generate(3, 256, 8, 1, seed=2)
    m.Lo[0][5, 7] = np.nan
    d = [torch.from_numpy(x).cuda() for x in m.arrays()]
    with pytest.raises(np.linalg.LinAlgError):
        sg.pobtaf(*d)
