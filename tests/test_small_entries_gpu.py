"""GPU: every entry of the native FP64 factor and selected inverse, not only the
large ones.

The matrices are M-matrices (no positive entry off the diagonal): then no
difference in the factorization, the inversion or the back-sweep cancels, and
FP64 sums give every entry to a few roundings of its own size, however small it
is beside the largest of its row.  Couplings decay from entry to entry, so the
entries of one row span 60 orders of magnitude and more.

Bound: an entry is a chain over n blocks of sums of up to 3 b + a products of
such entries, each term with its own roundings: n (3 b + a) 2^-53 times a small
factor on each side (computed against FP64 as well); 8 is used.
"""

import numpy as np
import pytest
import torch

import oracle
import serinv_gb300 as sg

pytestmark = pytest.mark.gpu

# n, b, a, every how many blocks a dense one (whose products need no small entries)
CASES = [(3, 192, 16, 0), (4, 224, 0, 0), (33, 192, 8, 0), (3, 250, 33, 0), (6, 240, 8, 2), (9, 256, 0, 3), (3, 448, 8, 0),
         (2, 512, 0, 0), (3, 512, 64, 0)]


def _m_matrix(n, b, a, dense=0):
    D = np.zeros((n, b, b))
    i = np.arange(b)
    diag, off = (1.5, 0.3) if b < 300 else (2.4, 0.8)  # no entry below 1e-290
    D[:, i, i] = diag + 0.1 * np.cos(i)
    D[:, i[1:], i[:-1]] = -off - 0.05 * np.sin(i[1:])
    D[:, i[:-1], i[1:]] = D[:, i[1:], i[:-1]]
    if dense:
        D[dense - 1::dense] -= 0.2 / b
    Lo = np.zeros((n - 1, b, b))
    Lo[:, i, i] = -0.2
    Lo[:, i[1:], i[:-1]] = -0.01
    Ar = np.zeros((n, a, b))
    for r in range(a):
        Ar[:, r] = -0.02 * 0.4 ** np.abs(i - (r * b) // max(a, 1))
    T = np.eye(a) * (2.0 + n) - 0.01
    return D, Lo, Ar, T


def _entry_err(got, ref):
    got, ref = got.cpu().numpy(), np.asarray(ref)
    zero = ref == 0
    assert np.all(got[zero] == 0)
    return float(np.max(np.abs(got[~zero] - ref[~zero]) / np.abs(ref[~zero]), initial=0.0))


@pytest.mark.parametrize("case", CASES)
def test_entries_of_factor_and_inverse(case):
    n, b, a, dense = case
    m = _m_matrix(n, b, a, dense)
    bound = 2 * 8 * n * (3 * b + a) * 2.0 ** -53
    d = [torch.from_numpy(x).cuda() for x in m]
    ref = [x.copy() for x in m]
    oracle.pobtaf(*ref)
    small = min(float(np.abs(x[x != 0]).min()) for x in ref if x.size)
    assert 1e-290 < small < (1e-30 if not dense else 1e-4)  # decaying, and no entry near the subnormal range
    sg.pobtaf(*d)
    for g, r in zip(d, ref):
        assert _entry_err(g, r) <= bound
    # the inverse from the oracle's factor, so that its errors are its own
    d = [torch.from_numpy(x).cuda() for x in ref]
    oracle.pobtasi(*ref)
    sg.pobtasi(*d)
    for g, r in zip(d, ref):
        assert _entry_err(g, r) <= bound
