"""Products whose output is one of their operands.  Rows of A against a whole B of
up to 32 columns may be written over A whatever their number (each row of the
output takes its own row of A only); an output of up to 32 x 32 may be any operand
(one tile reads all of it before it writes)."""

import pytest
import torch

from serinv_gb300 import dgemm

pytestmark = pytest.mark.gpu


def _pair(M, N, K, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.rand((M, K), generator=g, device="cuda", dtype=torch.float64) - 0.5,
            torch.rand((K, N), generator=g, device="cuda", dtype=torch.float64) - 0.5)


def _bound(A, B):  # K products and sums on either side
    return 2 * (A.shape[1] + 2) * 2.0 ** -53 * (A.abs() @ B.abs())


@pytest.mark.parametrize("M", [1, 7, 8, 9, 31, 32, 33, 100, 700, 6000])
@pytest.mark.parametrize("N", [3, 8, 16, 31, 32])
def test_rows_of_a(M, N):
    A, B = _pair(M, N, N, M + N)
    ref, bound = A @ B, _bound(A, B)
    assert bool(((dgemm(A, B, A) - ref).abs() <= bound).all())


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 24, 31, 32])
@pytest.mark.parametrize("N", [9, 16, 31, 32])
def test_b(M, N):
    A, B = _pair(M, N, M, 3 * M + N)
    ref, bound = A @ B, _bound(A, B)
    for _ in range(20):
        C = B.clone()
        assert bool(((dgemm(A, C, C) - ref).abs() <= bound).all())


@pytest.mark.parametrize("N", [9, 17, 25, 32])
def test_transposed_a_and_b(N):
    A, B = _pair(N, N, N, N)
    for ta, tb in ((True, False), (False, True), (True, True)):
        a, b = (A.T if ta else A), (B.T if tb else B)
        ref, bound = a @ b, _bound(a, b)
        for _ in range(20):
            X, Y = A.clone(), B.clone()
            assert bool(((dgemm(X, B, X, transA=ta, transB=tb) - ref).abs() <= bound).all())
            assert bool(((dgemm(A, Y, Y, transA=ta, transB=tb) - ref).abs() <= bound).all())
