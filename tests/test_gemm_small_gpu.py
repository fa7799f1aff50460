"""Products of few tiles (8 x 8, 16 x 16 and 8 x 32 kernels) at the edges of
their tiles and of the 64-wide staging of k."""

import itertools

import pytest
import torch

from serinv_gb300 import dgemm

pytestmark = pytest.mark.gpu

SIZES = [(1, 9, 1), (7, 10, 63), (8, 16, 64), (9, 33, 65), (64, 64, 64), (80, 64, 130), (129, 130, 147), (256, 200, 31),
         (257, 260, 257)]


@pytest.mark.parametrize("M,N,K", SIZES)
@pytest.mark.parametrize("ta,tb", list(itertools.product([False, True], repeat=2)))
def test_small_products(M, N, K, ta, tb):
    g = torch.Generator(device="cuda").manual_seed(M * N + K)
    A = torch.rand((K, M) if ta else (M, K), generator=g, device="cuda", dtype=torch.float64) - 0.5
    B = torch.rand((N, K) if tb else (K, N), generator=g, device="cuda", dtype=torch.float64) - 0.5
    C = torch.rand((M, N), generator=g, device="cuda", dtype=torch.float64)
    a, b = (A.T if ta else A), (B.T if tb else B)
    ref = -1.5 * (a @ b) + 0.5 * C
    out = dgemm(A, B, C.clone(), alpha=-1.5, beta=0.5, transA=ta, transB=tb)
    # each side rounds K products and sums (unit roundoff 2^-53) plus the scaling and the addition of C
    bound = 2 * (K + 3) * 2.0 ** -53 * (1.5 * (a.abs() @ b.abs()) + 0.5 * C)
    assert bool(((out - ref).abs() <= bound).all())
