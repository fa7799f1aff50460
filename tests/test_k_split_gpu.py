"""GPU: K-split tensor-core products over tiles with rows and columns past the
edge and zero rows: their partial sums are read from the cluster's CTAs and then
dropped, and no CTA leaves before such a read is done.
"""

import ctypes

import pytest
import torch

from serinv_gb300 import _lib

pytestmark = pytest.mark.gpu


def _product(M, N, K, prec, A, B, ws, need):
    C = torch.full((M, N), 3.0, dtype=torch.float64, device="cuda")
    rc = _lib.load().sgb_dgemm(prec, b"N", b"N", M, N, K, -1.0, A.data_ptr(), K, B.data_ptr(), N, 1.0, C.data_ptr(), N,
                               ws.data_ptr(), need, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    return C


@pytest.mark.parametrize("shape", [(1, 1, 512), (130, 70, 512), (257, 33, 576), (60, 200, 300)])
@pytest.mark.parametrize("prec", ["mixed", "mixed:3"])
def test_ragged_k_split_products(shape, prec):
    M, N, K = shape
    lib, code = _lib.load(), _lib.precision_code(prec)
    need = ctypes.c_size_t(0)
    assert lib.sgb_dgemm_workspace_size(code, M, N, K, ctypes.byref(need)) == 0
    ws = torch.zeros(need.value, dtype=torch.uint8, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(7)
    A = torch.rand((M, K), generator=g, device="cuda", dtype=torch.float64) - 0.5
    B = torch.rand((K, N), generator=g, device="cuda", dtype=torch.float64) - 0.5
    A[M // 2] = 0.0
    ref = 3.0 - A @ B
    first = _product(M, N, K, code, A, B, ws, need.value)
    # S slices keep 7 S bits below the row maxima (0.5 each here), K products of that error
    bound = K * 0.25 * 2.0 ** (-7 * (6 if prec == "mixed" else 3) + 1)
    assert float((first - ref).abs().max()) <= bound
    assert torch.equal(first[M // 2], torch.full((N,), 3.0, dtype=torch.float64, device="cuda"))
    for _ in range(30):
        assert torch.equal(_product(M, N, K, code, A, B, ws, need.value), first)
