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


# FP32 diagonal tiles: eight columns a warp, the last tile of every width
@pytest.mark.parametrize("b", [65, 71, 72, 73, 95, 98, 127])
def test_fp32_tile_widths(b):
    m = generate(3, b, 9, 1, seed=b, dtype=np.float32)
    d = [torch.from_numpy(x.copy()).cuda() for x in m.arrays()]
    ref = [x.astype(np.float64) for x in m.arrays()]
    sg.pobtaf(*d)
    oracle.pobtaf(*ref)
    for x, y in zip(d, ref):
        assert np.linalg.norm(x.cpu().numpy() - y) <= 1e-5 * max(np.linalg.norm(y), 1e-300)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("bad", [(0,), (7,), (8, 9), (31,), (32, 70), (47, 33), (70,)])
def test_first_bad_pivot(bad, dtype):
    b = 71
    D = np.repeat(4 * np.eye(b, dtype=dtype)[None], 3, 0)
    D[:, 1:, :-1] += np.eye(b - 1, dtype=dtype)
    for k in bad:
        D[1, k, k] = -1 if k != 33 else np.nan
    d = [torch.from_numpy(x).cuda() for x in (D, np.zeros((2, b, b), dtype))]
    with pytest.raises(np.linalg.LinAlgError, match=f"^{b + min(bad) + 1}-th"):
        sg.pobtf(*d)


# FP64 column blocks in two halves (from b = 416 on; 576: the longest product of the exact form)
@pytest.mark.parametrize("b,a", [(415, 3), (416, 0), (417, 64), (449, 33), (500, 1), (576, 130)])
@pytest.mark.parametrize("last", [True, False])
def test_halves(b, a, last):
    m = generate(2, b, a, 1, seed=b)
    d = [torch.from_numpy(x.copy()).cuda() for x in m.arrays()]
    ref = [x.copy() for x in m.arrays()]
    sg.pobtaf(*d, factorize_last_block=last)
    oracle.pobtaf(*ref, factorize_last_block=last)
    got = [x.cpu().numpy() for x in d]
    if not last:  # of what is left unfactored the lower triangles are defined
        got[0][-1], ref[0][-1] = np.tril(got[0][-1]), np.tril(ref[0][-1])
        got[3], ref[3] = np.tril(got[3]), np.tril(ref[3])
    for x, y in zip(got, ref):
        assert np.linalg.norm(x - y) <= 1e-12 * max(np.linalg.norm(y), 1e-300)


@pytest.mark.parametrize("bad", [100, 223, 224, 300, 430])
def test_halves_first_bad_pivot(bad):
    D = np.repeat(4 * np.eye(431)[None], 2, 0)
    D[:, 1:, :-1] += np.eye(430)
    D[0, bad, bad] = -1
    d = [torch.from_numpy(x).cuda() for x in (D, np.zeros((1, 431, 431)))]
    with pytest.raises(np.linalg.LinAlgError, match=f"^{bad + 1}-th"):
        sg.pobtf(*d)
