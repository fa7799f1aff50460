"""GPU: bounded waits of pobtas and pobtasi that give up (poll limit 0, no real
hang) are reported, and what runs after them is right.

pobtas in one cluster launch: every CTA takes in what its peers sent before any
of them leaves, so a sweep changes nothing that runs after it; when the waits
give up the whole right-hand side is NaN.
"""

import ctypes

import numpy as np
import pytest
import torch

import oracle
import serinv_gb300 as sg
from serinv_gb300 import _lib
from serinv_gb300.algs import _bta_struct
from serinv_gb300.refine import pobtas_refine
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


def test_a_solve_that_gave_up_is_reported():
    """The status word in the workspace's first bytes; raised where the call synchronises."""
    m = _factor(4, 64, 8, 2, np.float64, seed=67)
    d = [torch.from_numpy(x).cuda() for x in m.arrays()]
    with _SpinLimit(0):
        with pytest.raises(_lib.SgbError, match="timed out"):
            sg.pobtas(*d, torch.from_numpy(m.B).cuda(), check_spd=True)
        with pytest.raises(_lib.SgbError, match="timed out"):
            sg.pobtas(*m.arrays(), m.B.copy())  # host arrays
        with pytest.raises(_lib.SgbError, match="timed out"):
            pobtas_refine(*m.copy().arrays(), *m.arrays(), m.B.copy(), iters=1)
    ref = m.B.copy()
    oracle.pobtas(*m.arrays(), ref)
    B = torch.from_numpy(m.B).cuda()
    sg.pobtas(*d, B, check_spd=True)
    assert rel_err(B.cpu().numpy(), ref) <= 1e-12


@pytest.mark.parametrize("case", [(4, 3, 2, 2, False), (3, 40, 5, 700, False), (4, 64, 8, 3, True), (3, 20, 4, 0, False)])
def test_status_word_is_set_on_every_route(case):
    """One launch, products of very many columns, partial solves, no columns."""
    n, b, a, nrhs, partial = case
    m = _factor(n, b, a, max(nrhs, 1), np.float64, seed=71)
    lib = _lib.load()
    d = [torch.from_numpy(x).cuda() for x in m.arrays()]
    B = torch.from_numpy(np.ascontiguousarray(m.B[:, :nrhs])).cuda()
    desc = _bta_struct(*d)
    need = ctypes.c_size_t(0)
    assert lib.sgb_pobtas_workspace_size(ctypes.byref(desc), nrhs, 0, ctypes.byref(need)) == 0
    for trans in (b"N", b"T"):
        ws = torch.full((need.value,), 0x5a, dtype=torch.uint8, device="cuda")
        assert lib.sgb_pobtas(ctypes.byref(desc), B.data_ptr() or None, nrhs, max(nrhs, 1), trans, int(partial), 0,
                              ws.data_ptr(), need.value, torch.cuda.current_stream().cuda_stream) == 0
        assert int(ws[:4].view(torch.int32).item()) == 0


@pytest.mark.parametrize("shape,dt", [((3, 224, 16), np.float64), ((33, 192, 0), np.float64)])
def test_a_selected_inverse_that_gave_up_is_reported(shape, dt):
    """The native FP64 form on tensor-core products: on device arrays, on host
    arrays, and not at all where the caller asks for no check."""
    n, b, a = shape
    m = _factor(n, b, a, 1, dt, seed=73)
    d = [torch.from_numpy(x).cuda() for x in m.arrays()]
    assert _lib.load().sgb_pobtasi_has_waits(ctypes.byref(_bta_struct(*d)), 0) == 1
    with _SpinLimit(0):
        with pytest.raises(_lib.SgbError, match="timed out"):
            sg.pobtasi(*[x.clone() for x in d])
        with pytest.raises(_lib.SgbError, match="timed out"):
            sg.pobtasi(*[x.pin_memory() for x in (y.cpu() for y in d)])
        with pytest.raises(_lib.SgbError, match="timed out"):
            sg.pobtasi(*[y.cpu() for y in d], device_streaming=True)
        sg.pobtasi(*[x.clone() for x in d], check_spd=False)
    ref = [x.copy() for x in m.arrays()]
    oracle.pobtasi(*ref)
    sg.pobtasi(*d)
    for g, r in zip(d, ref):
        assert rel_err(g.cpu().numpy(), r) <= 1e-12


def test_selected_inverse_can_be_captured():
    """The status is not read while the stream is captured."""
    m = _factor(3, 224, 0, 1, np.float64, seed=79)
    d = [torch.from_numpy(x).cuda() for x in m.arrays()]
    X = [x.clone() for x in d]
    sg.pobtasi(*[x.clone() for x in d])
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        sg.pobtasi(*X)
    for x, y in zip(X, d):
        x.copy_(y)
    g.replay()
    ref = [x.copy() for x in m.arrays()]
    oracle.pobtasi(*ref)
    for x, r in zip(X, ref):
        assert rel_err(x.cpu().numpy(), r) <= 1e-12
