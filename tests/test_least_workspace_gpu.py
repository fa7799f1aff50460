"""Sweeps in the least workspace: what a caller has sized without the slice buffers
of the native form, and a device whose memory does not hold them."""

import ctypes

import numpy as np
import pytest
import torch

import oracle
import serinv_gb300 as sg
from serinv_gb300 import _lib, algs
from serinv_gb300.algs import _bta_struct
from serinv_gb300.synthetic import generate

from _golden import rel_err

pytestmark = pytest.mark.gpu

# real blocks from 224 on, complex ones from 112 on (their embedding's), have slice buffers
SIZES = [(3, 224, 8, np.float64), (3, 112, 4, np.complex128), (33, 192, 0, np.float64), (3, 64, 8, np.float64)]


def _least(desc, op, ring=-1):
    n = ctypes.c_size_t(0)
    assert _lib.load().sgb_least_workspace_size(ctypes.byref(desc), op, 0, ring, ctypes.byref(n)) == 0
    return n.value


def _close(got, ref):
    for g, r in zip(got, ref):
        assert rel_err(g.cpu().numpy() if isinstance(g, torch.Tensor) else g, r) <= 1e-12


@pytest.mark.parametrize("n,b,a,dt", SIZES)
def test_c_calls(n, b, a, dt):
    lib = _lib.load()
    m = generate(n, b, a, 1, seed=91, dtype=dt)
    d = [torch.from_numpy(x).cuda() for x in m.arrays()]
    ref = [x.copy() for x in m.arrays()]
    s = torch.cuda.current_stream().cuda_stream
    desc = _bta_struct(*d)
    for op, call, orc in ((1, "pobtaf", oracle.pobtaf), (2, "pobtasi", oracle.pobtasi)):
        full = ctypes.c_size_t(0)
        assert getattr(lib, f"sgb_{call}_workspace_size")(ctypes.byref(desc), 0, ctypes.byref(full)) == 0
        least = _least(desc, op)
        rows = 2 * b if dt == np.complex128 else b
        sliced = rows >= 224 or (op == 2 and n >= 32 and rows >= 192)
        assert least < full.value if sliced else least == full.value
        ws = torch.empty(least, dtype=torch.uint8, device="cuda")
        args = [ctypes.byref(desc), 1, 0, ws.data_ptr()]
        tail = [None, s] if op == 1 else [s]
        assert getattr(lib, f"sgb_{call}")(*args, least - 1, *tail) == _lib.SGB_ERR_WORKSPACE
        assert getattr(lib, f"sgb_{call}")(*args, least, *tail) == 0
        orc(*ref)
        _close(d, ref)


def test_permuted_form():
    """The middle-partition factorization has no slices of its own to size for."""
    lib = _lib.load()
    m = generate(4, 224, 8, 1, seed=93)
    d = [torch.from_numpy(x).cuda() for x in m.arrays()]
    buf = torch.zeros((4, 224, 224), dtype=torch.float64, device="cuda")
    ref, rbuf = [x.copy() for x in m.arrays()], np.zeros((4, 224, 224))
    oracle.pobtaf_permuted(*ref, rbuf)
    desc = _bta_struct(*d)
    least = _least(desc, 1)
    ws = torch.empty(least, dtype=torch.uint8, device="cuda")
    assert lib.sgb_pobtaf_permuted(ctypes.byref(desc), buf.data_ptr(), 0, ws.data_ptr(), least, None,
                                   torch.cuda.current_stream().cuda_stream) == 0
    _close(d, ref)
    _close([buf[1:]], [rbuf[1:]])


@pytest.mark.parametrize("form", ["device", "pinned", "streamed"])
def test_python_calls_without_room_for_the_slices(form, monkeypatch):
    m = generate(4, 224, 8, 1, seed=95)
    ref = [x.copy() for x in m.arrays()]
    oracle.pobtaf(*ref)
    real, sizes = algs._workspace, []

    def short(nbytes, device):
        sizes.append(nbytes)
        if len(sizes) % 2 == 1:
            raise torch.OutOfMemoryError("no room")
        return real(nbytes, device)

    monkeypatch.setattr(algs, "_workspace", short)
    t = [torch.from_numpy(x) for x in m.copy().arrays()]
    t = [x.cuda() for x in t] if form == "device" else [x.pin_memory() for x in t] if form == "pinned" else t
    kw = {"device_streaming": True} if form == "streamed" else {}
    sg.pobtaf(*t, **kw)
    _close(t, ref)
    sg.pobtasi(*t, **kw)
    oracle.pobtasi(*ref)
    _close(t, ref)
    assert len(sizes) == 4 and sizes[1] < sizes[0] and sizes[3] < sizes[2]


def test_no_smaller_form_is_still_out_of_memory(monkeypatch):
    m = generate(3, 64, 8, 1, seed=97)
    d = [torch.from_numpy(x).cuda() for x in m.arrays()]

    def none(nbytes, device):
        raise torch.OutOfMemoryError("no room")

    monkeypatch.setattr(algs, "_workspace", none)
    with pytest.raises(torch.OutOfMemoryError):
        sg.pobtaf(*d)
