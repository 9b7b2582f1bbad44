"""Caller-owned amplitudes of any element alignment (rq_expectation_batch_noalloc).

A complex-f32 array is aligned to 8 bytes, so a view that starts at an odd element is not aligned to
the 16 bytes of the vector loads.  Reference: the same sums in numpy (FP64); both sides add 2^n products
whose total is at most 1, in different orders: 1e-13 absolute.
"""
import ctypes as C

import numpy as np
import pytest

from ruqu_b200 import _capi
from ruqu_b200.state import pauli_array
from test_gpu_pauli_batch import _reference, _strings


def _call(ptr, n, prec, strings):
    arr, off = pauli_array(strings)
    out = np.full(len(strings), np.nan)
    rc = _capi.lib.rq_expectation_batch_noalloc(
        C.c_void_p(ptr), n, prec, arr, off.ctypes.data_as(C.POINTER(C.c_uint32)), len(strings),
        out.ctypes.data_as(C.POINTER(C.c_double)), None)
    return rc, out


@pytest.mark.gpu
@pytest.mark.parametrize("n", [13, 14, 16])
@pytest.mark.parametrize("offset", [0, 1, 3])
def test_f32_views_at_any_element(n, offset):
    import torch
    g = torch.Generator().manual_seed(n + offset)
    a = torch.view_as_complex(torch.randn(1 << n, 2, generator=g, dtype=torch.float64))
    a = (a / a.abs().square().sum().sqrt()).to(torch.complex64)
    buf = torch.zeros((1 << n) + 4, dtype=torch.complex64, device="cuda")
    view = buf[offset:offset + (1 << n)]
    view.copy_(a)
    torch.cuda.synchronize()
    assert view.data_ptr() % 16 == 8 * (offset & 1)
    strings = _strings(n, False)
    for part in (strings[:128], strings[128:], [s for s in strings if all(o == 3 for _, o in s)][:9]):
        if not part:
            continue
        rc, got = _call(view.data_ptr(), n, _capi.RQ_F32, part)
        assert rc == 0, _capi.last_error()
        assert np.max(np.abs(got - _reference(a.numpy().astype(np.complex128), part))) < 1e-13
    assert torch.equal(view.cpu(), a)


@pytest.mark.parametrize("prec,address", [(_capi.RQ_F32, 0x10004), (_capi.RQ_F64, 0x10008)])
def test_addresses_that_hold_no_whole_amplitude_are_rejected(prec, address):
    """Refused on the host, before anything reads the address."""
    rc, out = _call(address, 14, prec, [[(0, 3)]])
    assert rc == _capi.RQ_ERR_INVALID_ARGUMENT
    assert np.isnan(out).all()
