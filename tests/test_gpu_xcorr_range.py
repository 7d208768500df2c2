"""gxc_xcorr in FP32 up to the end of its range: sums between half of the largest float and the largest float are finite, on
every route to the split X-stage."""
import ctypes as C

import numpy as np
import pytest

import gcorr_gb300 as G
from gcorr_gb300 import _lib as L

pytestmark = pytest.mark.gpu


# read in place; through the re-laid copy (odd fftwidth)
@pytest.mark.parametrize("fftwidth", [16, 17])
@pytest.mark.parametrize("nant", [3, 12])
def test_sums_near_the_largest_float(nant, fftwidth):
    import torch
    nchan, nfft = 16, 12
    ants = torch.full((2 * nant, nfft, fftwidth), 2.0 ** 62, dtype=torch.complex64, device="cuda")
    ants[1] *= -1.0
    nbl = nant * (nant + 1) // 2
    out = torch.zeros((nbl, 4, nchan), dtype=torch.complex64, device="cuda")
    st = G.lib().gxc_xcorr(C.c_void_p(ants.data_ptr()), nant, nfft, nchan, fftwidth, L.GXC_PRECISION_FP32,
                           L.GXC_XENGINE_TENSOR, 1, C.c_void_p(out.data_ptr()),
                           C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == L.GXC_OK, L.status_name(st)
    # the sums are 12 x 2^124, three quarters of 2^128; a mean of 12 equal powers of two is exact
    sign = np.ones(2 * nant)
    sign[1] = -1.0
    pairs = [(i, j) for i in range(nant) for j in range(i + 1, nant)] + [(i, i) for i in range(nant)]
    exp = np.array([[sign[2 * i + p] * sign[2 * j + q] for p in range(2) for q in range(2)] for i, j in pairs]) * 2.0 ** 124
    got = out.cpu().numpy()
    assert np.array_equal(got, np.broadcast_to(exp[..., None], got.shape).astype(np.complex64))
