"""gxc_xcorr on device data read where it is (launch_xstage_direct) and on what still goes through the re-laid copy (an odd
fftwidth, a base that is not 16-byte aligned, more FFTs than a cluster takes): integer data, whose sums are exact, so
every route must give the same bits; and scaled noise against FP64."""
import ctypes as C

import numpy as np
import pytest

import gcorr_gb300 as G
from gcorr_gb300 import _lib as L
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _xcorr(ants, nant, nfft, nchan, fftwidth, precision, autos):
    import torch
    nbl = nant * (nant - 1) // 2 + (nant if autos else 0)
    out = torch.full((nbl, 4, nchan), float("nan"), dtype=torch.complex64, device="cuda")
    st = G.lib().gxc_xcorr(C.c_void_p(ants.data_ptr()), nant, nfft, nchan, fftwidth, precision, L.GXC_XENGINE_AUTO,
                           int(autos), C.c_void_p(out.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == L.GXC_OK, L.status_name(st)
    return out.cpu().numpy()


def _sums(d, nant, nfft, nchan, fftwidth, autos):
    """FP64 sums over the FFTs on the GPU, [nbl][4][nchan]."""
    import torch
    d = d.reshape(nant, 2, nfft, fftwidth)[..., :nchan].to(torch.complex128)
    pairs = [(i, j) for i in range(nant - 1) for j in range(i + 1, nant)] + ([(i, i) for i in range(nant)] if autos else [])
    v = torch.stack([(d[i, p] * d[j, q].conj()).sum(0) for i, j in pairs for p in range(2) for q in range(2)])
    return v.reshape(len(pairs), 4, nchan).cpu().numpy()


# nant, nchan, nfft, fftwidth, elements before the data: parts of one drain period, ragged and empty last parts, the
# most FFTs of a cluster and one more; each row count of the kernel; the routes through the copy
@pytest.mark.parametrize("nant,nchan,nfft,fftwidth,lead", [
    (2, 16, 1, 16, 0), (4, 128, 63, 256, 0), (5, 128, 129, 128, 2), (16, 64, 513, 64, 0), (32, 128, 1025, 130, 0),
    (3, 384, 2049, 384, 0), (16, 1024, 300, 1024, 0), (7, 128, 8192, 128, 0), (6, 16, 8193, 16, 0), (4, 128, 200, 129, 0),
    (4, 128, 200, 256, 1), (1, 128, 100, 128, 0)])
@pytest.mark.parametrize("precision", [L.GXC_PRECISION_FP32, L.GXC_PRECISION_FP16])
@pytest.mark.parametrize("autos", [True, False])
def test_routes(nant, nchan, nfft, fftwidth, lead, precision, autos):
    import torch
    if nant == 1 and not autos:
        pytest.skip("no baseline")
    gen = torch.Generator(device="cuda").manual_seed(nant + nfft)
    n = 2 * nant * nfft * fftwidth
    buf = torch.full((lead + n,), float("nan"), dtype=torch.complex64, device="cuda")
    ants = buf[lead:]
    ants.copy_(torch.complex(*(torch.randint(-5, 6, (n,), generator=gen, device="cuda").float() for _ in range(2))))
    s = _sums(ants, nant, nfft, nchan, fftwidth, autos)  # |sum| <= 50 * 8193 < 2^24
    exp = np.empty(s.shape, np.complex64)
    exp.real = s.real.astype(np.float32) / np.float32(nfft)
    exp.imag = s.imag.astype(np.float32) / np.float32(nfft)
    assert np.array_equal(_xcorr(ants, nant, nfft, nchan, fftwidth, precision, autos), exp)
    ants.copy_(torch.randn(n, generator=gen, device="cuda", dtype=torch.complex64) * 37.0)
    x = torch.view_as_real(ants)
    rounded = torch.view_as_complex(x.half().float()) if precision == L.GXC_PRECISION_FP16 else ants
    ref = _sums(rounded, nant, nfft, nchan, fftwidth, autos) / nfft
    assert O.rel_rms_per_product(_xcorr(ants, nant, nfft, nchan, fftwidth, precision, autos), ref).max() < 1e-5
