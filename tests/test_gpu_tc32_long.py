"""The FP32-accurate F-stage with its first step on tensor cores at 16384 and 32768 points (csrc/fstage_tc32.cu), against the
FP64 oracle: the FFT count where it takes over from the register FFT and one less, two FFT blocks, flagged windows, a
rotator slope that changes at every FFT, both rotators, odd sample offsets."""
import numpy as np
import pytest

from gcorr_gb300 import FxKernel, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-5   # the FP32 tolerance of the parity tests


def _nfft(nant):
    """The smallest FFT count (and block) for which the kernel is chosen: one window per SM."""
    import torch
    return -(-torch.cuda.get_device_properties(0).multi_processor_count // nant)


def _check(w, d, mask=None, validity=None, rotator="exact", **kw):
    fx = FxKernel(w.nant, w.nchan, w.nfft, w.nbit, w.lo_hz, w.bw_hz, w.is_complex, precision="fp32", rotator=rotator, **kw)
    fx.setInputData([x.cuda() for x in d["inputs"]])
    fx.setDelays(d["poly"], d["fso"])
    if validity is not None:
        fx.setFrameValidity(validity, w.fft_len)
    fx.process()
    vis, counts = fx.visibilities(), fx.baseline_counts()
    fx.close()
    rot = O.ROT_EXACT if rotator == "exact" else O.ROT_FXKERNEL
    ref, rc = O.exact_process(O.config_from_workload(w, rot, True), [x.cpu().numpy() for x in d["inputs"]], d["poly"],
                              d["fso"], mask=mask)
    assert np.array_equal(counts, rc)
    assert O.rel_rms_per_product(vis, ref).max() < TOL


@pytest.mark.parametrize("nchan", [8192, 16384])
@pytest.mark.parametrize("nant,extra,blocks", [(8, 0, 1), (8, -1, 1), (6, 1, 1), (9, 5, 2)])
def test_edges_vs_fp64(nchan, nant, extra, blocks):
    full = _nfft(nant)
    w = synth.Workload(nant=nant, nchan=nchan, nfft=full + extra, bw_hz=64e6, seed=nchan + nant, offset_us=40.0)
    _check(w, synth.random_bytes(w), fft_block=full if blocks == 2 else 0)


@pytest.mark.parametrize("nchan,rotator", [(8192, "exact"), (16384, "exact"), (16384, "fxkernel")])
def test_changing_slope(nchan, rotator):
    w = synth.Workload(nant=6, nchan=nchan, nfft=_nfft(6) + 3, bw_hz=128e6, seed=nchan, offset_us=1.0)
    d = synth.random_bytes(w)
    tf = w.fft_time
    d["poly"][:, 0] = np.array([2e-3, -1e-3, 3e-3, 1e-4, -2e-4, 5e-4]) * tf * tf
    d["poly"][:, 1] = np.array([-5e-4, 2e-4, 1e-4, 3e-4, -1e-4, 0.0]) * tf
    _check(w, d, rotator=rotator)


@pytest.mark.parametrize("nchan", [8192, 16384])
def test_flagged_windows(nchan):
    import torch
    w = synth.Workload(nant=6, nchan=nchan, nfft=_nfft(6), bw_hz=64e6, seed=5, offset_us=0.0)
    d = synth.random_bytes(w)
    d["poly"][:] = 0.0
    flag = [0, 1, 7, 20, w.nfft - 1]
    v = torch.ones(w.nfft + 1, dtype=torch.uint8, device="cuda")
    v[flag] = 0
    mask = np.ones((6, w.nfft), np.uint8)
    mask[0, flag] = mask[3, flag] = 0
    _check(w, d, mask=mask, validity=[v, None, None, v, None, None])
