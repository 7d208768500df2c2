"""The register FFT with both polarisations of a window in one CTA (256 to 4096 points; at 256 points two windows per
CTA) at its edges, against the FP64 oracle: odd FFT counts and blocks that leave half of the last CTA without a window,
and flagged windows that share a CTA with valid ones."""
import numpy as np
import pytest

from gcorr_gb300 import FxKernel, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = {"fp32": 1e-5, "fp16": 1e-3, "fp8": 0.12}   # the parity tests' tolerances


@pytest.mark.parametrize("cplx,points", [(False, 256), (True, 256), (True, 512), (False, 1024), (True, 4096)])
@pytest.mark.parametrize("precision", ["fp32", "fp16", "fp8"])
@pytest.mark.parametrize("nfft,block,flag", [(1, 0, []), (33, 0, [0, 3, 4, 5]), (33, 7, [6, 7, 13, 32])])
def test_pairs_of_windows_vs_fp64(cplx, points, precision, nfft, block, flag):
    import torch
    w = synth.Workload(nant=3, nchan=points if cplx else points // 2, nfft=nfft, nbit=8 if cplx else 2, is_complex=cplx,
                       bw_hz=32e6, seed=points + nfft, offset_us=0.0)
    d = synth.random_bytes(w, device="cuda")
    d["poly"][:] = 0.0
    v = torch.ones(w.nfft + 1, dtype=torch.uint8, device="cuda")
    v[flag] = 0
    fx = FxKernel(w.nant, w.nchan, w.nfft, w.nbit, w.lo_hz, w.bw_hz, w.is_complex, precision=precision, fft_block=block)
    fx.setInputData(d["inputs"])
    fx.setDelays(d["poly"], d["fso"])
    fx.setFrameValidity([v, None, v], w.fft_len)
    fx.process()
    vis, counts = fx.visibilities(), fx.baseline_counts()
    fx.close()
    mask = np.ones((3, w.nfft), np.uint8)
    mask[0, flag] = mask[2, flag] = 0
    ref, rc = O.exact_process(O.config_from_workload(w, O.ROT_EXACT, True), [x.cpu().numpy() for x in d["inputs"]],
                              d["poly"], d["fso"], mask=mask)
    assert np.array_equal(counts, rc)
    assert O.rel_rms_per_product(vis, ref).max() < TOL[precision]
