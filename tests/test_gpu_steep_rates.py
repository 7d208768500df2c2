"""FP32 spectra of short scans (the register FFTs) at delay rates of 1e-4 and more, whose fringe turns thousands of times per
window, against the FP64 oracle: within the FP32 tolerance as at any other rate."""
import numpy as np
import pytest

from gcorr_gb300 import FxKernel, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-5   # the FP32 tolerance of the parity tests


@pytest.mark.parametrize("nchan,cplx,rotator", [(1024, False, "exact"), (4096, False, "exact"), (4096, False, "fxkernel"),
                                                (8192, False, "exact"), (16384, False, "exact"), (16384, False, "fxkernel"),
                                                (8192, True, "exact"), (16384, True, "exact")])
def test_steep_rates_vs_fp64(nchan, cplx, rotator):
    w = synth.Workload(nant=6, nchan=nchan, nfft=12, nbit=8 if cplx else 2, is_complex=cplx, bw_hz=128e6, seed=nchan,
                       offset_us=1.0)
    d = synth.random_bytes(w)
    tf = w.fft_time
    d["poly"][:, 0] = np.array([2e-3, -1e-3, 3e-3, 1e-4, -2e-4, 5e-4]) * tf * tf
    d["poly"][:, 1] = np.array([-5e-4, 2e-4, 1e-4, 3e-4, -1e-4, 0.0]) * tf
    rot = O.ROT_EXACT if rotator == "exact" else O.ROT_FXKERNEL
    ref, rc = O.exact_process(O.config_from_workload(w, rot, True), [x.numpy() for x in d["inputs"]], d["poly"], d["fso"])
    fx = FxKernel(w.nant, w.nchan, w.nfft, w.nbit, w.lo_hz, w.bw_hz, w.is_complex, precision="fp32", rotator=rotator)
    fx.setInputData([x.numpy() for x in d["inputs"]])
    fx.setDelays(d["poly"], d["fso"])
    fx.process()
    vis, counts = fx.visibilities(), fx.baseline_counts()
    fx.close()
    assert np.array_equal(counts, rc)
    assert O.rel_rms_per_product(vis, ref).max() < TOL
