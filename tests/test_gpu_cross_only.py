"""FP16 and FP8 handles without autocorrelations, and FP8 ones of more than 16 antennas, whose 8192-point windows take
their own F-stage (fstage_tc_cross.cu): products against the FP64 oracle, from one FFT to several per SM."""
import numpy as np
import pytest

from gcorr_gb300 import FxKernel, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = {"fp16": 1e-3, "fp8": 0.12}   # the parity tests' tolerances


@pytest.mark.parametrize("nchan", [1024, 4096])
@pytest.mark.parametrize("precision", ["fp16", "fp8"])
@pytest.mark.parametrize("nant,autos,nfft", [(4, False, 1), (4, False, 37), (4, False, 160), (17, True, 25)])
def test_products_vs_fp64(nchan, precision, nant, autos, nfft):
    w = synth.Workload(nant=nant, nchan=nchan, nfft=nfft, bw_hz=64e6, seed=nchan + nfft, offset_us=1.0, rho=0.5)
    d = synth.generate(w)
    fx = FxKernel(w.nant, w.nchan, w.nfft, w.nbit, w.lo_hz, w.bw_hz, precision=precision, autos=autos)
    fx.setInputData([x.cuda() for x in d["inputs"]])
    fx.setDelays(d["poly"], d["fso"])
    fx.process()
    vis, counts = fx.visibilities(), fx.baseline_counts()
    fx.close()
    ref, rc = O.exact_process(O.config_from_workload(w, O.ROT_EXACT, autos), [x.numpy() for x in d["inputs"]], d["poly"],
                              d["fso"])
    assert np.array_equal(counts, rc)
    assert O.rel_rms_per_product(vis, ref).max() < TOL[precision]
