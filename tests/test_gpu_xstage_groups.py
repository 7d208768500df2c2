"""The tensor-core X-stage with fewer MMA groups per CTA (few channel groups, each CTA taking half or a quarter of its
usual channels): FP16, FP8 and FP32 process() against the FP64 oracle, over channel counts that leave one, two and four
groups, with and without the split of the FFTs."""
import numpy as np
import pytest

from gcorr_gb300 import FxKernel, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = {"fp32": 1e-5, "fp16": 1e-3, "fp8": 0.12}   # the parity tests' tolerances


@pytest.mark.parametrize("nant", [2, 5, 7, 11, 20, 32])
@pytest.mark.parametrize("nchan", [128, 512, 2048])
@pytest.mark.parametrize("precision,nfft", [("fp32", 70), ("fp16", 70), ("fp16", 600), ("fp8", 600)])
def test_few_groups_vs_fp64(nant, nchan, precision, nfft):
    if nant * nchan * nfft > 2e7:
        nfft = 70
    w = synth.Workload(nant=nant, nchan=nchan, nfft=nfft, bw_hz=32e6, seed=nant + nchan, offset_us=1.0)
    d = synth.random_bytes(w)
    fx = FxKernel(w.nant, w.nchan, w.nfft, w.nbit, w.lo_hz, w.bw_hz, precision=precision, x_engine="tensor")
    fx.setInputData([x.cuda() for x in d["inputs"]])
    fx.setDelays(d["poly"], d["fso"])
    fx.process()
    vis, counts = fx.visibilities(), fx.baseline_counts()
    fx.close()
    ref, rc = O.exact_process(O.config_from_workload(w, O.ROT_EXACT, True), [x.numpy() for x in d["inputs"]], d["poly"],
                              d["fso"])
    assert np.array_equal(counts, rc)
    assert O.rel_rms_per_product(vis, ref).max() < TOL[precision]
