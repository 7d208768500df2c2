"""Baseline counts and flags from the validity bits: FFT counts around a word (32 FFTs) and around the size up to which
finalisation counts the FFTs itself (8192), one and several antennas, with and without autos."""
import numpy as np
import pytest

from gcorr_gb300 import FxKernel, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nfft", [1, 31, 32, 33, 8192, 8193, 8225])
@pytest.mark.parametrize("nant,autos", [(1, True), (3, True), (2, False)])
def test_counts_and_flags(nfft, nant, autos):
    w = synth.Workload(nant=nant, nchan=128, nfft=nfft, bw_hz=64e6, seed=nfft, offset_us=12.0)
    d = synth.random_bytes(w)
    ref, rc = O.exact_process(O.config_from_workload(w, O.ROT_EXACT, autos), [x.numpy() for x in d["inputs"]], d["poly"], d["fso"])
    fx = FxKernel(w.nant, w.nchan, w.nfft, w.nbit, w.lo_hz, w.bw_hz, precision="fp32", autos=autos)
    fx.setInputData([x.numpy() for x in d["inputs"]])
    fx.setDelays(d["poly"], d["fso"])
    for _ in range(2):  # the second run overwrites the first one's accumulators
        fx.process()
    vis, counts, flags = fx.visibilities(), fx.baseline_counts(), fx.valid_flags()
    fx.close()
    assert np.array_equal(counts, rc)
    pairs = [(j, k) for j in range(nant) for k in range(j + 1, nant)] + ([(j, j) for j in range(nant)] if autos else [])
    assert np.array_equal(counts, [int((flags[j] & flags[k]).sum()) for j, k in pairs])
    ok = rc > 0
    if ok.any():
        assert O.rel_rms_per_product(vis[ok], ref[ok]).max() < 1e-5
    assert not vis[~ok].any()
