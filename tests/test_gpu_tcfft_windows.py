"""The tensor-core F-stage's window pipeline at its edges: fewer windows than CTAs, one window, window counts that
do not divide by the CTAs or slots, and runs of flagged windows longer than its table ring, against the CUDA-core
FFT on the same input."""
import numpy as np
import pytest

from gcorr_gb300 import FxKernel, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# both paths round the output to FP16 (2.0e-4 rms relative); the tensor-core FFT adds three roundings of that size:
# per product sqrt(2 * (4 + 1)) * 2.0e-4 = 6.3e-4
TOL = 1e-3


@pytest.mark.parametrize("nant,nfft,flag", [(1, 1, None), (2, 3, None), (3, 50, None), (3, 51, (7, 40)), (5, 123, (0, 60)),
                                            (16, 40, (11, 12)), (7, 131, (40, 131))])
def test_window_pipeline_edges(nant, nfft, flag):
    import torch
    w = synth.Workload(nant=nant, nchan=4096, nfft=nfft, bw_hz=256e6, seed=700 + nfft, offset_us=0.0005)
    d = synth.random_bytes(w, device="cuda")
    res = []
    for engine in ("tensor", "cuda_core"):
        fx = FxKernel(w.nant, w.nchan, w.nfft, w.nbit, w.lo_hz, w.bw_hz, precision="fp16", fft_engine=engine)
        fx.setInputData(d["inputs"])
        fx.setDelays(d["poly"], d["fso"])
        if flag:  # one frame per FFT window; antenna 0 loses a stretch of them
            v = torch.ones(nfft + 1, dtype=torch.uint8, device="cuda")
            v[flag[0]:flag[1]] = 0
            fx.setFrameValidity([v] + [None] * (nant - 1), 8192)
        fx.process()
        assert fx.fft_engine_used == engine
        res.append((fx.visibilities(), fx.baseline_counts(), fx.valid_flags()))
        fx.close()
    assert np.array_equal(res[0][1], res[1][1]) and np.array_equal(res[0][2], res[1][2])
    if flag:
        assert (res[0][2][0] == 0).sum() >= flag[1] - flag[0]
    ok = res[0][1] > 0
    assert O.rel_rms_per_product(res[0][0][ok], res[1][0][ok]).max() < TOL
    assert not res[0][0][~ok].any()
