"""The FP32-accurate F-stage whose first step runs on tensor cores (csrc/fstage_tc32.cu; 2048 to 8192 points, 2-bit
real) at its edges, against the FP64 oracle: FFT counts that do not fill a group of windows, FFT blocks that end inside
one, flagged windows inside groups, a rotator slope that changes from FFT to FFT, one antenna, every output
type, and the size where the kernel takes over from the register FFT."""
import numpy as np
import pytest

from gcorr_gb300 import FxKernel, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FP32_TOL = 1e-5   # the FP32 tolerance of the parity tests
FP16_TOL = 1e-3   # one FP16 rounding per value, 2.0e-4 rms: 2.9e-4 per product
FP8_TOL = 0.12


def _run(w, d, **kw):
    fx = FxKernel(w.nant, w.nchan, w.nfft, w.nbit, w.lo_hz, w.bw_hz, w.is_complex, **kw)
    fx.setInputData([x.numpy() for x in d["inputs"]])
    fx.setDelays(d["poly"], d["fso"])
    fx.process()
    v, c = fx.visibilities(), fx.baseline_counts()
    fx.close()
    return v, c


def _full(nchan, nant):
    """The smallest FFT count (and block) for which the kernel is chosen: three groups of 16384 samples per SM."""
    import torch
    nw = 64 // (nchan // 64)
    return nw * -(-3 * torch.cuda.get_device_properties(0).multi_processor_count // nant)


@pytest.mark.parametrize("nchan", [1024, 2048, 4096])
@pytest.mark.parametrize("nant,extra,blocks", [(1, 0, 1), (3, 1, 1), (4, 3, 2), (2, -1, 1)])
def test_group_edges_vs_fp64(nchan, nant, extra, blocks):
    """extra FFTs past a whole number of groups; with two blocks the second one holds only `extra` FFTs; one FFT less
    than the kernel takes runs the register FFT."""
    full = _full(nchan, nant)
    w = synth.Workload(nant=nant, nchan=nchan, nfft=full + extra, bw_hz=64e6, seed=nchan + extra, offset_us=40.0)
    d = synth.random_bytes(w)
    ref, rc = O.exact_process(O.config_from_workload(w, O.ROT_EXACT, True), [x.numpy() for x in d["inputs"]], d["poly"], d["fso"])
    vis, counts = _run(w, d, precision="fp32", fft_block=full if blocks == 2 else 0)
    assert np.array_equal(counts, rc)
    assert O.rel_rms_per_product(vis, ref).max() < FP32_TOL


@pytest.mark.parametrize("nchan,rotator", [(1024, "exact"), (4096, "exact"), (4096, "fxkernel")])
@pytest.mark.parametrize("precision", ["fp32", "fp16", "fp8"])
def test_changing_slope_and_output_types(nchan, rotator, precision):
    """Slopes of many turns per window that change by more than their last bit at every FFT, and delays that drift by
    samples."""
    w = synth.Workload(nant=6, nchan=nchan, nfft=_full(nchan, 6) + 5, bw_hz=128e6, seed=nchan, offset_us=1.0)
    d = synth.random_bytes(w)
    tf = w.fft_time
    d["poly"][:, 0] = np.array([2e-3, -1e-3, 3e-3, 1e-4, -2e-4, 5e-4]) * tf * tf
    d["poly"][:, 1] = np.array([-5e-4, 2e-4, 1e-4, 3e-4, -1e-4, 0.0]) * tf
    rot = O.ROT_EXACT if rotator == "exact" else O.ROT_FXKERNEL
    ref, rc = O.exact_process(O.config_from_workload(w, rot, True), [x.numpy() for x in d["inputs"]], d["poly"], d["fso"])
    vis, counts = _run(w, d, precision=precision, rotator=rotator, fft_engine="cuda_core")
    assert np.array_equal(counts, rc)
    tol = {"fp32": FP32_TOL, "fp16": FP16_TOL, "fp8": FP8_TOL}[precision]
    assert O.rel_rms_per_product(vis, ref).max() < tol


@pytest.mark.parametrize("nchan,flag", [(1024, [0, 9, 17, 40]), (2048, [3, 4, 5, 6, 7, 8]), (4096, [0, 1, 2, 30])])
def test_flagged_windows_inside_groups(nchan, flag):
    import torch
    w = synth.Workload(nant=2, nchan=nchan, nfft=_full(nchan, 2), bw_hz=64e6, seed=5, offset_us=0.0)
    d = synth.random_bytes(w, device="cuda")
    d["poly"][:] = 0.0
    v = torch.ones(w.nfft + 1, dtype=torch.uint8, device="cuda")
    v[flag] = 0
    fx = FxKernel(w.nant, w.nchan, w.nfft, w.nbit, w.lo_hz, w.bw_hz, precision="fp32")
    fx.setInputData(d["inputs"])
    fx.setDelays(d["poly"], d["fso"])
    fx.setFrameValidity([v, None], w.fft_len)
    fx.process()
    vis, counts = fx.visibilities(), fx.baseline_counts()
    fx.close()
    mask = np.ones((2, w.nfft), np.uint8)
    mask[0, flag] = 0
    ref, rc = O.exact_process(O.config_from_workload(w, O.ROT_EXACT, True), [x.cpu().numpy() for x in d["inputs"]],
                              d["poly"], d["fso"], mask=mask)
    assert np.array_equal(counts, rc)
    assert O.rel_rms_per_product(vis, ref).max() < FP32_TOL
