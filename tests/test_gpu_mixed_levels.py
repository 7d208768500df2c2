"""The FP32-accurate F-stage with its first step on tensor cores: the decoded operand bit for bit, as the FP32 levels that it
stands for, and no bias of the power spectra against FP64 at any of its lengths; the decode of the FP16 and FP8 kernel for
handles without autocorrelations."""
import ctypes as C

import numpy as np
import pytest

from gcorr_gb300 import FxKernel, synth
from gcorr_gb300 import _lib as L
from oracle import oracle as O

pytestmark = pytest.mark.gpu

BW = 64e6


def _full(nchan, nant):
    """FFTs with which the kernel is chosen: three units of 16384 samples per SM, from 16384 points on one window per SM."""
    import torch
    nw, per = max(1, 4096 // nchan), 3 if nchan < 8192 else 1
    return nw * -(-per * torch.cuda.get_device_properties(0).multi_processor_count // nant)


@pytest.mark.parametrize("nchan,precision,autos,kernel", [
    (1024, "fp32", True, "fstage_tc32_kernel"), (2048, "fp32", True, "fstage_tc32_kernel"),
    (4096, "fp32", True, "fstage_tc32_kernel"), (8192, "fp32", True, "fstage_tc32_kernel"),
    (16384, "fp32", True, "fstage_tc32_kernel"), (1024, "fp16", True, "fstage_tc32_kernel"),
    (2048, "fp8", True, "fstage_tc32_kernel"), (4096, "fp16", False, "fstage_tc_cross_kernel"),
    (4096, "fp8", False, "fstage_tc_cross_kernel")])
def test_unpack_bit_exact(nchan, precision, autos, kernel):
    """gxc_probe_unpack writes the operands of the first step, scaled as the kernel scales them: every bit is the
    reference's level (fxkernel/src/fxkernel.cpp:15-28, :443-476), at odd and even offsets, over all byte values."""
    import torch
    nant, F = 16, 2 * nchan
    nfft = _full(nchan, nant)
    fx = FxKernel(nant, nchan, nfft, 2, 8.4e9, BW, False, precision=precision, autos=autos)
    assert fx.fstage_kernel == kernel
    rng = np.random.default_rng(nchan)
    n = fx.bytes_per_antenna
    inputs = [np.concatenate([rng.permutation(256) for _ in range(-(-n // 256))]).astype(np.uint8)[:n] for _ in range(nant)]
    ts = 1.0 / (2.0 * BW)
    poly = np.array([[1e-3 * ts, (a - 7.3) * 0.6 * ts, -(a + 1.0) * ts] for a in range(nant)])
    fx.setInputData([torch.from_numpy(x).cuda() for x in inputs])
    fx.setDelays(poly, np.zeros(nant))
    got = np.zeros((nant, 2, nfft, F), dtype=np.complex64)
    L.check(L.lib().gxc_probe_unpack(fx._h, C.c_void_p(got.ctypes.data)), fx._h, "gxc_probe_unpack")
    flags = fx.valid_flags()
    fx.close()
    cfg = O.make_config(nant, nchan, nfft, 2, False, 8.4e9, BW)
    parities, seen = set(), 0
    for a in range(nant):
        for t in range(nfft):
            g = O.geometry(cfg, poly[a], 0.0, t)
            assert int(flags[a, t]) == int(g.valid)
            if not g.valid:
                assert np.isnan(got[a, :, t].view(np.float32)).all(), "flagged window was written"
                continue
            parities.add(g.offset & 1)
            seen += 1
            for pol, ref in enumerate(O.unpack(cfg, inputs[a], g.offset, F)):
                assert np.array_equal(got[a, pol, t].view(np.uint32), ref.view(np.uint32)), (a, t, pol)
    assert parities == {0, 1} and seen > nant * nfft // 2


@pytest.mark.parametrize("nchan,nant,rotator,mhz", [
    (1024, 57, "exact", 64.), (2048, 57, "exact", 128.), (4096, 57, "exact", 32.), (4096, 57, "fxkernel", 128.),
    (8192, 38, "exact", 64.), (16384, 38, "exact", 128.), (16384, 38, "fxkernel", 64.)])
def test_power_spectra_have_no_bias(nchan, nant, rotator, mhz):
    """Mean signed error of the power of noise: below 3e-8 (a quarter of FP32's last bit, 2^-23), which is the stated 2e-8 and
    the spread between delay models.  The sum is over more than 100,000 independent errors of 1.6e-7."""
    import torch
    w = synth.Workload(nant=nant, nchan=nchan, nfft=_full(nchan, nant), bw_hz=mhz * 1e6, seed=nchan + nant, offset_us=1.0,
                       rho=0.05)
    d = synth.generate(w)
    fx = FxKernel(nant, nchan, w.nfft, 2, w.lo_hz, w.bw_hz, precision="fp32", rotator=rotator, x_engine="cuda_core")
    assert fx.fstage_kernel == "fstage_tc32_kernel"
    fx.setInputData([x.cuda() for x in d["inputs"]])
    fx.setDelays(d["poly"], d["fso"])
    fx.process()
    vis, counts = fx.visibilities(), fx.baseline_counts()
    fx.close()
    nx = nant * (nant - 1) // 2
    cfg = O.config_from_workload(w, O.ROT_EXACT if rotator == "exact" else O.ROT_FXKERNEL, True)
    err = ref = 0.0
    for a in range(nant):
        x = d["inputs"][a].numpy()
        p = np.zeros((2, nchan))
        for t in range(w.nfft):
            if O.geometry(cfg, d["poly"][a], d["fso"][a], t).valid:
                p += np.abs(np.asarray(O.exact_channelise(cfg, x, d["poly"][a], d["fso"][a], t))) ** 2
        p /= counts[nx + a]
        err += (vis[nx + a, [0, 3]].real.astype(np.float64) - p).sum()
        ref += p.sum()
    assert abs(err / ref) < 3e-8, err / ref
