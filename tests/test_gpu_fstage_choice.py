"""Which F-stage kernel a handle runs, as gxc_fft_engine and gxc_fstage_kernel tell it: the register FFT where CUDA_CORE is
asked for, and both sides of each line between the kernels that AUTO draws."""
import numpy as np
import pytest

from gcorr_gb300 import FxKernel, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _kernel(nant, nchan, nfft, precision="fp32", cplx=False, **kw):
    fx = FxKernel(nant, nchan, nfft, 8 if cplx else 2, 8.4e9, 64e6, cplx, precision=precision, **kw)
    got = fx.fft_engine_used, fx.fstage_kernel
    fx.close()
    return got


def _groups(nchan):
    """Windows of a work unit of the mixed kernel, and the FFTs of one antenna with which it starts to be chosen: three units
    of 16384 samples per SM, from 16384 points on one window per SM."""
    import torch
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    nw = max(1, 4096 // nchan)
    return nw, nw * nsm * (3 if nchan < 8192 else 1)


@pytest.mark.parametrize("nchan,register", [(1024, "fstage_kernel"), (2048, "fstage_kernel"), (4096, "fstage_pair_kernel"),
                                            (8192, "fstage_kernel"), (16384, "fstage_cluster_kernel")])
def test_fp32_lines(nchan, register):
    nw, full = _groups(nchan)
    assert _kernel(1, nchan, full) == ("mixed", "fstage_tc32_kernel")
    assert _kernel(1, nchan, full - nw) == ("cuda_core", register)
    assert _kernel(2, nchan, full, fft_block=full // 2) == ("mixed", "fstage_tc32_kernel")
    assert _kernel(2, nchan, full, fft_block=full // 2 - nw) == ("cuda_core", register)
    assert _kernel(1, nchan, full, fft_engine="cuda_core") == ("cuda_core", register)
    if nchan in (1024, 4096, 16384):  # the fxkernel rotator: where its table split falls on a row of the first step
        mixed = nchan != 1024
        assert _kernel(1, nchan, full, rotator="fxkernel")[0] == ("mixed" if mixed else "cuda_core")
    assert _kernel(1, nchan, full, cplx=True)[0] == "cuda_core"


@pytest.mark.parametrize("precision", ["fp16", "fp8"])
def test_fp16_and_fp8_engines(precision):
    assert _kernel(4, 4096, 3000, precision) == ("tensor", "fstage_tc_kernel")
    assert _kernel(4, 4096, 3000, precision, fft_engine="cuda_core") == ("cuda_core", "fstage_pair_kernel")
    assert _kernel(4, 4096, 3000, precision, autos=False) == ("tensor", "fstage_tc_cross_kernel")
    assert _kernel(4, 1024, 10000, precision) == ("mixed", "fstage_tc32_kernel")
    assert _kernel(4, 1024, 10000, precision, fft_engine="cuda_core") == ("cuda_core", "fstage_kernel")
    assert _kernel(4, 8192, 3000, precision) == ("cuda_core", "fstage_h_kernel")


def test_block_beyond_32_bit_channel_steps():
    """Spectra of 2^38 bytes: four channel tiles of a block are 2^32 bytes, more than fstage_tc_kernel steps over.  The handle
    is only made here; it takes the kernel that addresses it."""
    import torch
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 2 ** 38 + (3 << 30):
        pytest.skip("needs 278 GB of free device memory")
    assert _kernel(64, 4096, 131072, "fp16", fft_block=131071)[1] == "fstage_tc_kernel"
    assert _kernel(64, 4096, 131072, "fp16", fft_block=131072)[1] == "fstage_tc_cross_kernel"


@pytest.mark.parametrize("precision", ["fp16", "fp8"])
@pytest.mark.parametrize("nchan", [1024, 4096])
def test_choice_does_not_hang_on_the_antenna_count(nchan, precision):
    """Whatever the number of antennas: the same kernel for handles with autocorrelations, and one without."""
    for autos, kernels in ((True, {"fstage_tc_kernel" if nchan == 4096 else "fstage_tc32_kernel"}),
                           (False, {"fstage_tc_cross_kernel" if nchan == 4096 else
                                    "fstage_tc32_kernel" if precision == "fp16" else "fstage_kernel"})):
        assert {_kernel(n, nchan, 2000, precision, autos=autos)[1] for n in (2, 16, 17, 20, 64)} == kernels


@pytest.mark.parametrize("nchan", [1024, 4096, 16384])
def test_cuda_core_runs_the_register_fft(nchan):
    """A block that AUTO gives to the mixed kernel, with CUDA_CORE: the bits that a block too short for the mixed kernel
    gives.  All FFTs but one are flagged, so that no sum depends on the blocks."""
    import torch
    nw, full = _groups(nchan)
    w = synth.Workload(nant=2, nchan=nchan, nfft=full, bw_hz=64e6, seed=nchan, offset_us=0.0)
    d = synth.random_bytes(w, device="cuda")
    poly = np.zeros((2, 3))
    poly[1, 1] = 1e-13  # 0.00084 turns of 8.4 GHz per FFT, no whole sample
    v = torch.zeros(w.nfft + 1, dtype=torch.uint8, device="cuda")
    v[full - 3] = 1
    vis = {}
    for name, kw in (("auto", {}), ("asked", {"fft_engine": "cuda_core"}), ("short", {"fft_block": full // 2 - nw})):
        fx = FxKernel(w.nant, w.nchan, w.nfft, w.nbit, w.lo_hz, w.bw_hz, precision="fp32", x_engine="cuda_core", **kw)
        assert (fx.fft_engine_used == "mixed") == (name == "auto")
        fx.setInputData(d["inputs"])
        fx.setDelays(poly, np.zeros(2))
        fx.setFrameValidity([v, v], w.fft_len)
        fx.process()
        assert (fx.baseline_counts() == 1).all()
        vis[name] = fx.visibilities()
        fx.close()
    assert np.array_equal(vis["asked"].view(np.uint32), vis["short"].view(np.uint32))
    assert not np.array_equal(vis["auto"].view(np.uint32), vis["short"].view(np.uint32))
    assert O.rel_rms(vis["auto"], vis["short"]) < 1e-5


def test_autotune_tries_the_mixed_kernel(tmp_path):
    from gcorr_gb300.autotune import tune
    nw, full = _groups(2048)
    w = synth.Workload(nant=2, nchan=2048, nfft=full, bw_hz=64e6, seed=1)
    d = synth.random_bytes(w, device="cuda")
    job = dict(nant=2, nchan=2048, nfft=full, nbit=2, lo=w.lo_hz, bw=w.bw_hz, is_complex=False, inputs=d["inputs"],
               poly=d["poly"], fso=d["fso"], precision="fp32")
    t = tune(job, blocks=(full,), path=str(tmp_path / "tune.json"))
    assert {p["fft_engine"] for p in t["tried"]} == {"cuda_core", "auto"}
