"""The work that a user of this correlator has it do, as measurable cases.

One pass of a case is one sub-integration (or one batch, one stretch of a stream, one X-stage call) through
the public entry points: ``FxKernel``, ``Batch``, ``Pipeline`` and the C ABI's ``gxc_xcorr``.  ``listed()``
holds the cases, ``draw()`` more of the same ranges, ``prepare()`` makes the voltages, delay models and handles,
``run()`` makes one pass, ``work()`` states what a pass cannot do without, and ``exact()`` gives its result in
64 bits from the definition (unpack, fringe rotation, DFT, fractional-delay phase, conjugate products, mean over
the valid FFTs), with none of this package's code.
"""
import ctypes
import math

import numpy as np
import torch

import gcorr_gb300 as G
from gcorr_gb300 import synth
from gcorr_gb300.batch import Batch
from gcorr_gb300.pipeline import Pipeline

PRECISIONS = {"fp32": 0, "fp16": 1, "fp8": 2}


def _fx(name, nant, nchan, nfft, cplx, mhz, precision, rotator="exact", autos=True):
    return {"name": name, "kind": "process", "nant": nant, "nchan": nchan, "nfft": nfft, "complex": cplx, "mhz": float(mhz),
            "precision": precision, "rotator": rotator, "autos": autos}


def listed():
    return [
        # the smallest call: a short scan of a few antennas, as in fringe checks and unit runs; launches and latency
        _fx("quick_4ant_fp32", 4, 1024, 16, False, 64, "fp32"),
        # six VLBI stations, 64 MHz, a quarter of a second: the reference driver's usual size, in its default FP32
        _fx("vlbi_6ant_fp32", 6, 1024, 15625, False, 64, "fp32"),
        # sixteen antennas, 256 MHz, one second: the benchmark's workload in FP32 (four FFT blocks)
        _fx("array_16ant_fp32", 16, 4096, 62500, False, 256, "fp32"),
        # the same array, half a second, with FP16 spectra: the usual choice for production
        _fx("array_16ant_fp16", 16, 4096, 31250, False, 256, "fp16"),
        # and one second with FP8 spectra, for surveys with long integrations
        _fx("array_16ant_fp8", 16, 4096, 62500, False, 256, "fp8"),
        # thirty-two antennas, 512 MHz, a quarter of a second, 8192 channels (16384-point windows)
        _fx("array_32ant_fp16", 32, 8192, 15625, False, 512, "fp16"),
        # sixty-four antennas, 8-bit complex beamformer output, 16384 channels: the largest arrays
        _fx("array_64ant_complex_fp16", 64, 16384, 1953, True, 128, "fp16"),
        # spectral line: ten antennas, 16384 channels from 32768-point windows, FP32, an odd number of FFTs
        _fx("line_10ant_fp32", 10, 16384, 3901, False, 64, "fp32"),
        # seven stations of 8-bit complex data with few channels: short windows, an odd antenna count
        _fx("vlbi_7ant_complex_fp16", 7, 512, 32003, True, 32, "fp16"),
        # four uneven scans queued together as one graph
        {"name": "batch_4jobs_fp16", "kind": "batch", "precision": "fp16", "njobs": 4, "jobs_seed": 3, "scale": 0.25},
        # the X-stage alone on channelised voltages, as the reference's GPU kernels are called
        {"name": "xcorr_16ant_fp32", "kind": "xcorr", "nant": 16, "nchan": 1024, "nfft": 2048, "fftwidth": 1024,
         "precision": "fp32", "autos": True},
        # a stretch of four sub-integrations streamed from pinned host memory through the ingest pipeline
        {"name": "stream_6ant_fp32", "kind": "stream", "nant": 6, "nchan": 1024, "nfft": 15625, "complex": False,
         "mhz": 64.0, "precision": "fp32", "rotator": "exact", "autos": True, "nsub": 4},
    ]


# limits of a drawn case: samples, multiply-accumulate operations and visibilities of the largest listed ones
_MOST_SAMPLES = 16 * 2 * 62500 * 8192
_MOST_FLOPS = 1.1e12
_MOST_VIS = 2080 * 4 * 16384


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["process", "batch", "xcorr", "stream"], [12, 1, 2, 1])[0]
    if kind == "batch":
        return {"kind": "batch", "precision": rng.choice(["fp32", "fp16"]), "njobs": rng.randint(2, 6),
                "jobs_seed": rng.randint(1, 1000), "scale": rng.uniform(0.05, 0.25)}
    if kind == "xcorr":
        nchan = 128 * rng.randint(1, 16)
        nant = rng.randint(2, 32)
        nfft = max(8, min(_log_uniform(rng, 16, 4096), int(2 ** 26 / (2 * nant * nchan))))
        return {"kind": "xcorr", "nant": nant, "nchan": nchan, "nfft": nfft, "fftwidth": nchan * rng.choice([1, 2]),
                "precision": rng.choice(["fp32", "fp16"]), "autos": rng.random() < 0.5}
    while True:
        cplx = rng.random() < 0.35
        nchan = 2 ** (rng.randint(8, 14) if cplx else rng.randint(7, 14))
        F = nchan if cplx else 2 * nchan
        nant = _log_uniform(rng, 2, 64)
        precision = rng.choices(["fp32", "fp16", "fp8"], [5, 4, 1])[0]
        # FP8 spectra are for long integrations, over which their rounding averages out; FP16 for production lengths
        lo = {"fp32": 4, "fp16": 2500, "fp8": 50000}[precision]
        nbl = nant * (nant + 1) // 2
        hi = min(62500.0, _MOST_SAMPLES / (2 * nant * F), _MOST_FLOPS / (32.0 * nbl * nchan))
        if nbl * 4 * nchan > _MOST_VIS or hi < 2 * lo and precision != "fp8" or hi < lo:
            continue
        nfft = _log_uniform(rng, lo, hi)
        square = math.isqrt(nchan) ** 2 == nchan
        c = {"kind": kind, "nant": nant, "nchan": nchan, "nfft": nfft, "complex": cplx,
             "mhz": float(rng.choice([32, 64, 128, 256])), "precision": precision,
             "rotator": "fxkernel" if square and not cplx and rng.random() < 0.25 else "exact", "autos": rng.random() < 0.8}
        if kind == "stream":
            c["nfft"] = max(4, nfft // 4)
            if precision != "fp32":
                c["precision"] = "fp32"
            c["nsub"] = rng.randint(2, 4)
        return c


# ---------------------------------------------------------------- inputs
def _workload(c, seed):
    return synth.Workload(nant=c["nant"], nchan=c["nchan"], nfft=c["nfft"], nbit=8 if c["complex"] else 2,
                          is_complex=c["complex"], lo_hz=8.4e9, bw_hz=c["mhz"] * 1e6, rho=0.05, seed=seed)


def _code_table():
    """Byte for each of 65536 equally likely numbers: four independent 2-bit codes of unit-variance noise
    quantised at +-0.98 sigma."""
    hi = 0.5 * math.erfc(0.98 / math.sqrt(2.0))
    p = np.array([hi, 0.5 - hi, 0.5 - hi, hi])
    b = np.arange(256)
    pb = p[b & 3] * p[(b >> 2) & 3] * p[(b >> 4) & 3] * p[b >> 6]
    cum = np.cumsum(pb) / pb.sum()
    return np.searchsorted(cum, (np.arange(65536) + 0.5) / 65536.0).clip(0, 255).astype(np.uint8)


def _voltages(w, seed):
    """One buffer per antenna: receiver noise with a few per cent of a common signal, quantised and packed."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    n = w.bytes_per_antenna
    rho = w.rho
    if w.is_complex:
        common = torch.randn(n, generator=gen, device="cuda", dtype=torch.float32) * (w.sigma8 * math.sqrt(rho))

        def one():
            x = torch.randn(n, generator=gen, device="cuda", dtype=torch.float32).mul_(w.sigma8 * math.sqrt(1.0 - rho))
            return x.add_(common).round_().clamp_(-127, 127).to(torch.int8).view(torch.uint8)
    else:
        table = torch.from_numpy(_code_table()).cuda()

        def noise():
            return table[torch.randint(0, 65536, (n,), generator=gen, device="cuda", dtype=torch.int32)]
        common = noise()

        def one():
            own = noise()
            return torch.where(torch.rand(n, generator=gen, device="cuda", dtype=torch.float32) < rho, common, own)
    return [one() for _ in range(w.nant)]


class _DeviceArray:
    """Device memory of the library as an array that torch can take without a copy; keeps its owner (the kernel or
    batch that frees it) alive as long as the tensor."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<c8", "data": (ptr, False), "version": 3}


def _visibility_view(owner, ptr, nbl, nchan):
    return torch.as_tensor(_DeviceArray(owner, int(ptr), (nbl, 4, nchan)), device="cuda")


def _nbl(c):
    return c["nant"] * (c["nant"] - 1) // 2 + (c["nant"] if c["autos"] else 0)


def _jobs(c):
    """The uneven scans of a batch: antennas, channels, formats and lengths as the suite's eight-job workload draws
    them, shortened to `scale` of their length."""
    ws = synth.config3_jobs(c["jobs_seed"])[:c["njobs"]]
    jobs = []
    for w in ws:
        nfft = max(2500 if c["precision"] != "fp32" else 16, int(w.nfft * c["scale"]))
        jobs.append({"nant": w.nant, "nchan": w.nchan, "nfft": min(nfft, w.nfft), "complex": w.is_complex,
                     "mhz": w.bw_hz / 1e6, "precision": c["precision"], "rotator": "exact", "autos": True})
    return jobs


def _channelised(c, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    n = 2 * c["nant"] * c["nfft"] * c["fftwidth"]
    return torch.randn(2 * n, generator=gen, device="cuda", dtype=torch.float32)


# ---------------------------------------------------------------- one pass
def prepare(case, seed):
    c = case
    if c["kind"] == "process":
        w = _workload(c, seed)
        poly, fso = synth.delay_model(w)
        inputs = _voltages(w, seed)
        fx = G.FxKernel(w.nant, w.nchan, w.nfft, w.nbit, w.lo_hz, w.bw_hz, w.is_complex, precision=c["precision"],
                        rotator=c["rotator"], autos=c["autos"])
        return {"case": c, "fx": fx, "inputs": inputs, "poly": poly, "fso": fso,
                "vis": _visibility_view(fx, fx.device_visibilities_ptr(), _nbl(c), c["nchan"])}
    if c["kind"] == "batch":
        descr, shapes = [], []
        for k, j in enumerate(_jobs(c)):
            w = _workload(j, seed * 16 + k)
            poly, fso = synth.delay_model(w)
            descr.append({"nant": w.nant, "nchan": w.nchan, "nfft": w.nfft, "nbit": w.nbit, "lo": w.lo_hz, "bw": w.bw_hz,
                          "is_complex": w.is_complex, "precision": c["precision"], "inputs": _voltages(w, seed * 16 + k),
                          "poly": poly, "fso": fso})
            shapes.append((_nbl(j), w.nchan))
        torch.cuda.synchronize()
        b = Batch(descr)
        vis = [_visibility_view(b, G.lib().gxc_device_visibilities(b.handle(i)), *s) for i, s in enumerate(shapes)]
        return {"case": c, "batch": b, "vis": vis}
    if c["kind"] == "xcorr":
        return {"case": c, "ants": _channelised(c, seed),
                "out": torch.zeros((_nbl(c), 4, c["nchan"]), dtype=torch.complex64, device="cuda")}
    # stream: pinned host buffers of two sub-integrations that alternate, and device buffers for the results
    w = _workload(c, seed)
    poly, fso = synth.delay_model(w)
    host = [[x.cpu().pin_memory() for x in _voltages(w, seed + s)] for s in (0, 1)]
    pipe = Pipeline(w.nant, w.nchan, w.nfft, w.nbit, w.lo_hz, w.bw_hz, w.is_complex, slots=2, integrate=True,
                    precision=c["precision"], rotator=c["rotator"], autos=c["autos"])
    out = [torch.zeros((_nbl(c), 4, c["nchan"]), dtype=torch.complex64, device="cuda") for _ in range(c["nsub"])]
    return {"case": c, "pipe": pipe, "host": host, "poly": poly, "fso": fso, "out": out}


def run(state):
    c = state["case"]
    stream = torch.cuda.current_stream().cuda_stream
    if c["kind"] == "process":
        fx = state["fx"]
        fx.setInputData(state["inputs"])
        fx.setDelays(state["poly"], state["fso"])
        fx.process(stream, sync=False)
        return state["vis"]
    if c["kind"] == "batch":
        state["batch"].launch(stream)
        return state["vis"]
    if c["kind"] == "xcorr":
        st = G.lib().gxc_xcorr(ctypes.c_void_p(state["ants"].data_ptr()), c["nant"], c["nfft"], c["nchan"], c["fftwidth"],
                               PRECISIONS[c["precision"]], 0, int(c["autos"]), ctypes.c_void_p(state["out"].data_ptr()),
                               ctypes.c_void_p(stream))
        if st:
            raise RuntimeError(f"gxc_xcorr: status {st}")
        return state["out"]
    pipe = state["pipe"]
    for k, out in enumerate(state["out"]):
        seq = pipe.submit(state["host"][k & 1], state["poly"], state["fso"], out)
    pipe.wait(seq)
    return state["out"]


# ---------------------------------------------------------------- what a pass cannot do without
def _work_one(c):
    F = c["nchan"] if c["complex"] else 2 * c["nchan"]
    nbl = _nbl(c)
    data = c["nant"] * c["nfft"] * F * (4 if c["complex"] else 0.5)
    # real data: half of a complex transform's operations give the half band that is kept
    fft = 2 * c["nant"] * c["nfft"] * (5.0 if c["complex"] else 2.5) * F * math.log2(F)
    products = 8.0 * 4 * nbl * c["nchan"] * c["nfft"]
    return data + nbl * 4 * c["nchan"] * 8.0, fft + products


def work(case):
    c = case
    if c["kind"] == "batch":
        parts = [_work_one(j) for j in _jobs(c)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    if c["kind"] == "xcorr":
        return {"bytes": 2.0 * c["nant"] * c["nfft"] * c["nchan"] * 8 + _nbl(c) * 4 * c["nchan"] * 8.0,
                "flops": 8.0 * 4 * _nbl(c) * c["nchan"] * c["nfft"]}
    b, f = _work_one(c)
    n = c.get("nsub", 1)
    return {"bytes": b * n, "flops": f * n}


# ---------------------------------------------------------------- the result in 64 bits
def _windows(c, poly, fso):
    """Per antenna and FFT: first sample, validity, fractional delay (s), and the delay line a*x + b of the FFT."""
    F = c["nchan"] if c["complex"] else 2 * c["nchan"]
    bw = c["mhz"] * 1e6
    Ts = 1.0 / bw if c["complex"] else 1.0 / (2.0 * bw)
    i = np.arange(c["nfft"], dtype=np.float64)[None, :]
    p = [poly[:, k][:, None] for k in range(3)]

    def delay(x):
        return p[0] * x * x + p[1] * x + p[2]
    d0, d1, d2 = delay(i), delay(i + 0.5), delay(i + 1.0)
    a = d2 - d0
    b = d0 + (d1 - (a * 0.5 + d0)) / 3.0
    ndf = (a * 0.5 + b - fso[:, None]) / Ts
    nd = np.trunc(ndf + 0.5)
    frac = -((ndf - nd) * Ts)
    off = i * F - nd
    last = float((c["nfft"] - 1) * F)
    low, high = off == -1, off == last + 1
    off = off + low - high
    frac = frac + low * Ts - high * Ts
    return off.astype(np.int64), (off >= 0) & (off <= last), frac, a, b


def _exact_process(c, inputs, poly, fso):
    F = c["nchan"] if c["complex"] else 2 * c["nchan"]
    nant, nchan, nfft = c["nant"], c["nchan"], c["nfft"]
    lo, bw = 8.4e9, c["mhz"] * 1e6
    off, valid, frac, a, b = _windows(c, poly, fso)
    dev = inputs[0].device
    f64 = dict(dtype=torch.float64, device=dev)
    n = torch.arange(F, device=dev)
    if c["rotator"] == "fxkernel":  # tables of stride entries that advance stride samples per substride samples
        stride = math.isqrt(nchan)
        turns_n = (n % (F // stride)).to(torch.float64) + (n // (F // stride)).to(torch.float64) * stride
    else:
        turns_n = n.to(torch.float64)
    chan = torch.arange(nchan, **f64)
    levels = torch.tensor([-3.3359, -1.0, 1.0, 3.3359], dtype=torch.float32, device=dev).to(torch.float64)
    V = torch.zeros((nchan, 2 * nant, 2 * nant), dtype=torch.complex128, device=dev)
    step = max(1, min(nfft, int((2 << 30) / (2 * nant * F * 16))))
    for t0 in range(0, nfft, step):
        t1 = min(nfft, t0 + step)
        X = torch.empty((nchan, 2 * nant, t1 - t0), dtype=torch.complex128, device=dev)
        for j in range(nant):
            o = torch.from_numpy(np.where(valid[j, t0:t1], off[j, t0:t1], 0)).to(dev)
            ok = torch.from_numpy(valid[j, t0:t1]).to(**f64)
            pos = o[:, None] + n[None, :]
            c0 = torch.from_numpy(np.mod((b[j, t0:t1] - np.trunc(b[j, t0:t1])) * lo, 1.0)).to(dev)
            c1 = torch.from_numpy(a[j, t0:t1] * lo / F).to(dev)
            turns = -torch.remainder(c0[:, None] + c1[:, None] * turns_n[None, :], 1.0)
            rot = torch.polar(ok[:, None].expand(-1, F).contiguous(), 2.0 * math.pi * turns)
            slope = torch.from_numpy(bw / nchan * frac[j, t0:t1]).to(dev)
            phase = torch.polar(torch.ones((t1 - t0, nchan), **f64), 2.0 * math.pi * slope[:, None] * chan[None, :])
            for pol in range(2):
                if c["complex"]:
                    v = inputs[j].view(torch.int8).view(-1, 4)[pos.reshape(-1), 2 * pol:2 * pol + 2].to(torch.float64)
                    x = torch.view_as_complex(v).view(pos.shape)
                else:
                    code = (inputs[j][pos >> 1] >> (4 * (pos & 1) + 2 * pol).to(torch.uint8)) & 3
                    x = levels[code.to(torch.int64)]
                S = torch.fft.fft(x * rot, dim=1)[:, :nchan] * phase
                X[:, 2 * j + pol, :] = S.t()
        V += X @ X.conj().transpose(1, 2)
        del X
    ok = torch.from_numpy(valid).to(**f64)
    both = (ok @ ok.t()).clamp(min=1.0)
    pairs = [(j, k) for j in range(nant) for k in range(j + 1, nant)] + ([(j, j) for j in range(nant)] if c["autos"] else [])
    jj = torch.tensor([p[0] for p in pairs], device=dev)
    kk = torch.tensor([p[1] for p in pairs], device=dev)
    out = torch.empty((len(pairs), 4, nchan), dtype=torch.complex128, device=dev)
    for l in range(2):
        for m in range(2):
            out[:, 2 * l + m, :] = V[:, 2 * jj + l, 2 * kk + m].t() / both[jj, kk][:, None]
    return out


def exact(case, seed):
    c = case
    if c["kind"] == "process":
        w = _workload(c, seed)
        return _exact_process(c, _voltages(w, seed), *synth.delay_model(w))
    if c["kind"] == "batch":
        out = []
        for k, j in enumerate(_jobs(c)):
            w = _workload(j, seed * 16 + k)
            out.append(_exact_process(j, _voltages(w, seed * 16 + k), *synth.delay_model(w)))
        return out
    if c["kind"] == "xcorr":
        nant, nfft, nchan = c["nant"], c["nfft"], c["nchan"]
        x = torch.view_as_complex(_channelised(c, seed).view(2 * nant, nfft, c["fftwidth"], 2))[:, :, :nchan]
        V = torch.zeros((nchan, 2 * nant, 2 * nant), dtype=torch.complex128, device=x.device)
        for t0 in range(0, nfft, 256):
            X = x[:, t0:t0 + 256].to(torch.complex128).permute(2, 0, 1)
            V += X @ X.conj().transpose(1, 2)
        pairs = [(j, k) for j in range(nant) for k in range(j + 1, nant)] + ([(j, j) for j in range(nant)] if c["autos"] else [])
        jj = torch.tensor([p[0] for p in pairs], device=x.device)
        kk = torch.tensor([p[1] for p in pairs], device=x.device)
        return torch.stack([V[:, 2 * jj + l, 2 * kk + m].t() / nfft for l in range(2) for m in range(2)], dim=1)
    w = _workload(c, seed)
    delays = synth.delay_model(w)
    two = [_exact_process(c, _voltages(w, seed + s), *delays) for s in (0, 1)]
    return [two[k & 1] for k in range(c["nsub"])]
