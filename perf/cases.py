"""What the correlator is timed on: calls of the public entry points over the
range of jobs a user runs.

Kinds of case
  subint  one subint through ``Correlator.subint_device``: station data, control
          words and delay interpolators in, the Core result array out, all on
          the device (how a Core thread, a serving slot or the bench drives it)
  host    the same subint through ``Correlator.subint`` from pinned host buffers
  batch   one subint of each of several uneven resident jobs replayed as one
          CUDA graph (``Batch``)
  mux     one stretch of multi-thread VDIF through ``VdifMux`` (station ingest)

Station streams are noise with a common component that carries the station's
delay and fringe phase, quantised and packed as VDIF with a fraction of invalid
frames; delays are seeded quadratics.
"""
import math
import random

import numpy as np
import torch

from difx_b200 import capi
from difx_b200.gxcorr import Batch, Correlator, VdifMux
from difx_b200.jobfiles import JobSpec, Subband

PAYLOAD = 8000                 # VDIF payload bytes per frame
HEADER = 32
START_SEC = 1                  # the subint starts this long after the scan start
XSTEP = {"fp32": capi.GX_XSTEP_FP32, "fp16": capi.GX_XSTEP_TC_FP16, "split": capi.GX_XSTEP_TC_FP16_HILO,
         "auto": capi.GX_XSTEP_AUTO}


def _subint(name, stations, pols, subbands, bw, nchan, nbits, blocks, xstep, kind="subint", cplx=False, lower=False,
            delay_us=20000.0, rho=0.02, avg=1, pcal=False, muxed=False):
    return {"name": name, "kind": kind, "stations": stations, "pols": pols, "subbands": subbands, "bw": bw,
            "nchan": nchan, "nbits": nbits, "cplx": cplx, "lower": lower, "blocks": blocks, "xstep": xstep,
            "delay_us": delay_us, "rho": rho, "avg": avg, "pcal": pcal, "muxed": muxed}


def listed():
    return [
        # a small real-time array's 8 ms subint: launches and host latency decide
        _subint("small_4st_8ms", 4, 2, 4, 16, 128, 2, 1000, "fp32", rho=0.05),
        # the same array at 200 ms subints, short transforms
        _subint("array_4st_128ch", 4, 2, 4, 16, 128, 2, 25000, "fp32", rho=0.05),
        # 16 stations at 2 Gbps, full polarisation, FP32 visibilities
        _subint("array_16st_256ch", 16, 2, 8, 32, 256, 2, 6250, "fp32"),
        # 64 dual-polarisation stations, 8-bit complex, tensor-core X-step with split operands
        _subint("wide_64st_4096ch_split", 64, 2, 4, 64, 4096, 8, 500, "split", cplx=True, rho=0.01),
        # its 2-bit real variant with single FP16 operands, 8192-point transforms
        _subint("wide_64st_2bit_fp16", 64, 2, 4, 64, 4096, 2, 500, "fp16", rho=0.01),
        # the same array with FP32 visibilities, a short subint with an odd block count
        _subint("wide_64st_4096ch_fp32", 64, 2, 4, 64, 4096, 8, 125, "fp32", cplx=True, rho=0.01),
        # a 1-bit survey job of an odd station count, very short transforms
        _subint("narrow_11st_64ch_1bit", 11, 1, 8, 8, 64, 1, 25013, "fp32", delay_us=100.0, rho=0.1),
        # spectral-line job: 8-bit real lower sidebands, phase-cal tones, averaged output
        _subint("line_8st_4096ch_pcal", 8, 2, 2, 16, 4096, 8, 1563, "fp32", lower=True, delay_us=100.0, avg=8, pcal=True),
        # multiplexed multi-thread VDIF with per-thread validity
        _subint("muxed_6st_512ch", 6, 2, 4, 32, 512, 2, 6251, "fp32", delay_us=100.0, muxed=True),
        # real-time input from host memory: upload, correlate, read back
        _subint("host_16st_256ch", 16, 2, 8, 32, 256, 2, 5000, "fp32", kind="host"),
        # uneven jobs of a correlator that serves many projects at once
        {"name": "batch_8_uneven", "kind": "batch", "jobs": 8, "mix": 4040, "samples": 1.5e7},
        # ingest of a 16-thread station
        {"name": "mux_16thread", "kind": "mux", "threads": 16, "nbits": 2, "fps": 4000, "frames": 1000},
    ]


def _draw_job(rng, most_samples, most_flops):
    """One job of the listed ranges: sizes over their logarithm, at most so many station-band samples and X-step operations."""
    while True:
        stations = int(round(math.exp(rng.uniform(math.log(3), math.log(64)))))
        pols = rng.choice([1, 2, 2])
        nbits = rng.choice([1, 2, 2, 8])
        cplx = nbits == 8 and rng.random() < 0.6
        subbands = rng.choice([1, 2, 4, 8])
        ts = pols * subbands * nbits * (2 if cplx else 1)
        if ts < 8 or ts > 128 or (not cplx and ts > 64):
            continue
        nchan = rng.choice([64, 128, 256, 512, 1024, 2048, 4096])
        inputs = stations * pols
        tensor = 48 <= inputs <= 128
        xstep = rng.choice(["split", "split", "fp16", "fp32"]) if tensor else "fp32"
        fft = nchan if cplx else 2 * nchan
        per_block = stations * pols * subbands * fft
        samples = math.exp(rng.uniform(math.log(8e6), math.log(most_samples)))
        blocks = int(samples / per_block)
        if xstep == "fp32":
            blocks = min(blocks, int(most_flops / (4.0 * inputs * (inputs + 1) * nchan * subbands)))
        results = stations * (stations - 1) // 2 * pols * pols * nchan * subbands
        if blocks < 3 or blocks > 60000 or results > 1.4e8:
            continue
        return _subint("", stations, pols, subbands, rng.choice([8, 16, 32, 64]), nchan, nbits, blocks, xstep, cplx=cplx,
                       lower=rng.random() < 0.25, delay_us=rng.choice([100.0, 20000.0]), rho=rng.choice([0.005, 0.02, 0.1]),
                       avg=rng.choice([1, 1, 1, 1, 4]))


def draw(rng):
    u = rng.random()
    if u < 0.07:
        return {"kind": "batch", "jobs": rng.randint(4, 12), "mix": rng.randint(1, 10 ** 6),
                "samples": math.exp(rng.uniform(math.log(4e6), math.log(3e7)))}
    if u < 0.14:
        return {"kind": "mux", "threads": rng.choice([2, 4, 8, 16]), "nbits": rng.choice([1, 2, 8]), "fps": 4000,
                "frames": int(math.exp(rng.uniform(math.log(100), math.log(2000))))}
    case = _draw_job(rng, 1.0e9, 1.2e11)
    if u < 0.22 and case["stations"] <= 24:
        case = dict(_draw_job(rng, 2.0e8, 3.0e10), kind="host")
    elif u < 0.30:
        case.update(nchan=max(512, case["nchan"]), nbits=2, cplx=False, pols=2, subbands=4, stations=min(case["stations"], 12),
                    bw=32, xstep="fp32", muxed=True, avg=1, lower=False, blocks=rng.randint(500, 2500))
    elif u < 0.38:
        case.update(nchan=max(1024, case["nchan"]), bw=16, stations=min(case["stations"], 10), xstep="fp32",
                    pcal=True, blocks=rng.randint(300, 1500))
    case.pop("name", None)
    return case


# ------------------------------------------------------------- what a case is

def _jobs(case):
    """The correlation jobs of a case."""
    if case["kind"] != "batch":
        return [case]
    rng = random.Random(case["mix"])
    out = []
    while len(out) < case["jobs"]:
        j = _draw_job(rng, case["samples"], 2.0e9)
        if j["stations"] <= 32:
            out.append(dict(j, xstep="auto", avg=1, delay_us=100.0))
    return out


def _fft(c):
    return c["nchan"] if c["cplx"] else 2 * c["nchan"]


def _rate(c):
    return c["bw"] * 10 ** 6 * (1 if c["cplx"] else 2)     # time samples per second


def _bits(c):
    return c["pols"] * c["subbands"] * c["nbits"] * (2 if c["cplx"] else 1)   # per time sample of all bands


def _lo(c, f):
    return 6000.0 + c["bw"] * f + (c["bw"] if c["lower"] else 0.0)


def _spec(c):
    return JobSpec(nstations=c["stations"], pols=("R", "L")[:c["pols"]],
                   subbands=[Subband(_lo(c, f), float(c["bw"]), "L" if c["lower"] else "U", c["nchan"])
                             for f in range(c["subbands"])],
                   nbits=c["nbits"], sampling="COMPLEX" if c["cplx"] else "REAL", payload_bytes=PAYLOAD,
                   subint_ns=c["blocks"] * (1000 * c["nchan"] // c["bw"]), execute_seconds=20, int_time=1.0,
                   chans_to_avg=c["avg"], pcal_interval_mhz=1 if c["pcal"] else 0,
                   mux_threads=c["pols"] * c["subbands"] if c["muxed"] else 0)


def _delays(c, seed):
    """Quadratic delay model of each station, us, in seconds from the subint start."""
    rng = np.random.default_rng([seed, 5])
    n = c["stations"]
    return np.stack([rng.uniform(-0.9, 0.9, n) * c["delay_us"], rng.uniform(-3.0, 3.0, n), rng.uniform(-1e-4, 1e-4, n)], 1)


def _products(c):
    if c["pols"] == 1:
        return [(0, 0)]
    return [(0, 0), (1, 1), (0, 1), (1, 0)]


# ------------------------------------------------------------- station data

def _streams(c, seed):
    """Per station: packed VDIF frames on the device, (sec, ns) of the first one, its sample count."""
    dev = "cuda"
    gen = torch.Generator(device=dev).manual_seed(1000003 * seed + 17)
    tau = _delays(c, seed)
    fs, nb, cplx = _rate(c), c["pols"] * c["subbands"], c["cplx"]
    fsamp = PAYLOAD * 8 // _bits(c)
    fps = fs // fsamp
    span = c["blocks"] * _fft(c)
    rng = np.random.default_rng([seed, 7])
    windows = []
    for s in range(c["stations"]):
        t1 = span / fs
        d = [np.polyval(tau[s][::-1], t) * 1e-6 for t in np.linspace(0.0, t1, 9)]
        f0 = int(math.floor((START_SEC - max(d) - 2e-6) * fps)) - 1
        f1 = int(math.ceil((START_SEC + t1 - min(d) + _fft(c) / fs + 2e-6) * fps)) + 1
        windows.append((f0, f1 - f0))
    # one common signal per band over what the delays reach (analytic for real sampling)
    first = int(START_SEC * fs) - 4 * _fft(c) - 4 * fsamp
    total = span + 8 * _fft(c) + 8 * fsamp
    sky = torch.randn(nb, total, dtype=torch.complex64, device=dev, generator=gen)
    if not cplx:
        z = torch.fft.fft(sky.real.contiguous().to(torch.complex64))
        z[:, total // 2:] = 0
        sky = torch.fft.ifft(z) * 2
        del z
    lo = torch.tensor([_lo(c, b // c["pols"]) for b in range(nb)], dtype=torch.float64, device=dev)
    out = []
    for s, (f0, nf) in enumerate(windows):
        n = nf * fsamp
        u = torch.arange(f0 * fsamp, f0 * fsamp + n, device=dev, dtype=torch.float64)
        t = u / fs - START_SEC
        d = tau[s][0] + tau[s][1] * t + tau[s][2] * t * t
        at = (u + torch.round(d * (fs * 1e-6)) - first).long().clamp_(0, total - 1)
        x = torch.empty(nb, n, dtype=torch.complex64 if cplx else torch.float32, device=dev)
        for b in range(nb):
            ph = torch.remainder(lo[b] * d, 1.0).float() * (2 * math.pi)
            v = sky[b][at] * torch.polar(torch.ones_like(ph), ph)
            noise = torch.randn(n, dtype=x.dtype, device=dev, generator=gen)
            x[b] = math.sqrt(c["rho"]) * (v if cplx else v.real) + math.sqrt(1 - c["rho"]) * noise
        if c["pcal"]:    # 1 MHz comb, as the stations inject it
            k = torch.arange(n, device=dev, dtype=torch.float64) + f0 * fsamp
            comb = sum(torch.polar(torch.full_like(k, 0.1), 2 * math.pi * torch.remainder(k * (m * 10 ** 6 / fs), 1.0) + m)
                       for m in range(1, c["bw"]))
            x += (comb if cplx else comb.real).to(x.dtype)
        parts = torch.view_as_real(x).permute(1, 0, 2).reshape(n, 2 * nb) if cplx else x.t()
        nbits = c["nbits"]
        if nbits == 1:
            codes = (parts >= 0).to(torch.uint8)
        elif nbits == 2:
            codes = ((parts >= -0.98).to(torch.uint8) + (parts >= 0) + (parts >= 0.98)).to(torch.uint8)
        else:
            codes = torch.clamp(torch.round(128.0 + 16.0 * parts), 0, 255).to(torch.uint8)
        codes = codes.contiguous()
        if nbits < 8:
            per = 8 // nbits
            q = codes.reshape(-1, per).to(torch.int32)
            codes = sum(q[:, i] << (i * nbits) for i in range(per)).to(torch.uint8)
        fr = f0 + np.arange(nf)
        bad = rng.random(nf) < 0.01
        h = np.zeros((nf, 8), np.uint32)
        h[:, 0] = (3600 + fr // fps).astype(np.uint32) | (bad.astype(np.uint32) << 31)
        h[:, 1] = (fr % fps).astype(np.uint32)
        h[:, 2] = (PAYLOAD + HEADER) // 8 | (nb.bit_length() - 1 << 24)
        h[:, 3] = (cplx << 31) | (nbits - 1 << 26) | s
        if c["muxed"]:   # some frames lack a thread or two
            full = (1 << nb) - 1
            mask = np.full(nf, full)
            for f in np.nonzero(rng.random(nf) < 0.05)[0]:
                for k in rng.integers(0, nb, 2):
                    mask[f] &= ~(1 << int(k))
            h[:, 4] = (4 << 24) | (nb << 16)
            h[:, 5] = 0xACABFEED
            h[:, 6] = mask
        buf = torch.empty(nf, PAYLOAD + HEADER, dtype=torch.uint8, device=dev)
        buf[:, :HEADER] = torch.from_numpy(h.view(np.uint8)).to(dev)
        buf[:, HEADER:] = codes.reshape(nf, PAYLOAD)
        out.append((buf, h, f0 // fps, int(round((f0 % fps) * 1e9 / fps))))
    return out


def _interp(c, seed):
    """Delay interpolators of the subint: quadratics in FFT blocks."""
    tau, bd = _delays(c, seed), 1e-6 * c["nchan"] / c["bw"]
    return np.stack([tau[:, 2] * bd * bd, tau[:, 1] * bd, tau[:, 0]], 1)


def _control(c, sec, ns):
    n = c["blocks"]
    w = np.full((n + 29) // 30, (1 << 30) - 1, np.int32)
    if n % 30:
        w[-1] = (1 << (n % 30)) - 1
    return np.concatenate([np.array([0, sec, ns], np.int32), w])


def _sections(corr, c, res):
    """The parts of a result array: cross records, their weights, autocorrelations, their weights, phase-cal tones."""
    rl, bl, bw, ac, acw = corr.offsets()
    w0 = int(bw[bw >= 0].min()) if (bw >= 0).any() else int(ac[0])
    bpa = 2 if c["pols"] == 2 else 1
    a1 = int(acw[0])
    e = int(acw[-1]) + (bpa * c["pols"] * c["subbands"] + 1) // 2
    out = {"cross": res[:w0], "weights": res[w0:int(ac[0])], "auto": res[int(ac[0]):a1], "auto_weights": res[a1:e]}
    if c["pcal"]:
        out["tones"] = res[e:rl]
    return out


_stream = None


def _work_stream():
    """The program's own stream: one for all its correlators."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def _device_job(c, seed, budget=0):
    streams = _streams(c, seed)
    cws = [_control(c, sec, ns) for _, _, sec, ns in streams]
    sd = capi.SubintDesc(0, START_SEC, 0, 0.0, [b.data_ptr() for b, *_ in streams], [b.numel() for b, *_ in streams],
                         [w.ctypes.data for w in cws], len(cws[0]), _interp(c, seed))
    corr = Correlator.from_desc(capi.job_desc_from_spec(_spec(c), xstep=XSTEP[c["xstep"]], spectra_budget_bytes=budget))
    return corr, sd, [b for b, *_ in streams], cws


def _mux_input(case, seed):
    fb, th = PAYLOAD + HEADER, case["threads"]
    n = th * case["frames"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    buf = torch.randint(0, 256, (n, fb), dtype=torch.uint8, device="cuda", generator=gen)
    k = np.arange(n)
    fr = k // th
    rng = np.random.default_rng([seed, 9])
    h = np.zeros((n, 8), np.uint32)
    h[:, 0] = (1000 + fr // case["fps"]).astype(np.uint32) | ((rng.random(n) < 0.005).astype(np.uint32) << 31)
    h[:, 1] = (fr % case["fps"]).astype(np.uint32) | (40 << 24)
    h[:, 2] = fb // 8
    h[:, 3] = 0x4142 | ((k % th).astype(np.uint32) << 16) | (case["nbits"] - 1 << 26)
    buf[:, :HEADER] = torch.from_numpy(h.view(np.uint8)).cuda()
    keep = rng.random(n) >= 0.002          # a few packets are lost
    keep[:th] = True
    return buf[torch.from_numpy(keep).cuda()].reshape(-1)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mux":
        src = _mux_input(case, seed)
        m = VdifMux(PAYLOAD + HEADER, case["fps"], case["nbits"], list(range(case["threads"])), nsort=32,
                    ngap=case["fps"] // 4, flags=0x02 | 0x40)
        dest = torch.zeros(m.output_frame_bytes * (case["frames"] + 1), dtype=torch.uint8, device="cuda")
        state = {"kind": kind, "mux": m, "src": src, "dest": dest, "stream": _work_stream()}
    elif kind == "batch":
        parts = [_device_job(c, seed * 100 + i, 2 << 30) for i, c in enumerate(_jobs(case))]
        res = [torch.empty(p[0].result_length, dtype=torch.complex64, device="cuda") for p in parts]
        b = Batch([p[0] for p in parts], [r.data_ptr() for r in res], mode="graph", nstreams=4)
        state = {"kind": kind, "batch": b, "subs": [p[1] for p in parts], "keep": parts,
                 "out": [_sections(p[0], c, r) for p, c, r in zip(parts, _jobs(case), res)]}
    else:
        corr, sd, bufs, cws = _device_job(case, seed)
        if kind == "host":
            bufs = [b.cpu().pin_memory() for b in bufs]
            sd = capi.SubintDesc(0, START_SEC, 0, 0.0, [b.data_ptr() for b in bufs], [b.numel() for b in bufs],
                                 [w.ctypes.data for w in cws], len(cws[0]), _interp(case, seed))
            res = torch.empty(corr.result_length, dtype=torch.complex64).pin_memory()
            state = {"kind": kind, "corr": corr, "sd": sd, "keep": (bufs, cws, res), "res": res.numpy(),
                     "out": _sections(corr, case, res)}
        else:
            res = torch.empty(corr.result_length, dtype=torch.complex64, device="cuda")
            state = {"kind": kind, "corr": corr, "sd": sd, "keep": (bufs, cws), "res": res,
                     "out": _sections(corr, case, res), "stream": _work_stream()}
    torch.cuda.synchronize()
    return state


def run(state):
    kind = state["kind"]
    if kind == "subint":
        state["corr"].subint_device(state["sd"], state["res"].data_ptr(), state["stream"].cuda_stream)
    elif kind == "host":
        state["corr"].subint(state["sd"], state["res"])
    elif kind == "batch":
        state["batch"].run(state["subs"])
    else:
        st = state["mux"].run(state["src"].data_ptr(), state["src"].numel(), state["dest"].data_ptr(),
                              state["dest"].numel(), -1, state["stream"].cuda_stream)
        return {"frames": state["dest"], "output_frames": int(st.output_frames), "src_used": int(st.src_used)}
    return state["out"]


def work(case):
    if case["kind"] == "mux":
        n = case["threads"] * case["frames"] * (PAYLOAD + HEADER)
        return {"bytes": 2 * n, "flops": 0}
    total = {"bytes": 0, "flops": 0}
    for c in _jobs(case):
        inputs, bands = c["stations"] * c["pols"], c["pols"] * c["subbands"]
        samples = c["stations"] * bands * c["blocks"] * _fft(c)
        pairs = c["stations"] * (c["stations"] - 1) // 2 * c["pols"] ** 2 + c["stations"] * c["pols"] ** 2
        total["bytes"] += (c["stations"] * c["blocks"] * _fft(c) * _bits(c) // 8 +
                           8 * pairs * c["subbands"] * c["nchan"] // c["avg"])
        total["flops"] += int(samples * (5 * math.log2(_fft(c)) + 9) +
                              4 * inputs * (inputs + 1) * c["nchan"] * c["subbands"] * c["blocks"])
    return total


# ------------------------------------------------------------- in 64 bits

def exact(case, seed):
    if case["kind"] == "mux":
        return None
    if case["kind"] == "batch":
        return [_exact_job(c, seed * 100 + i) for i, c in enumerate(_jobs(case))]
    return _exact_job(case, seed)


def _levels(nbits):
    if nbits == 1:
        v = [-1.0, 1.0]
    elif nbits == 2:
        v = [-3.3359, -1.0, 1.0, 3.3359]
    else:
        v = [(b - 128) / 3.3 for b in range(256)]
    return torch.tensor(np.array(v, np.float32).astype(np.float64), device="cuda")


def _exact_job(c, seed):
    """The FX correlation of the same frames: per FFT block the nearest sample to the delay at the block's centre,
    fringe rotation by the delay's line over the block, the transform, the fractional-sample slope and the sums over blocks."""
    dev = "cuda"
    F, N, nb, npol, nst, nblk, cplx = (_fft(c), c["nchan"], c["pols"] * c["subbands"], c["pols"], c["stations"],
                                       c["blocks"], c["cplx"])
    fsamp = PAYLOAD * 8 // _bits(c)
    sub = 2 if cplx else 1
    dt = 1.0 / (c["bw"] * (1.0 if cplx else 2.0))       # us
    ip, lev, nbits = _interp(c, seed), _levels(c["nbits"]), c["nbits"]
    blk = np.arange(nblk, dtype=np.float64)
    streams = _streams(c, seed)
    band_w = torch.zeros(nst, nb, nblk, dtype=torch.float64, device=dev)
    stat_w = torch.zeros(nst, nblk, dtype=torch.float64, device=dev)
    geo = []
    tones = []
    for s, (buf, h, sec, ns) in enumerate(streams):
        q = ip[s]
        quad = lambda x: q[0] * x * x + q[1] * x + q[2]
        start = (START_SEC - sec) * 1e6 + (0 - ns) / 1000.0 + blk * F * dt - quad(blk + 0.5)
        near = (start / dt + 0.5).astype(np.int64)
        err = start - near * dt
        d0, d1, d2 = quad(blk), quad(blk + 0.5), quad(blk + 1)
        a = d2 - d0
        b = d0 + (d1 - (a * 0.5 + d0)) / 3.0
        b -= np.trunc(b)
        valid = (h[:, 0] >> 31) == 0
        fr0 = near // fsamp
        nfr = (near + F - 1) // fsamp - fr0 + 1
        ok = np.zeros((nblk, int(nfr.max())), bool)      # frames of each block
        have = np.zeros((nblk, int(nfr.max()), nb))      # per band, with the threads' masks
        size = np.zeros(ok.shape)
        for k in range(ok.shape[1]):
            f = np.minimum(fr0 + k, len(h) - 1)
            inside = k < nfr
            # complex data: the first frame of a block is judged by its contents alone
            ok[:, k] = inside & (valid[f] | (cplx and k == 0))
            size[:, k] = np.where(inside, np.minimum(near + F, (f + 1) * fsamp) - np.maximum(near, f * fsamp), 0)
            m = h[f, 6] if c["muxed"] else np.full(nblk, (1 << nb) - 1)
            skip = (h[f, 0] >> 31) != 0
            for bd in range(nb):
                have[:, k, bd] = ok[:, k] & ((((m >> bd) & 1) == 1) | skip)
        good = (ok * size).sum(1)
        kept = (have * size[:, :, None]).sum(1)          # [block][band]
        sw = (good - (good[:, None] - kept).sum(1) / nb) / F if c["muxed"] else good / F
        sw = np.maximum(sw, 0.0)
        stat_w[s] = torch.from_numpy(sw)
        band_w[s] = torch.from_numpy((kept / F if c["muxed"] else np.repeat(sw[:, None], nb, 1)).T.copy())
        geo.append((torch.from_numpy(near).to(dev), torch.from_numpy(err).to(dev), torch.from_numpy(a).to(dev),
                    torch.from_numpy(b).to(dev), torch.from_numpy(have * (sw > 0)[:, None, None]).to(dev),
                    torch.from_numpy(fr0).to(dev)))
    n = torch.arange(F, device=dev)
    ch = torch.arange(N, device=dev, dtype=torch.float64)

    def samples(s, bd, k0, k1):
        """Decoded samples [block][F] of one band; invalid ones are zero."""
        near, _, _, _, have, fr0 = geo[s]
        pay = streams[s][0][:, HEADER:].reshape(-1)
        at = near[k0:k1, None] + n
        bit = at * _bits(c) + bd * sub * nbits
        m = torch.gather(have[k0:k1, :, bd], 1, (at // fsamp - fr0[k0:k1, None]))
        code = lambda o: lev[((pay[(bit + o) >> 3].to(torch.int32) >> ((bit + o) & 7).to(torch.int32)) & ((1 << nbits) - 1)).long()]
        return (torch.complex(code(0), code(nbits)) if cplx else code(0)) * m

    def spectra(s, bd, k0, k1):
        _, err, a, b, _, _ = geo[s]
        lo = _lo(c, bd // npol) * (-1.0 if cplx and c["lower"] else 1.0)
        turns = lo * (a[k0:k1, None] * (n / F) + b[k0:k1, None])
        turns = turns - torch.round(turns)
        x = torch.fft.fft(samples(s, bd, k0, k1) * torch.polar(torch.ones_like(turns), -2 * math.pi * turns))
        if not cplx:
            x = x[:, N:] if c["lower"] else x[:, :N]
        elif c["lower"]:
            x = torch.conj(torch.roll(torch.flip(x, [1]), 1, 1)).resolve_conj()
        f = 2 * math.pi * c["bw"] / N * (ch - (N if c["lower"] else 0))
        arg = err[k0:k1, None] * f
        return x * torch.polar(torch.ones_like(arg), arg)

    prods, ni, avg = _products(c), nst * npol, c["avg"]
    i1, i2 = np.triu_indices(nst, 1)
    cross, auto = [], [[None] * (nb * (2 if npol == 2 else 1)) for _ in range(nst)]
    for f in range(c["subbands"]):
        vis = torch.zeros(N, ni, ni, dtype=torch.complex128, device=dev)
        step = max(1, min(nblk, int(2.0e8 / (ni * max(N, 1)))))
        for k0 in range(0, nblk, step):
            k1 = min(nblk, k0 + step)
            X = torch.empty(N, ni, k1 - k0, dtype=torch.complex128, device=dev)
            for s in range(nst):
                for p in range(npol):
                    X[:, s * npol + p] = spectra(s, f * npol + p, k0, k1).t()
            vis += torch.bmm(X, X.conj().transpose(1, 2))
            del X
        mean = lambda v: v.reshape(v.shape[0], N // avg, avg).mean(2) if avg > 1 else v
        rows = torch.tensor(np.stack([i1 * npol + p for p, _ in prods], 1).reshape(-1), device=dev)
        cols = torch.tensor(np.stack([i2 * npol + p for _, p in prods], 1).reshape(-1), device=dev)
        cross.append(torch.cat([mean(vis[:, r, q].t()).reshape(-1)
                                for r, q in zip(rows.split(512), cols.split(512))]) if len(rows) else vis.new_zeros(0))
        for s in range(nst):
            for p in range(npol):
                auto[s][f * npol + p] = mean(vis[:, s * npol + p, s * npol + p][None])[0]
                if npol == 2:
                    auto[s][nb + f * npol + p] = mean(vis[:, s * npol + p, s * npol + 1 - p][None])[0]
        del vis

    def as_pairs(v):
        v = torch.cat([v, v.new_zeros(len(v) % 2)])
        return torch.complex(v[0::2], v[1::2])

    weights, auto_w = [], []
    for f in range(c["subbands"]):
        for a, b in zip(i1, i2):
            weights.append(as_pairs(torch.stack([(band_w[a, f * npol + p] * band_w[b, f * npol + q]).sum() for p, q in prods])
                                    if c["muxed"] else (stat_w[a] * stat_w[b]).sum().repeat(len(prods))))
    for s in range(nst):
        w = [band_w[s, b].sum() for b in range(nb)]
        if npol == 2:
            w += [(band_w[s, b] * band_w[s, b ^ 1]).sum() if c["muxed"] else stat_w[s].sum() for b in range(nb)]
        auto_w.append(as_pairs(torch.stack(w)))
    out = {"cross": torch.cat(cross), "weights": torch.cat(weights),
           "auto": torch.cat([torch.cat(x) for x in auto]), "auto_weights": torch.cat(auto_w)}
    if c["pcal"]:
        fs, mhz = _rate(c), 10 ** 6
        bins = fs // mhz
        for s, (buf, h, sec, ns) in enumerate(streams):
            s0 = int((sec * 1e9 + ns) / (dt * 1e3) + 0.5)
            for bd in range(nb):
                acc = torch.zeros(bins, dtype=torch.complex128, device=dev)
                for k0 in range(0, nblk, 256):
                    k1 = min(nblk, k0 + 256)
                    x = samples(s, bd, k0, k1).to(torch.complex128).reshape(-1)
                    at = ((geo[s][0][k0:k1, None] + n + s0) % bins).reshape(-1)
                    acc.index_add_(0, at, x)
                t = torch.fft.fft(acc)
                k = torch.arange(1, c["bw"] + 1, device=dev)
                tones.append(torch.where(k < bins, t[k % bins], torch.zeros_like(t[0])))
        out["tones"] = torch.cat(tones)
    return out
