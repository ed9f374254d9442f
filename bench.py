#!/usr/bin/env python
"""Benchmark: Gsamp/s correlated through the FX hot path, tensor-core X-step
against the FP32 plain X-step.

Workloads (--config):
  c3 (default)  64 stations x 2 pol; 8-bit complex VDIF (sigma = 16 counts,
                rho = 0.01 common component); 4 subbands x 64 MHz; 4096
                channels per subband (4096-point complex FFTs); 1% seeded
                invalid frames; seeded quadratic delay models (|tau| <= 20 ms,
                rates <= 3 us/s); all four polarisation products on all 2016
                baselines plus autocorrelations.  One step = one 128 ms subint
                (2000 FFT blocks per station, 4.19 Gsamples = station x band
                complex time samples, 8.4 GB of VDIF).
  c2            16 stations; 2-bit real VDIF at 2 Gbps/station (2 pol x 8
                subbands x 32 MHz); 256 channels; 1% invalid frames; one step =
                one 200 ms subint (3.28 Gsamples).
Inputs are larger than L2, so no L2 flush is needed between steps.

Arms:
  default            gxcorr with the X-step of --xstep (c3: split-FP16 tensor
                     cores, the form that keeps every visibility within 1e-3 of
                     FP64).  value = device-resident gx_subint_device steps timed
                     with CUDA events; e2e = gx_subint with pinned host buffers
                     (H2D of the raw VDIF and D2H of the result array inside the
                     timed region).  On c3 the FP32 plain and single-FP16 X-steps
                     are timed in the same run ("compare").
  --impl reference   the reference correlator's own CPU path (oracle/_ref, compiled
                     from its sources: Configuration/Mode/Core::processdata) on
                     every host core, on a bounded sample of the same workload.

Multi-GPU (torchrun): each rank correlates its own subints (the reference's
time-division axis); no collective on the data path; value = all ranks'
samples / max-over-ranks time (weak scaling).
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

from difx_b200 import capi, synth  # noqa: E402
from difx_b200.jobfiles import JobSpec, Subband, write_job  # noqa: E402

METRIC = "Gsamp/s correlated"
UNIT = "Gsamp/s"
XSTEPS = {"fp32": capi.GX_XSTEP_FP32, "tc": capi.GX_XSTEP_TC_FP16, "tc_hilo": capi.GX_XSTEP_TC_FP16_HILO}
DEFAULT_SUBINT_MS = {"c3": 128.0, "c3_2bit": 128.0, "c2": 200.0, "c1": 200.0, "c4": 0.0, "c5": 0.0, "mux": 0.0}
DEFAULT_XSTEP = {"c3": "tc_hilo", "c3_2bit": "tc_hilo", "c2": "fp32", "c1": "fp32", "c4": "tc_hilo", "c5": "tc_hilo", "mux": "fp32"}
RHO = {"c3": 0.01, "c3_2bit": 0.01, "c2": 0.02, "c1": 0.05}


def workload_spec(name="c3", subint_ns=None) -> JobSpec:
    if subint_ns is None:
        subint_ns = int(round(DEFAULT_SUBINT_MS[name] * 1e6))
    if name == "c3":
        return JobSpec(name=f"bench_{name}", nstations=64,
                       subbands=[Subband(6000.0 + 64 * i, 64.0, "U", 4096) for i in range(4)],
                       nbits=8, sampling="COMPLEX", payload_bytes=8000, subint_ns=subint_ns, execute_seconds=20,
                       int_time=1.0, max_delay_us=20000.0, max_rate_us_per_s=3.0, seed=2027)
    if name == "c3_2bit":
        # the 2-bit real variant: 8192-point real transforms, 16-bit time samples
        return JobSpec(name=f"bench_{name}", nstations=64,
                       subbands=[Subband(6000.0 + 64 * i, 64.0, "U", 4096) for i in range(4)],
                       nbits=2, payload_bytes=8000, subint_ns=subint_ns, execute_seconds=20,
                       int_time=1.0, max_delay_us=20000.0, max_rate_us_per_s=3.0, seed=2028)
    if name == "c2":
        return JobSpec(name=f"bench_{name}", nstations=16,
                       subbands=[Subband(8200.0 + 32 * i, 32.0, "U", 256) for i in range(8)],
                       nbits=2, payload_bytes=8000, subint_ns=subint_ns, execute_seconds=20, int_time=1.0,
                       max_delay_us=20000.0, max_rate_us_per_s=3.0, seed=2026)
    if name == "c1":
        return JobSpec(name=f"bench_{name}", nstations=4,
                       subbands=[Subband(8400.0 + 16 * i, 16.0, "U", 128) for i in range(4)],
                       nbits=2, payload_bytes=8000, subint_ns=subint_ns, execute_seconds=20, int_time=0.5,
                       max_delay_us=20000.0, max_rate_us_per_s=3.0, seed=2025)
    raise ValueError(name)


def with_nchan(spec: JobSpec, nchan: int) -> JobSpec:
    """The workload with nchan channels per subband and a subint of the same
    number of FFT blocks (the same per-block work of the X-step, less memory)."""
    blocks = spec.blocks_per_send
    sub = [Subband(s.freq_mhz, s.bw_mhz, s.sideband, nchan) for s in spec.subbands]
    s2 = JobSpec(**{**spec.__dict__, "subbands": sub})
    return JobSpec(**{**s2.__dict__, "subint_ns": int(round(blocks * s2.fftchannels / s2.samples_per_second * 1e9))})


def samples_per_subint(spec: JobSpec) -> float:
    return spec.nstations * spec.nbands * spec.samples_per_second * spec.subint_ns * 1e-9


def build_input(spec: JobSpec, sub_start_ns: int, rho=0.02, invalid_frac=0.01, tile_ms=2.0):
    """Station buffers for one subint: a correlated segment repeated over the window."""
    tile_frames = max(1, int(tile_ms * 1e-3 * spec.frames_per_second))
    streams = []
    for s in range(spec.nstations):
        f0, nf = synth.subint_window(spec, s, sub_start_ns)
        streams.append(synth.make_station_stream_tiled(spec, s, f0, nf, tile_frames, rho=rho, seed=spec.seed,
                                                       invalid_frac=invalid_frac))
    return synth.build_subint(spec, streams, sub_start_ns)


class ClockSampler:
    """nvidia-smi clocks and throttle reasons during the timed region.

    Started before the warm-up (so that nvidia-smi's start-up does not fall in
    the timed region); mark() brackets the timed region and summary() keeps
    the samples taken inside it (at least the first three from its start)."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.lines = []      # (monotonic time, csv line)
        self.window = [None, None]

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "100"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
            t0 = time.monotonic()
            while not self.lines and time.monotonic() - t0 < 10.0:
                time.sleep(0.05)
        except Exception:
            self.proc = None
        return self

    def mark(self, which: int):
        self.window[which] = time.monotonic()

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append((time.monotonic(), line.strip()))

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        sm, smax, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        t0, t1 = self.window
        lines = self.lines
        if t0 is not None and lines:
            t1 = t0 if t1 is None else t1
            inside = [x for x in lines if t0 <= x[0] <= t1 + 0.1]
            mid = 0.5 * (t0 + t1)
            lines = inside if len(inside) >= 3 else sorted(lines, key=lambda x: abs(x[0] - mid))[:3]
        for _, l in lines:
            p = [x.strip() for x in l.split(",")]
            if len(p) < 9:
                continue
            try:
                sm.append(float(p[1]))
                smax = float(p[2])
            except ValueError:
                continue
            for n, v in zip(names, p[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": smax, "reasons": sorted(reasons),
                "samples": len(sm)}


# subint of the bounded CPU sample per workload (whole FFT blocks)
REF_SAMPLE_NS = {"c3": 2_048_000, "c3_2bit": 2_048_000, "c2": 4_000_000, "c1": 8_000_000}


class ReferenceSampler:
    """The reference's own CPU path (Core::processdata on every host core)
    opened once over a bounded sample of the workload: one Configuration /
    Core / Modes and one synthetic input, reused for every timed sample and
    freed by close()."""

    def __init__(self, spec_name: str):
        from oracle import pyoracle
        self.err = None
        self.ref = None
        if not pyoracle.reference_available():
            self.err = "reference harness not built (oracle/_ref/libdifxref.so)"
            return
        ncores = os.cpu_count() or 1
        self.spec = workload_spec(spec_name, subint_ns=REF_SAMPLE_NS[spec_name])
        d = tempfile.mkdtemp(prefix="gxref_")
        paths = write_job(self.spec, d)
        with open(paths["threads"], "w") as f:
            f.write(f"{'NUMBER OF CORES:':<20}1\n{ncores}\n")
        self.ref = pyoracle.Reference(paths["input"])
        self.si = build_input(self.spec, 100_000_000, rho=RHO[spec_name], tile_ms=2.0)
        self.ref.process(self.si)  # warm-up: first touch of the Core's result slots and thread arrays

    def rate(self, target_s: float = 15.0, max_subints: int = 50):
        t0 = time.perf_counter()
        n = 0
        while True:
            self.ref.process(self.si)
            n += 1
            el = time.perf_counter() - t0
            if el >= target_s or n >= max_subints:
                break
        rate = n * samples_per_subint(self.spec) / el / 1e9
        sample = (f"{n} subints of {self.spec.subint_ns / 1e6:g} ms ({self.spec.blocks_per_send} FFT blocks) of the "
                  f"same workload, {self.ref.nthreads} process threads, {el:.1f} s")
        return {"value": rate, "unit": UNIT, "cores": int(self.ref.nthreads), "kind": "reference", "sample": sample}

    def close(self):
        if self.ref is not None:
            self.ref.close()
            self.ref = None


def reference_rate(spec_name: str, target_s: float = 15.0, max_subints: int = 50):
    """One bounded timed sample of the reference's CPU path (the cpu_baseline leg)."""
    rs = ReferenceSampler(spec_name)
    if rs.ref is None:
        return None, rs.err
    try:
        return rs.rate(target_s, max_subints), None
    finally:
        rs.close()


def peak_rss_gb() -> float:
    import resource
    return resource.getrusage(resource.RUSAGE_SELF).ru_maxrss / 1e6


def run_reference_arm(args):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return 0
    rs = ReferenceSampler(args.config)
    if rs.ref is None:
        print(json.dumps({"impl": "reference", "unavailable": rs.err}))
        return 0
    steps = []
    base = None
    try:
        for _ in range(max(1, args.steps)):
            base = rs.rate(target_s=max(3.0, 15.0 / max(1, args.steps)))
            steps.append(base["value"])
    finally:
        rs.close()
    v = statistics.median(steps)
    base["value"] = v
    base["peak_rss_gb"] = round(peak_rss_gb(), 2)
    spec = workload_spec(args.config, subint_ns=int(round(args.subint_ms * 1e6)))
    if args.nchan:
        spec = with_nchan(spec, args.nchan)
    if args.pcal_mhz:
        spec = JobSpec(**{**spec.__dict__, "pcal_interval_mhz": args.pcal_mhz})
    line = {"metric": METRIC, "value": v, "unit": UNIT, "n_gpus": args.gpus, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": samples_per_subint(spec) / (v * 1e9) * 1e3,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic (seeded correlated VDIF)", "impl": "reference",
            "config": config_dict(spec, args), "cpu_baseline": base,
            "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line))
    return 0


def config_dict(spec: JobSpec, args):
    kind = f"{spec.nbits}-bit {'complex' if spec.is_complex else 'real'} VDIF"
    return {"workload": f"{args.config.upper()}: {spec.nstations} stations, {kind}, "
                        f"{len(spec.subbands)} subbands x {len(spec.pols)} pol x {spec.bw_mhz:g} MHz, "
                        f"{spec.nchan} ch/subband, 1% invalid frames, {spec.subint_ns / 1e6:g} ms subints",
            "stations": spec.nstations, "bands_per_station": spec.nbands, "nchan": spec.nchan,
            "fft_points": spec.fftchannels, "subint_ms": spec.subint_ns / 1e6,
            "samples_per_step": samples_per_subint(spec), "xstep": args.xstep,
            "l2": "inputs larger than L2 (no flush)", "parallelism": f"subint-parallel x{args.gpus}",
            "phase_cal_mhz": spec.pcal_interval_mhz}


def load_peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return json.load(f)
    except Exception:
        return {}


def x_flops(spec: JobSpec) -> float:
    """Hermitian-unique X-step flops of one subint: 8 x NI (NI + 1) / 2 x nchan x blocks per subband."""
    ni = spec.nstations * len(spec.pols)
    return 8.0 * ni * (ni + 1) / 2 * spec.nchan * spec.blocks_per_send * len(spec.subbands)


def time_device(corr, sd_dev, dres, stream, steps, warmup, local, dist=None, clocks=False):
    """Device-resident steps on one stream: (ms for all steps, stage ms of the last step, launches, clocks)."""
    import torch
    sptr = stream.cuda_stream
    clk = ClockSampler(local) if clocks else None
    if clk:
        clk.__enter__()
    for _ in range(warmup):
        corr.subint_device(sd_dev, dres.data_ptr(), sptr)
    corr.synchronize()
    stream.synchronize()
    if dist:
        dist.barrier()
    torch.cuda.synchronize()
    launches = 0
    ev0 = torch.cuda.Event(enable_timing=True)
    ev1 = torch.cuda.Event(enable_timing=True)
    if clk:
        clk.mark(0)
    ev0.record(stream)
    for _ in range(steps):
        corr.subint_device(sd_dev, dres.data_ptr(), sptr)
        launches += corr.launch_count()
    ev1.record(stream)
    ev1.synchronize()
    if clk:
        clk.mark(1)
        clk.__exit__()
    corr.synchronize()
    dev_ms = ev0.elapsed_time(ev1)
    stage = corr.stage_times()
    torch.cuda.synchronize()
    return dev_ms, stage, launches, (clk.summary() if clk else None)


# DRAM bytes (dram__bytes_read.sum + dram__bytes_write.sum) that ncu measured
# for one launch of the F-step kernel, per FFT block of the launch, by
# (workload, kernel): C3 captured at a 16 ms subint (250 blocks x 64
# stations).  Traffic grows with the blocks a launch processes, so a step's
# traffic is this figure times its blocks.
F_DRAM_BYTES_PER_BLOCK = {("bench_c3", "fstep_pair_kernel"): (1.066021e9 + 4.136721e9) / 250}


def f_kernel_name(spec: JobSpec) -> str:
    """The F-step kernel the library runs for this job."""
    return "fstep_pair_kernel" if 128 <= spec.fftchannels <= 8192 else "fstep_cta_kernel"


def roofline(spec: JobSpec, xstep: str, stage, peaks):
    f_ms, x_ms, fin_ms = float(stage[0]), float(stage[1]), float(stage[2])
    hbm_peak = peaks.get("hbm_gbs", 6650.0)
    src = "of measured" if "hbm_gbs" in peaks else "of fallback"
    nblk = spec.blocks_per_send
    in_bytes = nblk * spec.nstations * spec.fftchannels * (spec.bits_per_timesample // 8)
    spec_bytes = nblk * spec.nstations * spec.nbands * spec.nchan * 8
    stages = {"F": f_ms, "X": x_ms, "finalise": fin_ms}
    if f_ms >= x_ms:
        k = f_kernel_name(spec)
        a = (in_bytes + spec_bytes) / (f_ms * 1e-3) / 1e9
        traffic, tsrc = None, None
        if (spec.name, k) in F_DRAM_BYTES_PER_BLOCK:
            traffic = F_DRAM_BYTES_PER_BLOCK[(spec.name, k)] * nblk
            tsrc = "ncu DRAM bytes of one 250-block launch (16 ms subint), scaled to the step's blocks"
        return {"kernel": k, "bound": "hbm", "achieved": a, "peak": hbm_peak, "unit": "GB/s", "frac": a / hbm_peak,
                "traffic": traffic, "traffic_source": tsrc, "peak_source": src,
                "algorithmic_bytes_per_step": in_bytes + spec_bytes, "stage_ms": stages}
    if xstep == "fp32":
        a = x_flops(spec) / (x_ms * 1e-3) / 1e12
        p = 148 * 128 * 2 * (peaks.get("sm_max_mhz", 1965.0) * 1e6) / 1e12
        return {"kernel": "xmac_fp32_kernel", "bound": "fp32-core", "achieved": a, "peak": p, "unit": "TFLOP/s",
                "frac": a / p, "traffic": None,
                "peak_source": "nominal FP32 CUDA-core peak (148 SM x 128 FMA/clk x max SM clock)",
                "stage_ms": stages}
    # tensor-core X-step: HBM-bound on the FP32 spectra it reads; tensor pipe reported beside
    a = spec_bytes / (x_ms * 1e-3) / 1e9
    nprod = 9 if xstep == "tc_hilo" else 3          # 128x128 real products per channel and block
    tflops = nprod * 2 * 128 * 128 * spec.nchan * nblk * len(spec.subbands) / (x_ms * 1e-3) / 1e12
    tpk = peaks.get("bf16_tflops", 1590.0)
    return {"kernel": "xmac_tc_kernel", "bound": "hbm", "achieved": a, "peak": hbm_peak, "unit": "GB/s",
            "frac": a / hbm_peak, "traffic": None, "peak_source": src, "algorithmic_bytes_per_step": spec_bytes,
            "tensor": {"executed_tflops": tflops, "peak": tpk, "frac": tflops / tpk,
                       "useful_tflops": x_flops(spec) / (x_ms * 1e-3) / 1e12,
                       "peak_source": "measured dense bf16 (FP16 runs at the same rate)"},
            "stage_ms": stages}


def c5_jobs(njobs=12, seed=2030):
    """Serving workload: real-time jobs of 4-48 stations, 2-bit real VDIF at
    1, 2 or 4 Gbps per station (8 x 32 MHz, 16 x 32 MHz or 16 x 64 MHz bands),
    256-2048 channels, subints of 0.2-1 s (whole FFT blocks)."""
    rng = np.random.default_rng(seed)
    out = []
    for j in range(njobs):
        nst = int(rng.integers(4, 49))
        gbps = int(rng.choice([1, 2, 4]))
        nsub, bw = {1: (4, 32.0), 2: (8, 32.0), 4: (8, 64.0)}[gbps]
        nchan = int(rng.choice([256, 512, 1024, 2048]))
        block_ns = int(round(nchan / bw * 1000))
        subint_ns = int(round(rng.uniform(0.2, 1.0) * 1e9 / block_ns)) * block_ns
        out.append(JobSpec(name=f"c5_{j}", nstations=nst, subbands=[Subband(8000.0 + bw * i, bw, "U", nchan)
                                                                   for i in range(nsub)],
                           nbits=2, payload_bytes=8000, subint_ns=subint_ns, execute_seconds=20, int_time=1.0,
                           max_delay_us=100.0, max_rate_us_per_s=3.0, seed=3000 + j))
    return out


def c4_jobs(njobs=200, seed=4040):
    """Uneven batch: 200 jobs of U{3..32} stations, 64/256/1024/4096 channels,
    1-, 2- or 8-bit samples (8-bit real or complex), 1-16 recorded bands
    (subbands x polarisations, a power of two as VDIF requires, and enough of
    them that a time sample fills whole bytes) at 8-64 MHz,
    0.1-1 s subints (whole FFT blocks), correlation coefficient 0.005-0.1."""
    rng = np.random.default_rng(seed)
    out = []
    for j in range(njobs):
        nst = int(rng.integers(3, 33))
        nchan = int(rng.choice([64, 256, 1024, 4096]))
        nbits = int(rng.choice([1, 2, 8]))
        # a time sample of all bands fills whole bytes: 1-bit >= 8 bands, 2-bit >= 4
        nbands = int(rng.choice([b for b in (1, 2, 4, 8, 16) if b * nbits >= 8]))
        bw = float(rng.choice([8.0, 16.0, 32.0, 64.0]))
        cplx = nbits == 8 and rng.random() < 0.5
        pols = ("R", "L") if nbands > 1 and rng.random() < 0.5 else ("R",)
        nsub = nbands // len(pols)
        sub = float(rng.uniform(0.1, 1.0))
        rho = float(rng.uniform(0.005, 0.1))
        block_ns = nchan / bw * 1000   # N channels from N complex or 2N real samples
        subint_ns = max(1, int(round(sub * 1e9 / block_ns))) * int(round(block_ns))
        out.append((JobSpec(name=f"c4_{j}", nstations=nst, pols=pols,
                            subbands=[Subband(4000.0 + bw * i, bw, "U", nchan) for i in range(nsub)],
                            nbits=nbits, sampling="COMPLEX" if cplx else "REAL", payload_bytes=8000,
                            subint_ns=subint_ns, execute_seconds=4, int_time=1.0, max_delay_us=100.0,
                            max_rate_us_per_s=3.0, seed=5000 + j), rho))
    return out


def run_c4(args):
    """One subint of each of 200 uneven resident jobs per step (gx_batch):
    per-job launches on one stream against the branch-stream schedule
    replayed as one CUDA graph (branch count tuned on the first steps)."""
    import torch
    from difx_b200.gxcorr import Batch, Correlator
    t_setup = time.perf_counter()
    staged = []
    for spec, rho in c4_jobs():
        d = tempfile.mkdtemp(prefix="gxc4_")
        paths = write_job(spec, d)
        # one synthesised station stream, shared by every station of the job
        one = JobSpec(**{**spec.__dict__, "nstations": 1})
        si = build_input(one, 200_000_000, rho=rho)
        m = Correlator.from_input(paths["input"], device=-1)
        interp = np.array([m.interpolator(s, 0, si.sec, si.ns) for s in range(spec.nstations)])
        m.close()
        dev = torch.from_numpy(si.data[0]).cuda()
        n = spec.nstations
        sd = capi.SubintDesc(si.scan, si.sec, si.ns, 0.0, [dev.data_ptr()] * n, [len(si.data[0])] * n,
                             [si.control[0].ctypes.data] * n, len(si.control[0]), interp)
        staged.append((spec, sd, dev, si))
    torch.cuda.synchronize()
    corrs, res = [], []
    for spec, *_ in staged:
        # spectra buffers sized for efficient passes, at most 2 GB per job
        c = Correlator.from_desc(capi.job_desc_from_spec(spec, xstep=capi.GX_XSTEP_AUTO,
                                                         spectra_budget_bytes=2 << 30))
        corrs.append(c)
        res.append(torch.empty(2 * c.result_length, dtype=torch.float32, device="cuda"))
    subs = [sd for _, sd, _, _ in staged]
    ptrs = [r.data_ptr() for r in res]
    setup_s = time.perf_counter() - t_setup
    samples = sum(samples_per_subint(s) for s, *_ in staged)
    steps = max(1, args.c4_steps)

    def timed(b, nsteps, clk=None):
        dev_ms, wall = [], time.perf_counter()
        if clk:
            clk.mark(0)
        for _ in range(nsteps):
            b.run(subs)
            dev_ms.append(b.synchronize())
        if clk:
            clk.mark(1)
        return float(np.sum(dev_ms)), (time.perf_counter() - wall) * 1e3

    modes = {}
    # per-job launches: one job after another on one stream
    b = Batch(corrs, ptrs, mode="serial")
    timed(b, 1)
    ms, wall = timed(b, steps)
    modes["per_job_launches"] = {"gsamp_s": samples * steps / (ms * 1e-3) / 1e9, "device_ms_per_step": ms / steps,
                                 "wall_ms_per_step": wall / steps, "gpu_launches_per_step": b.info()[2]}
    b.close()
    # launch shapes per shape class (X-step channel tile and stage depth,
    # F-step blocks per CTA), from the default shapes' graph step to the tuned one
    b = Batch(corrs, ptrs, mode="graph", nstreams=16)
    timed(b, 1)
    ms_default, _ = timed(b, steps)
    t_tile = time.perf_counter()
    nclasses = b.tune_tiles(subs, reps=2)
    tile_tune_s = time.perf_counter() - t_tile
    tiles = {}
    for c in corrs:
        t = c.tiles()
        tiles[f"x{t[0]}_f{t[1]}"] = tiles.get(f"x{t[0]}_f{t[1]}", 0) + 1
    b.close()
    # branch streams replayed as one graph; the branch count is tuned on the first steps
    with ClockSampler(0) as clk:
        b = Batch(corrs, ptrs, mode="graph", nstreams=0)
        tune = []
        while b.info()[1]:
            b.run(subs)
            tune.append(b.synchronize())
        k = b.info()[0]
        ms, wall = timed(b, steps, clk)
        launches = b.info()[2]
        b.close()
    clocks = clk.summary()
    modes["graph"] = {"gsamp_s": samples * steps / (ms * 1e-3) / 1e9, "device_ms_per_step": ms / steps,
                      "wall_ms_per_step": wall / steps, "branches": k, "tuning_ms": tune,
                      "gpu_launches_per_step": launches, "host_launches_per_step": 1,
                      "tile_tuner": {"shape_classes": nclasses, "tuning_s": tile_tune_s, "chosen": tiles,
                                     "default_tiles_device_ms_per_step_16_branches": ms_default / steps}}
    # the same schedule issued stream by stream (no graph)
    b = Batch(corrs, ptrs, mode="streams", nstreams=k)
    timed(b, 1)
    ms_s, wall_s = timed(b, steps)
    modes["streams"] = {"gsamp_s": samples * steps / (ms_s * 1e-3) / 1e9, "device_ms_per_step": ms_s / steps,
                        "wall_ms_per_step": wall_s / steps, "branches": k}
    b.close()
    forms = {}
    for c in corrs:
        forms[c.info.xstep] = forms.get(c.info.xstep, 0) + 1
        c.close()
    value = modes["graph"]["gsamp_s"]
    line = {"metric": "C4 batch: Gsamp/s correlated over 200 uneven jobs (one subint each per step)", "value": value,
            "unit": "Gsamp/s", "n_gpus": 1, "steps": steps, "warmup": len(tune), "ms_per_step": ms / steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "per job: f32, or f16 hi+lo operands with f32 accumulation (GX_XSTEP_AUTO)",
            "data": "synthetic (seeded VDIF, one stream per job shared by its stations), inputs device-resident",
            "config": {"workload": "C4: 200 jobs, U{3..32} stations, 64/256/1024/4096 ch, 1/2/8-bit, 1-16 bands "
                                   "at 8-64 MHz, 0.1-1 s subints", "samples_per_step": samples,
                       "xstep_forms": {{0: "fp32", 2: "tc_hilo"}.get(f, str(f)): n for f, n in forms.items()},
                       "l2": "inputs larger than L2 (no flush)", "setup_s": setup_s},
            "modes": modes, "graph_vs_per_job_launches": value / modes["per_job_launches"]["gsamp_s"],
            "gpu_launches": launches, "clocks": clocks}
    print(json.dumps(line))
    return 0


def mux_stream(nthreads=16, fps=4000, seconds=1, fb=8032, nbits=2, seed=77):
    """Frame-aligned multi-thread VDIF: nthreads x fps frames per second of
    2-bit samples, thread-interleaved in time order (as a recorder writes them)."""
    rng = np.random.default_rng(seed)
    n = nthreads * fps * seconds
    buf = rng.integers(0, 256, (n, fb), dtype=np.uint8)
    fr = np.arange(n) // nthreads
    hdr = np.zeros((n, 8), np.uint32)
    hdr[:, 0] = (1000 + fr // fps).astype(np.uint32)
    hdr[:, 1] = (fr % fps).astype(np.uint32) | (40 << 24)
    hdr[:, 2] = fb // 8
    hdr[:, 3] = 0x4142 | ((np.arange(n) % nthreads).astype(np.uint32) << 16) | ((nbits - 1) << 26)
    buf[:, :32] = hdr.view(np.uint8).reshape(n, 32)
    return buf.reshape(-1)


def run_mux(args):
    """Device VDIF multiplexing of a 1 s, 16-thread, 2-bit stream (the VDIF
    DataStream's corner turn): input bytes per second of device time."""
    import torch
    from difx_b200.gxcorr import VdifMux
    nthreads, fps, fb, nbits = 16, 4000, 8032, 2
    src = mux_stream(nthreads, fps, 1, fb, nbits)
    m = VdifMux(fb, fps, nbits, list(range(nthreads)), nsort=32, ngap=fps // 4, flags=0x02 | 0x40)
    nout = len(src) // fb // nthreads
    dest_bytes = m.output_frame_bytes * (nout + 1)
    d_src = torch.from_numpy(src).cuda()
    d_dest = torch.empty(dest_bytes, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream()
    for _ in range(args.warmup):
        m.run(d_src.data_ptr(), len(src), d_dest.data_ptr(), dest_bytes, -1, stream.cuda_stream)
    torch.cuda.synchronize()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    t0 = time.perf_counter()
    ev0.record(stream)
    for _ in range(args.steps):
        st = m.run(d_src.data_ptr(), len(src), d_dest.data_ptr(), dest_bytes, -1, stream.cuda_stream)
    ev1.record(stream)
    ev1.synchronize()
    ms = ev0.elapsed_time(ev1) / args.steps
    wall_ms = (time.perf_counter() - t0) * 1e3 / args.steps
    peaks = load_peaks()
    hbm = peaks.get("hbm_gbs", 6650.0)
    moved = len(src) + st.output_frames * m.output_frame_bytes
    line = {"metric": "VDIF multiplex: input GB/s (device classification + corner turn, host decisions)",
            "value": len(src) / (ms * 1e-3) / 1e9, "unit": "GB/s", "n_gpus": 1, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "u8", "data": "synthetic (seeded 2-bit samples, valid headers)",
            "config": {"workload": f"1 s of {nthreads}-thread 2-bit VDIF, {fb}-byte frames, {fps} frames/s per thread",
                       "input_bytes": len(src), "output_frames": st.output_frames,
                       "l2": "inputs larger than L2 (no flush)"},
            "wall_ms_per_step": wall_ms,
            "roofline": {"kernel": "vmux_turn_kernel + vmux_classify_kernel + host decisions", "bound": "hbm",
                         "achieved": moved / (ms * 1e-3) / 1e9, "peak": hbm, "unit": "GB/s",
                         "frac": moved / (ms * 1e-3) / 1e9 / hbm, "traffic": None,
                         "peak_source": "of measured" if "hbm_gbs" in peaks else "of fallback"},
            "gpu_launches": 2 * args.steps}
    if not args.no_cpu_baseline:
        try:
            from oracle import pyoracle
            if pyoracle.vmux_available():
                _, ref = pyoracle.ref_vdifmux(src.tobytes(), dest_bytes, fb, fps, nbits, list(range(nthreads)), 32,
                                              fps // 4, 0x02 | 0x40)
                line["cpu_baseline"] = {"value": len(src) / (ref[22] * 1e-9) / 1e9, "unit": "GB/s", "cores": 1,
                                        "kind": "reference",
                                        "sample": "the reference's vdifmux (single thread, OpenMP off) on the same 1 s stream"}
        except Exception as e:   # the baseline is reported, never required
            line["cpu_baseline"] = {"unavailable": str(e)[:200]}
    print(json.dumps(line))
    return 0


def run_c5(args):
    """Continuous batching of subint requests from 12 resident jobs through
    gx_server (device-resident inputs, HBM budget), Poisson arrivals."""
    import torch
    from difx_b200.gxcorr import Correlator, Server
    specs = c5_jobs()
    rng = np.random.default_rng(7)
    staged = []
    for spec in specs:
        d = tempfile.mkdtemp(prefix="gxc5_")
        paths = write_job(spec, d)
        # one synthesised station stream, shared by every station of the job (throughput
        # does not depend on the sample values; the control words and windows are the same)
        one = JobSpec(**{**spec.__dict__, "nstations": 1})
        si = build_input(one, 200_000_000, rho=0.02)
        m = Correlator.from_input(paths["input"], device=-1)
        interp = np.array([m.interpolator(s, 0, si.sec, si.ns) for s in range(spec.nstations)])
        m.close()
        dev = torch.from_numpy(si.data[0]).cuda()
        staged.append((spec, si, interp, dev))
    torch.cuda.synchronize()
    out = {}
    for form in (args.xstep, "fp32"):
        # about 1 GB of spectra per resident job (128 rows bound the padded inputs of either X-step)
        chunks = [max(64, min(s.blocks_per_send, int(1e9 / (len(s.subbands) * 128 * s.nchan * 8))))
                  for s, *_ in staged]
        corrs = [Correlator.from_desc(capi.job_desc_from_spec(s, xstep=XSTEPS[form], block_chunk=ch))
                 for (s, *_), ch in zip(staged, chunks)]
        budget = min(140 << 30, sum(c.device_bytes() for c in corrs) + (16 << 30))
        srv = Server(slots=args.c5_slots, hbm_budget_bytes=budget, device_inputs=True)
        ids = [srv.attach(c) for c in corrs]
        sds, res = [], []
        for (spec, si, interp, dev), c in zip(staged, corrs):
            n = spec.nstations
            sds.append(capi.SubintDesc(si.scan, si.sec, si.ns, 0.0, [dev.data_ptr()] * n, [len(si.data[0])] * n,
                                       [si.control[0].ctypes.data] * n, len(si.control[0]), interp))
            res.append(torch.empty(2 * c.result_length, dtype=torch.float32).pin_memory())
        # calibration: every job alone (also the warm-up)
        alone = []
        for j in range(len(staged)):
            for _ in range(2):
                t = srv.submit(ids[j], sds[j], res[j].data_ptr(), request_bytes=0)
                ms = srv.wait(t)
            alone.append(ms)
        srv.stats(reset=True)
        samples = [samples_per_subint(s) for s, *_ in staged]
        mean_alone_s = float(np.mean(alone)) / 1e3
        subint_ms = [s.subint_ns / 1e6 for s, *_ in staged]

        def run_load(rate, seconds):
            """Poisson arrivals at `rate` requests/s for `seconds`: throughput and
            latency, also relative to each request's subint duration."""
            n_req = max(20, int(rate * seconds))
            gaps = rng.exponential(1.0 / rate, n_req)
            picks = rng.integers(0, len(staged), n_req)
            srv.stats(reset=True)
            tickets = []
            t0 = time.perf_counter()
            tnext = t0
            for g, j in zip(gaps, picks):
                tnext += g
                dt = tnext - time.perf_counter()
                if dt > 0:
                    time.sleep(dt)
                tickets.append((int(j), srv.submit(ids[j], sds[j], res[j].data_ptr(), request_bytes=0)))
            lat = [(j, srv.wait(t)) for j, t in tickets]
            wall = time.perf_counter() - t0
            st = srv.stats()
            rel = np.array([ms / subint_ms[j] for j, ms in lat])
            return {"offered_load": rate * mean_alone_s, "offered_rate_req_s": rate, "requests": len(lat),
                    "sustained_gsamp_s": sum(samples[j] for j, _ in lat) / wall / 1e9,
                    "latency_ms": {"p50": st.p50_ms, "p95": st.p95_ms, "p99": st.p99_ms, "mean": st.mean_ms,
                                   "max": st.max_ms},
                    "latency_over_subint": {"p50": float(np.percentile(rel, 50)),
                                            "p95": float(np.percentile(rel, 95)),
                                            "p99": float(np.percentile(rel, 99))},
                    "fraction_within_subint": float(np.mean(rel <= 1.0))}

        if args.c5_rate > 0:
            loads = [run_load(args.c5_rate, args.c5_seconds)]
        else:
            # offered load = arrival rate x mean one-at-a-time service time
            loads = [run_load(f / mean_alone_s, args.c5_seconds) for f in (0.2, 0.35, 0.5, 0.7)]
        srv.close()
        for c in corrs:
            c.close()
        ok = [x for x in loads if x["latency_over_subint"]["p99"] < 1.0]
        out[form] = {"alone_ms_mean": float(np.mean(alone)), "loads": loads,
                     # service time alone / subint duration per job: above 1 the job cannot be real time
                     "alone_over_subint": [round(a / m, 3) for a, m in zip(alone, subint_ms)],
                     "max_load_p99_within_subint": max((x["offered_load"] for x in ok), default=None),
                     "at_max_load": max(ok, key=lambda x: x["offered_load"]) if ok else None}
    spec_rate = 50.0
    load50 = spec_rate * out["fp32"]["alone_ms_mean"] / 1e3
    head = out[args.xstep]["at_max_load"] or out[args.xstep]["loads"][0]
    line = {"metric": "C5 serving: sustained Gsamp/s at the highest offered load with p99 latency < subint duration",
            "value": head["sustained_gsamp_s"], "unit": UNIT, "n_gpus": 1, "higher_is_better": True,
            "dtype": args.xstep,
            "data": "synthetic (seeded 2-bit VDIF, one stream per job shared by its stations), inputs device-resident",
            "config": {"workload": "C5: 12 real-time jobs, 4-48 stations, 2-bit real VDIF at 1-4 Gbps/station, "
                                   "256-2048 channels, 0.2-1 s subints; Poisson arrivals; earliest-deadline-first "
                                   "admission (deadline = subint duration)",
                       "jobs": [{"stations": s.nstations, "bands": s.nbands, "bw_mhz": s.bw_mhz, "nchan": s.nchan,
                                 "subint_ms": s.subint_ns / 1e6} for s, *_ in staged],
                       "slots": args.c5_slots, "seconds_per_load": args.c5_seconds,
                       "arrival_rate_note": (f"loads swept as fractions of the measured one-at-a-time capacity; the "
                                             f"specified 50 requests/s at these job sizes would offer "
                                             f"{load50:.1f}x the FP32 form's serial capacity")},
            "forms": out,
            "tc_vs_fp32_at_max_load": (out[args.xstep]["at_max_load"]["sustained_gsamp_s"] /
                                       out["fp32"]["at_max_load"]["sustained_gsamp_s"]
                                       if out[args.xstep]["at_max_load"] and out["fp32"]["at_max_load"] else None)}
    print(json.dumps(line))
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="gxcorr", choices=["gxcorr", "reference"])
    ap.add_argument("--config", default="c3", choices=["c3", "c3_2bit", "c2", "c1", "c4", "c5", "mux"])
    ap.add_argument("--c4-steps", type=int, default=1, help="timed batch steps per mode (C4)")
    ap.add_argument("--c5-slots", type=int, default=4)
    ap.add_argument("--c5-seconds", type=float, default=8.0, help="seconds of arrivals per offered load")
    ap.add_argument("--c5-rate", type=float, default=0.0, help="requests per second (0: 70%% of capacity)")
    ap.add_argument("--xstep", default=None, choices=sorted(XSTEPS))
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-compare", action="store_true", help="skip the other X-step forms")
    ap.add_argument("--pcal-mhz", type=int, default=0,
                    help="PHASE CAL INT (MHZ) of every station (0: none); timing with phase-cal extraction")
    ap.add_argument("--nchan", type=int, default=0,
                    help="channels per subband (0: the workload's); smaller values give small profiling cases")
    ap.add_argument("--subint-ms", type=float, default=None,
                    help="subint length; smaller values give small profiling cases")
    args = ap.parse_args()
    if args.xstep is None:
        args.xstep = DEFAULT_XSTEP[args.config]
    if args.subint_ms is None:
        args.subint_ms = DEFAULT_SUBINT_MS[args.config]
    if args.impl == "reference":
        return run_reference_arm(args)
    if args.config == "c5":
        return run_c5(args)
    if args.config == "c4":
        return run_c4(args)
    if args.config == "mux":
        return run_mux(args)

    import torch
    from difx_b200.gxcorr import Correlator

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120), device_id=torch.device("cuda", local))

    spec = workload_spec(args.config, subint_ns=int(round(args.subint_ms * 1e6)))
    if args.nchan:
        spec = with_nchan(spec, args.nchan)
    if args.pcal_mhz:
        spec = JobSpec(**{**spec.__dict__, "pcal_interval_mhz": args.pcal_mhz})
    d = tempfile.mkdtemp(prefix=f"gxbench{rank}_")
    paths = write_job(spec, d)
    # each rank correlates its own subint of the job
    t_sub = 200_000_000 + rank * spec.subint_ns
    si = build_input(spec, t_sub, rho=RHO[args.config])
    model = Correlator.from_input(paths["input"], device=-1)
    interp = np.array([model.interpolator(s, 0, si.sec, si.ns) for s in range(spec.nstations)])
    model.close()
    maxbytes = max(len(x) for x in si.data)

    # device-resident inputs
    dev = [torch.from_numpy(x).to(f"cuda:{local}") for x in si.data]
    sd_dev = capi.SubintDesc(si.scan, si.sec, si.ns, 0.0, [t.data_ptr() for t in dev], [len(x) for x in si.data],
                             [x.ctypes.data for x in si.control], len(si.control[0]), interp)
    stream = torch.cuda.Stream(device=local)
    peaks = load_peaks()
    samples = samples_per_subint(spec)

    # the other X-step forms first (device-resident timing only), then the headline arm
    compare = {}
    if args.config in ("c3", "c3_2bit") and not args.no_compare:
        for name in sorted(XSTEPS):
            if name == args.xstep:
                continue
            c = Correlator.from_desc(capi.job_desc_from_spec(spec, xstep=XSTEPS[name]), device=local)
            dres = torch.zeros(2 * c.result_length, dtype=torch.float32, device=f"cuda:{local}")
            ms, stage, _, _ = time_device(c, sd_dev, dres, stream, max(2, args.steps // 2), 2, local, dist)
            c.close()
            del dres
            compare[name] = {"value": samples * max(2, args.steps // 2) * world / (ms * 1e-3) / 1e9,
                             "ms_per_step": ms / max(2, args.steps // 2),
                             "stage_ms": {"F": float(stage[0]), "X": float(stage[1]), "finalise": float(stage[2])}}
        torch.cuda.empty_cache()

    jd = capi.job_desc_from_spec(spec, xstep=XSTEPS[args.xstep], max_data_bytes=maxbytes)
    corr = Correlator.from_desc(jd, device=local)
    dres = torch.zeros(2 * corr.result_length, dtype=torch.float32, device=f"cuda:{local}")
    dev_ms, stage, launches, clocks = time_device(corr, sd_dev, dres, stream, args.steps, args.warmup, local, dist,
                                                  clocks=True)
    if dist:
        dist.barrier()
        t = torch.tensor([dev_ms], device=f"cuda:{local}")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        dev_ms = float(t.item())
    total_samples = samples * args.steps * world
    value = total_samples / (dev_ms * 1e-3) / 1e9

    # end to end through the public host-buffer entry point, pinned host memory
    del dev, dres
    torch.cuda.empty_cache()
    pinned = [torch.from_numpy(x).pin_memory() for x in si.data]
    res_host = torch.zeros(2 * corr.result_length, dtype=torch.float32).pin_memory()
    sd_host = capi.SubintDesc(si.scan, si.sec, si.ns, 0.0, [t.data_ptr() for t in pinned],
                              [len(x) for x in si.data], [x.ctypes.data for x in si.control],
                              len(si.control[0]), interp)
    res_host2 = torch.zeros(2 * corr.result_length, dtype=torch.float32).pin_memory()
    outs = [res_host.numpy().view(np.complex64), res_host2.numpy().view(np.complex64)]
    for _ in range(2):
        corr.subint(sd_host, out=outs[0])
    lat = []
    if dist:
        dist.barrier()
    # gx_subint_async keeps two subints in flight: one uploads while the other computes;
    # every step still copies its VDIF in and its result array out
    t0 = time.perf_counter()
    starts = []
    for i in range(args.steps):
        if i >= 2:
            corr.wait()
            lat.append((time.perf_counter() - starts[i - 2]) * 1e3)
        starts.append(time.perf_counter())
        corr.subint_async(sd_host, outs[i % 2])
    for i in range(max(0, args.steps - 2), args.steps):
        corr.wait()
        lat.append((time.perf_counter() - starts[i]) * 1e3)
    e2e_s = time.perf_counter() - t0
    if dist:
        t = torch.tensor([e2e_s], device=f"cuda:{local}")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        e2e_s = float(t.item())
    e2e = total_samples / e2e_s / 1e9

    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": dev_ms / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None,
            "dtype": {"fp32": "f32", "tc": "f16 operands, f32 accumulation",
                      "tc_hilo": "f16 hi+lo operands, f32 accumulation"}[args.xstep],
            "data": "synthetic (seeded correlated VDIF, 2 ms correlated segment repeated; seeded delay models)",
            "config": config_dict(spec, args),
            "e2e": {"value": e2e, "unit": UNIT, "h2d_bytes_per_step": int(sum(len(x) for x in si.data)),
                    "d2h_bytes_per_step": int(corr.result_length * 8),
                    "api": "gx_subint_async / gx_subint_wait, two subints in flight, pinned host buffers"},
            "latency_ms": {"p50": statistics.median(lat), "p99": float(np.percentile(lat, 99)),
                           "subint_ms": spec.subint_ns / 1e6},
            "gpu_launches": int(launches), "roofline": roofline(spec, args.xstep, stage, peaks), "clocks": clocks}
    if compare:
        compare[args.xstep] = {"value": value, "ms_per_step": dev_ms / args.steps,
                               "stage_ms": {"F": float(stage[0]), "X": float(stage[1]), "finalise": float(stage[2])}}
        fp = compare.get("fp32")
        if fp:
            line["tc_vs_fp32"] = {
                k: {"whole_path": compare[k]["value"] / fp["value"],
                    "x_step": fp["stage_ms"]["X"] / compare[k]["stage_ms"]["X"]}
                for k in compare if k != "fp32"}
        line["compare"] = compare
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        base, err = reference_rate(args.config)
        line["cpu_baseline"] = base if base else {"unavailable": err}
    corr.close()
    if dist:
        dist.barrier()
        dist.destroy_process_group()
    if rank == 0:
        print(json.dumps(line))
    return 0


if __name__ == "__main__":
    sys.exit(main())
