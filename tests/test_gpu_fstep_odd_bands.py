"""F-step of stations with an odd number of bands (csrc/gx_fstep_pair.cuh: one
band, two FFT blocks at a time) against the oracle: every transform length, real
and complex, each sample width down to one bit, both sidebands, odd and even
block counts, blocks of a pair that are not processed, one block alone, frames
shorter than the threads' spacing, bands blanked by a validity mask, post-F
fringe rotation; and the block spectra and the phase-cal sums of the same path.

Tolerances as the parity tests'.  Phase-cal tones formed in the F-step against
the separate kernels': both add n samples of a bin in FP32, in another order; a
sum's rounding errors of 2^-24 of a partial sum add up at random to at most
sqrt(n) 2^-24 of it, taken four times."""
import numpy as np
import pytest

from difx_b200 import capi
from difx_b200.jobfiles import JobSpec, Subband
from tests import jobs
from tests.test_gpu_parity import REC_TOL, W_TOL, _compare, _params

pytestmark = pytest.mark.gpu


def _spec(nbits, cplx, nsub, nchan, blocks, sideband="U", nst=2, bw=16.0, pols=("R",), **kw):
    f0 = 6000.0 + (bw if sideband == "L" else 0.0)
    base = dict(name=f"odd{nbits}{int(cplx)}{nsub}{len(pols)}_{nchan}_{blocks}{sideband}", nstations=nst, pols=pols,
                subbands=[Subband(f0 + bw * i, bw, sideband, nchan) for i in range(nsub)], nbits=nbits,
                sampling="COMPLEX" if cplx else "REAL", subint_ns=blocks * int(1000 * nchan / bw), execute_seconds=2,
                payload_bytes=4800 if nsub == 3 else 8000, max_delay_us=150.0, seed=nchan + nbits)
    base.update(kw)
    return JobSpec(**base)


CASES = ([(8, False, 1, n, b, s) for n, b, s in ((64, 67, "U"), (128, 41, "L"), (256, 38, "U"), (512, 25, "L"), (1024, 12, "U"),
                                                (2048, 7, "L"), (4096, 4, "U"))] +
         [(8, True, 1, n, b, s) for n, b, s in ((128, 67, "L"), (256, 40, "U"), (512, 33, "L"), (1024, 17, "U"), (2048, 10, "L"),
                                               (4096, 5, "U"), (8192, 3, "L"))] +
         [(1, False, 1, 64, 133, "U"), (2, False, 1, 64, 131, "L"), (2, False, 1, 128, 66, "U"), (4, False, 1, 512, 19, "U"),
          (4, True, 1, 256, 21, "L"), (8, False, 3, 64, 35, "U"), (8, True, 3, 2048, 7, "U"), (4, True, 3, 512, 11, "U"),
          (8, False, 1, 1024, 1, "U")])


@pytest.mark.parametrize("case", CASES, ids=lambda c: "b%d%s%d_%d_%d%s" % (c[0], "c" if c[1] else "r", *c[2:]))
def test_odd_band_counts(case, oracle_lib):
    from difx_b200 import gxcorr
    spec = _spec(*case)
    n = spec.blocks_per_send
    # single blocks of a pair, whole pairs and a run of them are not processed
    bad = [np.unique(np.r_[0, 3, np.arange(8, min(20, n // 2)), n - 1]) if n > 3 else np.arange(n - 1),
           np.array([1, 4, 5]) if n > 6 else np.array([], int)]
    prep = jobs.prepare(spec, [100_000_000], invalid_frac=0.05, bad_blocks=bad, interp_source="host")
    c = gxcorr.Correlator.from_desc(prep.jd)
    g = c.subint(prep.sds[0]).copy()
    o = oracle_lib.subint(prep.jd, prep.sds[0], _params(oracle_lib, spec))
    m, wrel = _compare(g, o, prep.jd, spec, oracle_lib)
    assert m < REC_TOL and wrel < W_TOL, (m, wrel)
    p = _params(oracle_lib, spec)
    for blk in {0, n // 2, n - 1}:   # one block alone: a unit without its second block
        gs, gw = c.spectra(1, blk, spec.nbands)
        os_, ow = oracle_lib.station_block(prep.jd, prep.sds[0], 1, blk, p)
        assert np.float32(gw) == np.float32(ow)
        scale = np.sqrt(np.mean(np.abs(os_) ** 2)) if ow > 0 else 1.0
        assert np.max(np.abs(gs - os_)) <= 1e-5 * max(scale, 1e-30) * np.sqrt(spec.fftchannels), blk
    c.close()


@pytest.mark.parametrize("kw", [dict(payload_bytes=400), dict(mux_threads=1, edv4_partial_frac=0.2), dict(fringe_rot_order=0)],
                         ids=["short_frames", "masked", "post_f"])
def test_odd_band_options(kw, oracle_lib):
    from difx_b200 import gxcorr
    # 400-byte payloads: 400 samples a frame, less than the 512 between a thread's samples
    spec = _spec(8, False, 1, 4096 if "payload_bytes" in kw else 512, 9, name="oddopt" + next(iter(kw)), **kw)
    prep = jobs.prepare(spec, [100_000_000], invalid_frac=0.05, interp_source="host")
    c = gxcorr.Correlator.from_desc(prep.jd)
    g = c.subint(prep.sds[0])
    c.close()
    o = oracle_lib.subint(prep.jd, prep.sds[0], _params(oracle_lib, spec))
    m, wrel = _compare(g, o, prep.jd, spec, oracle_lib)
    assert m < REC_TOL and wrel < W_TOL, (m, wrel)


# (bits, complex, subbands, channels, blocks, sideband, MHz, pols, more): the bins of 1 MHz tones divide the threads of a transform
PCAL = [(8, False, 1, 64, 330, "U", 4.0, ("R",), {}), (8, False, 1, 1024, 23, "L", 16.0, ("R",), {}),
        (8, False, 1, 4096, 13, "U", 16.0, ("R",), {}), (8, True, 1, 512, 43, "U", 16.0, ("R",), {}),
        (8, True, 1, 8192, 11, "L", 16.0, ("R",), {}),
        (2, False, 2, 64, 330, "U", 4.0, ("R", "L"), {}), (2, False, 2, 128, 170, "L", 8.0, ("R", "L"), {}),
        (8, False, 1, 256, 90, "U", 16.0, ("R", "L"), {}), (8, True, 1, 256, 170, "L", 16.0, ("R", "L"), {}),
        (8, True, 2, 1024, 43, "U", 16.0, ("R",), {}), (8, False, 2, 1024, 23, "U", 16.0, ("R", "L"), {}),
        (4, False, 2, 2048, 13, "L", 16.0, ("R", "L"), {}), (8, True, 2, 8192, 11, "U", 16.0, ("R", "L"), {}),
        (2, False, 4, 512, 43, "U", 16.0, ("R", "L"), dict(mux_threads=8, edv4_partial_frac=0.1))]


@pytest.mark.parametrize("case", PCAL, ids=lambda c: "b%d%s%dx%d_%d_%d%s%s" % (c[0], "c" if c[1] else "r", len(c[7]), *c[2:6],
                                                                               "m" if c[8] else ""))
def test_phase_cal_in_the_fstep(case):
    from difx_b200 import gxcorr
    nbits, cplx, nsub, nchan, blocks, side, bw, pols, kw = case
    spec = _spec(nbits, cplx, nsub, nchan, blocks, side, bw=bw, pols=pols, pcal_interval_mhz=1, **kw)
    bad = [np.array([0, 3, 6, 7, blocks - 1]), np.array([1])]
    prep = jobs.prepare(spec, [100_000_000], invalid_frac=0.05, bad_blocks=bad, interp_source="host")
    c = gxcorr.Correlator.from_desc(prep.jd)
    fused = c.subint(prep.sds[0]).copy()
    nf = c.launch_count()
    again = c.subint(prep.sds[0]).copy()
    c.set_tiles(0, 1)   # a block per group: more groups than the sums have slots, so the separate kernels run
    apart = c.subint(prep.sds[0]).copy()
    assert c.launch_count() == nf + 1
    off, nt = c.pcal_layout()
    c.close()
    np.testing.assert_array_equal(again, fused)
    tol = 4 * np.sqrt(blocks * spec.fftchannels / (bw * (1 if cplx else 2))) * 2.0 ** -24
    tones = np.zeros(fused.shape, bool)
    for s in range(spec.nstations):
        for b in range(spec.nbands):
            o, n = int(off[s, b]), int(nt[s, b])
            assert o >= 0 and n > 0
            tones[o:o + n] = True
            d = np.linalg.norm(fused[o:o + n].astype(np.complex128) - apart[o:o + n])
            assert 0 < np.linalg.norm(apart[o:o + n]) and d < tol * np.linalg.norm(apart[o:o + n]), (s, b, d)
    np.testing.assert_array_equal(fused[~tones], apart[~tones])
