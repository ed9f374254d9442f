"""The paired-band F-step (csrc/gx_fstep_pair.cuh) against the oracle at the
sizes and layouts where it takes another branch: every transform length, real
and complex, bands paired within and across frequencies, odd band counts, time
samples narrower than a byte or of three bytes, buffers at odd words, blocks that are not processed, block counts off the group size.

Tolerances as the parity tests': records within 1e-5 by the per-record metric
(FP32 transforms of up to 8192 points are within 2e-7 of their FP64 values),
weights within 1e-6."""
import numpy as np
import pytest

from difx_b200 import capi
from difx_b200.jobfiles import JobSpec, Subband
from tests import jobs
from tests.test_gpu_parity import REC_TOL, W_TOL, _compare, _params

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gx():
    from difx_b200 import gxcorr
    return gxcorr


def _spec(nbits, cplx, pols, nsub, nchan, blocks, sideband="U", nst=2, bw=16.0):
    f0 = 6000.0 + (bw if sideband == "L" else 0.0)
    block_ns = int(1000 * nchan / bw)
    return JobSpec(name=f"pair{nbits}{int(cplx)}{len(pols)}{nsub}_{nchan}_{blocks}{sideband}", nstations=nst,
                   subbands=[Subband(f0 + bw * i, bw, sideband, nchan) for i in range(nsub)], pols=pols, nbits=nbits,
                   sampling="COMPLEX" if cplx else "REAL", subint_ns=blocks * block_ns, execute_seconds=2,
                   payload_bytes=4800 if nsub == 3 else 8000, max_delay_us=150.0, seed=nchan + nbits)


def _check(gx, oracle_lib, spec, sd, prep):
    c = gx.Correlator.from_desc(prep.jd)
    g = c.subint(sd)
    c.close()
    o = oracle_lib.subint(prep.jd, sd, _params(oracle_lib, spec))
    m, wrel = _compare(g, o, prep.jd, spec, oracle_lib)
    assert m < REC_TOL and wrel < W_TOL, (m, wrel)
    return g


# (bits, complex, pols, subbands, channels, blocks, sideband)
LENGTHS = [(8, c, ("R", "L"), 2, n, b, s)
           for c, lens in ((False, (64, 128, 256, 512, 1024, 2048, 4096)), (True, (128, 256, 512, 1024, 2048, 4096, 8192)))
           for n, b, s in ((n, max(5, 70 - 7 * i), "UL"[i % 2]) for i, n in enumerate(lens))]
LAYOUTS = [(2, False, ("R",), 4, 64, 67, "L"),      # two frequencies to a pair
           (8, True, ("R",), 2, 128, 33, "U"),      # and complex, rotator stride of the threads
           (8, True, ("R",), 4, 4096, 5, "L"),
           (8, False, ("R",), 1, 512, 17, "U"),     # one band
           (8, False, ("R",), 3, 256, 19, "L"),     # three bands, three-byte time samples
           (8, True, ("R",), 3, 512, 9, "U"),
           (2, False, ("R",), 2, 128, 37, "U"),     # four bits to a time sample
           (1, False, ("R",), 2, 64, 41, "U"),      # two bits
           (1, False, ("R", "L"), 4, 4096, 3, "U"),
           (4, True, ("R", "L"), 1, 256, 21, "L"),
           (4, False, ("R", "L"), 4, 1024, 6, "U")]


@pytest.mark.parametrize("case", LENGTHS + LAYOUTS, ids=lambda c: "b%d%s%dx%d_%d_%d%s" % (
    c[0], "c" if c[1] else "r", len(c[2]), c[3], c[4], c[5], c[6]))
def test_lengths_and_layouts(case, gx, oracle_lib):
    spec = _spec(*case)
    # some blocks are not processed, a whole group of them at the start
    bad = [np.r_[np.arange(min(32, spec.blocks_per_send // 3)), spec.blocks_per_send - 1], np.array([1])]
    prep = jobs.prepare(spec, [100_000_000], invalid_frac=0.05, bad_blocks=bad, interp_source="host")
    _check(gx, oracle_lib, spec, prep.sds[0], prep)


@pytest.mark.parametrize("nbits,cplx,nchan", [(2, False, 256), (8, True, 1024), (8, False, 4096)])
def test_buffers_at_word_offsets(nbits, cplx, nchan, gx):
    """Station buffers that start at any 4-byte word (frame headers are read as
    words) give the result of ones on a large boundary."""
    import torch
    spec = _spec(nbits, cplx, ("R", "L"), 4 if nbits == 2 else 1, nchan, 12)
    prep = jobs.prepare(spec, [100_000_000], invalid_frac=0.05, interp_source="host")
    si = prep.subs[0]
    c = gx.Correlator.from_desc(prep.jd)
    got = []
    for off in (0, 4, 12):
        bufs = [torch.zeros(len(d) + 16, dtype=torch.uint8, device="cuda") for d in si.data]
        for b, d in zip(bufs, si.data):
            b[off:off + len(d)] = torch.from_numpy(np.array(d)).cuda()
        torch.cuda.synchronize()
        sd = capi.SubintDesc(si.scan, si.sec, si.ns, 0.0, [b.data_ptr() + off for b in bufs], [len(d) for d in si.data],
                             [x.ctypes.data for x in si.control], len(si.control[0]), prep.interps[0])
        out = torch.zeros(2 * c.result_length, dtype=torch.float32, device="cuda")
        c.subint_device(sd, out.data_ptr())
        c.synchronize()
        got.append(out.cpu().numpy())
    c.close()
    np.testing.assert_array_equal(got[1], got[0])
    np.testing.assert_array_equal(got[2], got[0])
