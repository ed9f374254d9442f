"""How long a sum of the tensor-core X-step stays in tensor memory.  The MMA
truncates its FP32 accumulator, so a long run loses a part of every sum that
grows with the run; a pass of more than 4096 blocks is cut into slices for that
reason.

Tolerance of the autocorrelations (sums that grow evenly, so that every loss has
one sign): each of the 6 MMAs that a 16-block step of the split form adds into a
real part loses at most one unit of 2^-23 of the sum, which is on average half of
the final one: 6 x 4096 / 16 x 2^-24 = 9.2e-5 for the longest run."""
import numpy as np
import pytest

from difx_b200 import capi, synth
from difx_b200.jobfiles import JobSpec, Subband
from tests import jobs

LONGEST = 4096
BLOCKS = 32768


def _spec():
    # 8 x 128 channels: one K-split slice, whose run is then the whole pass
    return JobSpec(name="tcrun", nstations=2, pols=("R",), subbands=[Subband(6000.0 + 16 * i, 16.0, "U", 128) for i in range(8)],
                   nbits=2, subint_ns=BLOCKS * 8000, execute_seconds=2, max_delay_us=50.0, seed=77)


@pytest.mark.gpu
@pytest.mark.parametrize("chunk", [0, BLOCKS, 10923])   # by the handle, one pass, three
def test_long_subint_autocorrelations(chunk):
    from difx_b200 import gxcorr
    spec = _spec()
    t0 = 100_000_000
    streams = []
    for s in range(spec.nstations):
        f0, nf = synth.subint_window(spec, s, t0)
        streams.append(synth.make_station_stream_tiled(spec, s, f0, nf, 64, rho=0.2, seed=5, invalid_frac=0.01))
    si = synth.build_subint(spec, streams, t0)
    sd = capi.subint_desc_host(si, jobs.interpolators(jobs.write_job(spec, jobs._TMP + "/tcrun")["input"], spec, si, "host"))
    got = []
    for form in (capi.GX_XSTEP_TC_FP16_HILO, capi.GX_XSTEP_FP32):
        c = gxcorr.Correlator.from_desc(capi.job_desc_from_spec(spec, xstep=form, block_chunk=chunk))
        assert c.info.blocks_per_send == BLOCKS
        got.append(c.subint(sd).copy())
        rl, bl, bw, ac, acw = c.offsets()
        c.close()
    a, b = (g[int(ac[0]):int(acw[0])].astype(np.complex128) for g in got)
    err = np.linalg.norm(a - b) / np.linalg.norm(b)
    assert err < 6 * LONGEST / 16 * 2.0 ** -24, err
