"""Tensor-core X-step over spectra with the two rows of a pair interleaved by
channel against the plain layout (which a handle uses while it also accumulates
kurtosis): the same values, converted and multiplied in the same order, so the
results are equal bit for bit.  Input counts off the MMA tile, both sidebands,
real and complex data, both precisions, one and several passes; and bands that
do not pair (one polarisation), against the FP32 form within the split form's
bound of 1e-5 per record."""
import numpy as np
import pytest

from difx_b200 import capi
from difx_b200.jobfiles import JobSpec, Subband
from tests import jobs

pytestmark = pytest.mark.gpu


def _job(stations, pols, nchan, cplx, side, blocks=37, nbits=8):
    f0 = 6000.0 + (16 if side == "L" else 0)
    return JobSpec(name=f"tp{stations}{pols}{nchan}{int(cplx)}{side}", nstations=stations, pols=("R", "L")[:pols],
                   subbands=[Subband(f0 + 16 * i, 16.0, side, nchan) for i in range(2)], nbits=nbits,
                   sampling="COMPLEX" if cplx else "REAL", subint_ns=blocks * int(1000 * nchan / 16), execute_seconds=2,
                   max_delay_us=50.0, seed=stations)


@pytest.mark.parametrize("form", [capi.GX_XSTEP_TC_FP16_HILO, capi.GX_XSTEP_TC_FP16])
@pytest.mark.parametrize("stations,nchan,cplx,side,chunk", [(3, 128, False, "U", 0), (9, 256, True, "L", 17),
                                                            (25, 128, True, "U", 0), (5, 4096, False, "L", 0)])
def test_paired_rows_equal_plain_rows(stations, nchan, cplx, side, chunk, form):
    from difx_b200 import gxcorr
    spec = _job(stations, 2, nchan, cplx, side)
    prep = jobs.prepare(spec, [100_000_000], rho=0.2, invalid_frac=0.05, interp_source="host")
    c = gxcorr.Correlator.from_desc(capi.job_desc_from_spec(spec, xstep=form, block_chunk=chunk))
    paired = c.subint(prep.sds[0]).copy()
    c.set_kurtosis(16)
    plain = c.subint(prep.sds[0]).copy()
    c.set_kurtosis(0)
    again = c.subint(prep.sds[0])
    c.close()
    np.testing.assert_array_equal(plain, paired)
    np.testing.assert_array_equal(again, paired)


def test_single_polarisation(oracle_lib):
    from difx_b200 import gxcorr
    spec = _job(7, 1, 256, False, "U")
    prep = jobs.prepare(spec, [100_000_000], rho=0.2, invalid_frac=0.05, interp_source="host")
    got = []
    for form in (capi.GX_XSTEP_TC_FP16_HILO, capi.GX_XSTEP_FP32):
        c = gxcorr.Correlator.from_desc(capi.job_desc_from_spec(spec, xstep=form))
        got.append(c.subint(prep.sds[0]).copy())
        offs = c.offsets()
        c.close()
    rl, bl, bw, ac, acw = offs
    recs = jobs.record_offsets(prep.jd, bl, ac, spec)
    assert jobs.record_metric(got[0], got[1], recs, spec.nchan) < 1e-5
