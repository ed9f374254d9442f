"""The FP32 X-step against the oracle at the input counts where its shape
changes (super-tiles of 8, 16 and 32 rows, one to three of them a side), with
one and with several passes of blocks (sums stored, then added to), K-split
slices that end off the stages, and both launch shapes.

Tolerance as the parity tests': records within 1e-5 by the per-record metric;
the two launch shapes add the same blocks in the same order, so they agree
exactly."""
import numpy as np
import pytest

from difx_b200 import capi
from difx_b200.jobfiles import JobSpec, Subband
from tests import jobs
from tests.test_gpu_parity import REC_TOL, W_TOL, _compare, _params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stations,pols,chunk", [(2, 1, 0), (7, 1, 50), (4, 2, 0), (9, 1, 0), (8, 2, 67), (17, 1, 0),
                                                 (16, 2, 96), (33, 1, 0), (32, 2, 70), (33, 2, 0)])
def test_input_counts(stations, pols, chunk, oracle_lib):
    from difx_b200 import gxcorr
    nchan, blocks = (64, 203) if stations < 32 else (64, 141)
    spec = JobSpec(name=f"xm{stations}{pols}{chunk}", nstations=stations, pols=("R", "L")[:pols],
                   subbands=[Subband(6000.0 + 16 * i, 16.0, "U", nchan) for i in range(4 // pols)], nbits=2,
                   subint_ns=blocks * 4000, execute_seconds=2, max_delay_us=50.0, seed=stations)
    prep = jobs.prepare(spec, [100_000_000], rho=0.2, invalid_frac=0.03, interp_source="host")
    jd = capi.job_desc_from_spec(spec, block_chunk=chunk)
    c = gxcorr.Correlator.from_desc(jd)
    g = c.subint(prep.sds[0]).copy()
    again = c.subint(prep.sds[0]).copy()   # nothing left over from the call before
    c.set_tiles(1, 0)
    other = c.subint(prep.sds[0])
    c.close()
    o = oracle_lib.subint(prep.jd, prep.sds[0], _params(oracle_lib, spec))
    m, wrel = _compare(g, o, prep.jd, spec, oracle_lib)
    assert m < REC_TOL and wrel < W_TOL, (m, wrel)
    np.testing.assert_array_equal(again, g)
    np.testing.assert_array_equal(other, g)
