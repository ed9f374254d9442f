"""Long sums of the FP32 X-step: slices of several runs, whose sums pass from the
registers they grow in to a second level (8 and 16 rows: registers, 32 rows: the
accumulators in memory), block counts off the runs and the stages, one and
several passes, and the largest K-split, as few channels get it.

One band of 64 channels keeps the oracle quick.  Tolerance as the parity tests':
records within 1e-5; the two launch shapes add the same blocks in the same order
and agree exactly."""
import numpy as np
import pytest

from difx_b200 import capi
from difx_b200.jobfiles import JobSpec, Subband
from tests import jobs
from tests.test_gpu_parity import REC_TOL, W_TOL, _compare, _params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stations,blocks,chunk", [
    (2, 4997, 0),        # 8 rows: 64 slices of 80 blocks
    (2, 9001, 0),        # 64 slices of two runs
    (3, 9000, 4500),     # in two passes
    (9, 9001, 0),        # 16 rows: 64 slices of two runs
    (9, 5003, 1999),     # three passes
    (17, 17409, 0),      # 32 rows: 64 slices of two runs
    (17, 6001, 3000),    # two passes
    (33, 5003, 0),       # off the diagonal too
])
def test_long_slices(stations, blocks, chunk, oracle_lib):
    from difx_b200 import gxcorr
    spec = JobSpec(name=f"xl{stations}_{blocks}_{chunk}", nstations=stations, pols=("R",),
                   subbands=[Subband(6000.0, 16.0, "U", 64)], nbits=8, subint_ns=blocks * 4000, execute_seconds=2,
                   max_delay_us=50.0, seed=stations)
    prep = jobs.prepare(spec, [100_000_000], rho=0.2, invalid_frac=0.03, interp_source="host")
    c = gxcorr.Correlator.from_desc(capi.job_desc_from_spec(spec, block_chunk=chunk))
    g = c.subint(prep.sds[0]).copy()
    c.set_tiles(1, 0)
    other = c.subint(prep.sds[0])
    c.close()
    o = oracle_lib.subint(prep.jd, prep.sds[0], _params(oracle_lib, spec))
    m, wrel = _compare(g, o, prep.jd, spec, oracle_lib)
    assert m < REC_TOL and wrel < W_TOL, (m, wrel)
    np.testing.assert_array_equal(other, g)
