"""Levels of 8-bit codes in the F-step: (code - 128) / 3.3, or with
SYMMETRIC_8_BIT_VDIF (code - 127.5) / 3.3, for which the kernel must leave its
integer arithmetic.  A stream of one constant code has F times its level in
channel 0 of an upper sideband (post-F rotation: only phases after the transform).

Tolerance: the transform's FP32 sums of equal terms, within 1e-5."""
import numpy as np
import pytest

from difx_b200 import capi
from difx_b200.jobfiles import JobSpec, Subband
from tests import jobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("pols", [("R",), ("R", "L")])
@pytest.mark.parametrize("nchan,code", [(256, 200), (4096, 3)])
def test_constant_code(nchan, code, pols, symmetric, monkeypatch):
    from difx_b200 import gxcorr
    if symmetric:
        monkeypatch.setenv("SYMMETRIC_8_BIT_VDIF", "1")
    else:
        monkeypatch.delenv("SYMMETRIC_8_BIT_VDIF", raising=False)
    spec = JobSpec(name=f"lev{nchan}{len(pols)}{int(symmetric)}", nstations=2, pols=pols, subbands=[Subband(6000.0, 16.0, "U", nchan)],
                   nbits=8, fringe_rot_order=0, subint_ns=4 * int(1000 * nchan / 16), execute_seconds=2, max_delay_us=50.0, seed=9)
    prep = jobs.prepare(spec, [100_000_000], interp_source="host")
    si = prep.subs[0]
    for d in si.data:
        d.reshape(-1, spec.framebytes)[:, 32:] = code
    c = gxcorr.Correlator.from_desc(prep.jd)
    c.subint(capi.subint_desc_host(si, prep.interps[0]))
    level = (code - (127.5 if symmetric else 128.0)) / 3.3
    for blk in (0, 3):
        x, w = c.spectra(0, blk, spec.nbands)
        assert w == 1.0
        dc = np.abs(np.asarray(x).reshape(spec.nbands, nchan)[:, 0])
        np.testing.assert_allclose(dc, 2 * nchan * abs(level), rtol=1e-5)
    c.close()
