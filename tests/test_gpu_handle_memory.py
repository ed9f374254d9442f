"""Device memory of a handle opened with the default pass length: long passes
(more than 4096 blocks) take a small part of the free memory, so that a program
that opens many handles, or allocates its own buffers after them, is not refused."""
import pytest

from difx_b200 import capi
from difx_b200.jobfiles import JobSpec, Subband

pytestmark = pytest.mark.gpu


def _job(stations, subbands, nchan, blocks):
    return JobSpec(name="mem", nstations=stations, subbands=[Subband(6000.0 + 32 * i, 32.0, "U", nchan) for i in range(subbands)],
                   nbits=2, subint_ns=blocks * int(1000 * nchan / 32), execute_seconds=2)


def test_long_passes_leave_room():
    import torch
    from difx_b200 import gxcorr
    # 32 inputs x 16 x 256 channels: 1 MB of spectra a block, 34 GB in passes of 32768
    per_block = 32 * 16 * 256 * 8
    free, _ = torch.cuda.mem_get_info()
    c = gxcorr.Correlator.from_desc(capi.job_desc_from_spec(_job(16, 16, 256, 32768)))
    assert c.info.blocks_per_send == 32768
    assert c.info.block_chunk <= max(4096, free // 8 // per_block)
    c.close()
