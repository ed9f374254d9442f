"""Device corner turn against the numpy restatement (tests/vdif_streams.py): thread
counts and widths of every store path, frames that are and are not 16-byte
aligned, payloads of a few words, several calls on one multiplexer (its buffers
grow).  Bytes are equal."""
import numpy as np
import pytest

from tests import vdif_streams as vs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nthreads,nbits,fb,offset", [(1, 2, 1032, 0), (2, 8, 1032, 0), (2, 1, 1032, 4), (4, 2, 1032, 0),
                                                      (4, 4, 1032, 8), (3, 2, 40, 0), (8, 1, 72, 0), (16, 2, 8032, 0),
                                                      (16, 2, 8032, 4), (16, 1, 2088, 0), (12, 8, 1032, 0)])
def test_corner_turn(nthreads, nbits, fb, offset):
    import torch
    from difx_b200 import gxcorr
    fps, ids = 1000, list(range(nthreads))
    m = gxcorr.VdifMux(fb, fps, nbits, ids, nsort=8, ngap=100, flags=0x02)
    ofb = m.output_frame_bytes
    for n, seed in ((30, 3), (57, 4)):
        src = vs.stream(ids, n, fb, fps, nbits, seed=seed)
        d_src = torch.from_numpy(np.frombuffer(src, np.uint8).copy()).cuda()
        d_dest = torch.zeros(ofb * (n + 5) + 16, dtype=torch.uint8, device="cuda")
        st = m.run(d_src.data_ptr(), len(src), d_dest.data_ptr() + offset, ofb * (n + 5), -1, 0)
        torch.cuda.synchronize()
        out = d_dest.cpu().numpy()[offset:].tobytes()
        assert st.output_frames >= n - 10
        frames = [src[i * fb:(i + 1) * fb] for i in range(len(src) // fb)]
        t0 = int(np.frombuffer(frames[0][:4], np.uint32)[0] & 0x3FFFFFFF) * fps + int(
            np.frombuffer(frames[0][4:8], np.uint32)[0] & 0xFFFFFF)
        for f in range(st.output_frames):
            h = np.frombuffer(out[f * ofb:f * ofb + 32], np.uint32)
            assert int(h[0] & 0x3FFFFFFF) * fps + int(h[1] & 0xFFFFFF) == t0 + f
            assert int(h[2] & 0xFFFFFF) * 8 == ofb and (h[3] >> 16) & 1023 == 0
            h0 = np.frombuffer(frames[0][:32], np.uint32)   # the prototype's remaining bits
            assert (h[0] >> 30) & 1 == (h0[0] >> 30) & 1 and h[1] >> 24 == h0[1] >> 24 and h[2] >> 29 == h0[2] >> 29
            assert h[3] & ~np.uint32(1023 << 16) == h0[3] & ~np.uint32(1023 << 16)
            if h[0] >> 31:
                continue
            want = vs.corner_turn([frames[f * nthreads + k][32:] for k in range(nthreads)], nbits, False)
            assert out[f * ofb + 32:(f + 1) * ofb] == want, f
    m.close()
