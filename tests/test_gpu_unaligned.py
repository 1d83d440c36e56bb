"""Frames whose rows start anywhere: the row loads of the 16 and 32 px kernels
(and the 64 px kernel's) on frames at every kind of offset from a 16-byte
boundary and with odd pitches, against the same frames packed and aligned.
The arithmetic is the same whatever the alignment: results are identical.
"""
import numpy as np
import pytest

import opiv_gb300 as og
from opiv_gb300 import synth

pytestmark = pytest.mark.gpu
LOOKS = {np.uint8: ((150, 255), 3.0, 255.0), np.uint16: ((1500, 4000), 20.0, 4095.0), np.float32: ((0.6, 1.0), 0.02, 1.0)}


@pytest.mark.parametrize("ia", [16, 32, 64])
@pytest.mark.parametrize("dtype,offsets", [(np.uint8, (0, 1, 7, 15)), (np.uint16, (0, 1, 4, 7)), (np.float32, (0, 1, 3))])
def test_rows_anywhere(dtype, offsets, ia):
    torch = pytest.importorskip("torch")
    size = np.dtype(dtype).itemsize
    h, w = 2 * ia + 3, 3 * ia + 16
    i0, noise, full = LOOKS[dtype]
    pair = synth.particle_pair(h, w, ppp=0.05, i0_range=i0, noise=noise, full_scale=full, dtype=dtype, seed=ia,
                               displacement=lambda x, y: (np.full_like(x, 1.4), np.full_like(y, -2.25)))
    # grids whose windows start on 16-byte blocks of an aligned frame
    plan = og.Plan(w, h, dtype, ia, 16, 9)

    def run(offset, pad):
        pitch = (w + pad) * size
        room = offset * size + pitch * h
        views = []
        for f in pair:
            raw = np.zeros(room, np.uint8)
            rows = np.lib.stride_tricks.as_strided(raw[offset * size:].view(dtype), (h, w), (pitch, size))
            rows[:] = f
            views.append(torch.from_numpy(raw).cuda())
        vec = torch.zeros((plan.n, 5), dtype=torch.float32, device="cuda")
        pk = torch.zeros(plan.n, dtype=torch.int32, device="cuda")
        plan.process_device(views[0].data_ptr() + offset * size, views[1].data_ptr() + offset * size, pitch,
                            vec.data_ptr(), pk.data_ptr())
        torch.cuda.synchronize()
        return vec.cpu().numpy(), pk.cpu().numpy()

    want = run(0, 16 - w % 16)
    assert (want[1] >= 0).any()
    for offset in offsets:
        for pad in (0, 1, 5):
            got = run(offset, pad)
            assert np.array_equal(got[0], want[0], equal_nan=True) and np.array_equal(got[1], want[1]), (offset, pad)
    plan.close()
