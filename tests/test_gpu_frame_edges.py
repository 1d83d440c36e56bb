"""Frames whose first and last pixels are a window's: rows whose 16-byte blocks
would leave the frame are read byte by byte, at every kind of offset from a
block boundary and with odd pitches, and give what the packed, aligned frames
give (the arithmetic is the same whatever the alignment).
"""
import numpy as np
import pytest

import opiv_gb300 as og
from opiv_gb300 import synth

pytestmark = pytest.mark.gpu
LOOKS = {np.uint8: ((150, 255), 3.0, 255.0), np.uint16: ((1500, 4000), 20.0, 4095.0), np.float32: ((0.6, 1.0), 0.02, 1.0)}


def pair_of(dtype, h, w, seed):
    i0, noise, full = LOOKS[dtype]
    return synth.particle_pair(h, w, ppp=0.05, i0_range=i0, noise=noise, full_scale=full, dtype=dtype, seed=seed,
                               displacement=lambda x, y: (np.full_like(x, 1.4), np.full_like(y, -2.25)))


def on_device(torch, pair, offset, pitch):
    """Views' first pixels and the tensors that hold them."""
    size = pair[0].itemsize
    h, w = pair[0].shape
    out = []
    for f in pair:
        raw = np.zeros(offset * size + pitch * (h - 1) + w * size, np.uint8)
        np.lib.stride_tricks.as_strided(raw[offset * size:].view(f.dtype), (h, w), (pitch, size))[:] = f
        out.append(torch.from_numpy(raw).cuda())
    return [t.data_ptr() + offset * size for t in out], out


@pytest.mark.parametrize("ia", [16, 32, 64])
@pytest.mark.parametrize("dtype,offsets", [(np.uint8, range(16)), (np.uint16, range(8)), (np.float32, range(4))])
def test_windows_at_the_corners(dtype, offsets, ia):
    torch = pytest.importorskip("torch")
    size = np.dtype(dtype).itemsize
    h, w = ia + 3 * 16, ia + 4 * 16   # the grid of step 16 ends at the last pixel
    pair = pair_of(dtype, h, w, ia)
    plan = og.Plan(w, h, dtype, ia, 16)
    assert plan.grid().min() == 0 and (plan.grid().max(axis=0) == (w - ia, h - ia)).all()

    def run(offset, pitch):
        at, hold = on_device(torch, pair, offset, pitch)
        vec = torch.zeros((plan.n, 5), dtype=torch.float32, device="cuda")
        pk = torch.zeros(plan.n, dtype=torch.int32, device="cuda")
        plan.process_device(at[0], at[1], pitch, vec.data_ptr(), pk.data_ptr())
        torch.cuda.synchronize()
        return vec.cpu().numpy(), pk.cpu().numpy()

    want = run(0, (w * size + 15) // 16 * 16)
    assert (want[1] >= 0).any()
    for offset in offsets:
        for pad in (0, 1, 3):
            got = run(offset, (w + pad) * size)
            assert np.array_equal(got[0], want[0], equal_nan=True) and np.array_equal(got[1], want[1]), (offset, pad)
    plan.close()


@pytest.mark.parametrize("dtype,offsets", [(np.uint8, (0, 5)), (np.uint16, (0, 3)), (np.float32, (0, 1))])
def test_displaced_windows(dtype, offsets):
    torch = pytest.importorskip("torch")
    size = np.dtype(dtype).itemsize
    h, w = 3 * 32 + 11, 4 * 32 + 7
    pair = pair_of(dtype, h, w, 5)
    mp = og.MultiPass(w, h, dtype, [(32, 16), (16, 8)])
    want = mp.process(*pair)
    for offset in offsets:
        for pad in (0, 1, 9):
            pitch = (w + pad) * size
            at, hold = on_device(torch, pair, offset, pitch)
            og._check(og.load().opiv_multipass_process_device(mp._h, at[0], at[1], pitch, None))
            torch.cuda.synchronize()
            for g, r in zip(mp.results(1), want):
                assert np.array_equal(g, r, equal_nan=g.dtype == np.float32), (offset, pad)
    mp.close()
