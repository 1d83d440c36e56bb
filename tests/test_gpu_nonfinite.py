"""Float frames with a NaN, an infinite or a huge pixel (one whose square is
not a float): every window is the oracle's, above all the healthy windows that
share a transform with a bad one (the FP32 kernels take windows in pairs).

Tolerances: integer peaks equal; u, v and sn within the FP32 kernel's
certified bounds (1e-4 px; 1e-5 of the plane's peak).
"""
import os

import numpy as np
import pytest

import opiv_gb300 as og
from opiv_gb300 import synth

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 4


def frames(ia, bad):
    """3 x 5 windows side by side; bad pixels in windows whose partners in
    the pair are healthy, the first and the second of a pair, in either frame."""
    h, w = 3 * ia, 5 * ia
    a, b = synth.particle_pair(h, w, ppp=0.06, i0_range=(0.6, 1.0), noise=0.02, full_scale=1.0, dtype=np.float32,
                               seed=ia, displacement=lambda x, y: (np.full_like(x, 1.4), np.full_like(y, -0.75)))
    for win, f in ((1, a), (6, a), (9, b)):
        f[(win // 5) * ia + ia // 3, (win % 5) * ia + ia // 2] = bad
    return a, b


@pytest.mark.parametrize("mode", [og.CORR_COMPLEX, og.CORR_REAL])
@pytest.mark.parametrize("ia", [16, 32, 64])
@pytest.mark.parametrize("bad", [np.nan, np.inf, 3e19])
def test_bad_pixels_stay_in_their_windows(orc, bad, ia, mode):
    a, b = frames(ia, bad)
    plan = og.Plan(a.shape[1], a.shape[0], np.float32, ia, ia, mode=mode)
    vec, pk = plan.process(a, b)
    ref_vec, ref_pk, _ = orc.process_windows(a.astype(np.float64), b.astype(np.float64), plan.grid(), ia, mode, False,
                                             THREADS)
    plan.close()
    code = np.where(ref_pk[:, 0] >= 0, ref_pk[:, 1] * ia + ref_pk[:, 0], -1)
    healthy = ~np.isin(np.arange(15), (1, 6, 9))
    assert (code[healthy] >= 0).all()
    assert np.array_equal(np.where(pk >= 0, pk & og.PEAK_MASK, -1), code)
    got = vec.astype(np.float64)
    assert np.array_equal(np.isnan(got), np.isnan(ref_vec))
    assert np.array_equal(got[:, :2], ref_vec[:, :2])
    assert np.nanmax(np.abs(got[:, 2:4] - ref_vec[:, 2:4])) <= 1e-4
    sn = ref_vec[:, 4]
    assert (np.abs(got[:, 4] - sn) <= 1e-5 * np.abs(sn) * (1 + np.abs(sn))).all()


@pytest.mark.parametrize("mode", [og.CORR_COMPLEX, og.CORR_REAL])
@pytest.mark.parametrize("ia", [16, 32, 64])
def test_planes_of_a_batch(ia, mode):
    rng = np.random.default_rng(ia)
    a, b = rng.random((9, ia, ia)), rng.random((9, ia, ia))
    a[1, 3, 5] = np.nan
    b[6, 0, 0] = np.nan
    got = og.cross_correlate_batch(a, b, mode)
    want = og.cross_correlate_batch(a, b, mode, exact=True)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.isnan(got[[1, 6]]).all()
    healthy = [0, 2, 3, 4, 5, 7, 8]
    scale = np.abs(want[healthy]).max(axis=(1, 2), keepdims=True)
    assert (np.abs(got[healthy] - want[healthy]) <= 1e-5 * scale).all()
