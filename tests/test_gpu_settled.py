"""Flagged windows that the exact correlation sums settle, in every mode,
window size and pixel type: counted, so that it is known that the sums and not
the FP64 transforms decided them, and against the oracle.

Texture on a level `ratio` times above it: the FP32 bound is then some 1e-2 to
4e-2 of a plane's peak, which no certified fit survives, and leaves a handful
of cells that could be the two peaks.  Tolerances: integer peaks equal; u, v
and sn are doubles rounded to float (half an ulp of values up to 64 px: 1.9e-6
px; 6e-8 of sn) plus FP64 rounding, which these fits magnify by less than 1e5.
"""
import os

import numpy as np
import pytest

import opiv_gb300 as og

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 4
LEVEL = {np.uint8: 240.0, np.uint16: 24000.0, np.float32: 3.0}
RATIO = {16: 200.0, 32: 100.0, 64: 60.0}


def level_frames(dtype, h, w, ratio, seed):
    rng = np.random.default_rng(seed)
    t = rng.normal(0.0, 1.0, (h + 8, w + 8))
    t = (t + np.roll(t, 1, 0) + np.roll(t, 1, 1) + np.roll(t, (1, 1), (0, 1))) / 2
    level = LEVEL[dtype]
    pair = [level * (1 + (f + 0.25 * rng.normal(0.0, 1.0, (h, w))) / ratio) for f in (t[3:3 + h, 5:5 + w], t[5:5 + h, 4:4 + w])]
    if dtype != np.float32:
        pair = [np.clip(np.rint(f), 0, np.iinfo(dtype).max) for f in pair]
    return [f.astype(dtype) for f in pair]


@pytest.mark.parametrize("limit", [False, True])
@pytest.mark.parametrize("mode", [og.CORR_COMPLEX, og.CORR_REAL])
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32])
@pytest.mark.parametrize("ia", [16, 32, 64])
def test_exact_sums_settle_windows(orc, ia, dtype, mode, limit):
    h, w = 4 * ia + 3, 5 * ia + 7
    a, b = level_frames(dtype, h, w, RATIO[ia], ia + mode)
    plan = og.Plan(w, h, dtype, ia, ia // 2 - 1, mode=mode, limit_search=limit)
    vec, pk = plan.process(a, b)
    flagged, settled = plan.exact_count(), plan.settled_count()
    ref_vec, ref_pk, _ = orc.process_windows(a.astype(np.float64), b.astype(np.float64), plan.grid(), ia, mode, limit,
                                             THREADS)
    plan.close()
    code = np.where(ref_pk[:, 0] >= 0, ref_pk[:, 1] * ia + ref_pk[:, 0], -1)
    assert np.array_equal(np.where(pk >= 0, pk & og.PEAK_MASK, -1), code)
    exact = (pk >= 0) & ((pk & og.PEAK_EXACT) != 0)
    assert exact.sum() <= flagged
    assert settled >= len(pk) // 2, (settled, flagged, len(pk))
    got, want = vec[exact].astype(np.float64), ref_vec[exact]
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[:, :2], want[:, :2])
    assert np.nanmax(np.abs(got[:, 2:4] - want[:, 2:4])) <= 3e-6
    assert np.nanmax(np.abs(got[:, 4] - want[:, 4]) / np.maximum(np.abs(want[:, 4]), 1e-30)) <= 1e-6
