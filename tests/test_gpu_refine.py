"""Windows that the FP32 kernel flags, decided from exact correlation sums
(or, where those cannot decide either, by the FP64 kernel): against the
oracle.  The frames make flagged windows the rule: particles on a high
pedestal, whose planes vary by little more than the FP32 rounding, and
two-level frames, whose planes are full of exact ties.

Tolerances: the decision is the reference's own up to its FP64 rounding, so
integer peaks are equal; u, v and sn are doubles rounded to float (half an
ulp of values up to 64 px: 1.9e-6 px; 6e-8 relative) plus that FP64 rounding,
magnified by the fit, which stays far below 1e-6 px here.
"""
import os

import numpy as np
import pytest

import opiv_gb300 as og

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 4


def frames(kind, dtype, h, w, seed):
    rng = np.random.default_rng(seed)
    texture = rng.normal(0.0, 1.0, (h + 8, w + 8))
    texture = (texture + np.roll(texture, 1, 0) + np.roll(texture, 1, 1) + np.roll(texture, (1, 1), (0, 1))) / 2
    a, b = texture[3:3 + h, 5:5 + w], texture[5:5 + h, 4:4 + w]
    if kind == "two_level":
        top = 1 if dtype == np.float32 else 255
        return tuple((f > 1.5).astype(dtype) * dtype(top) for f in (a, b))
    level, spread = {np.uint8: (200, 3), np.uint16: (4000, 200), np.float32: (3.0, 0.1)}[dtype]
    pair = [level + spread * f + spread * rng.normal(0.0, 0.5, f.shape) for f in (a, b)]
    if dtype != np.float32:
        pair = [np.clip(np.rint(f), 0, np.iinfo(dtype).max) for f in pair]
    return tuple(f.astype(dtype) for f in pair)


@pytest.mark.parametrize("mode", [og.CORR_COMPLEX, og.CORR_REAL])
@pytest.mark.parametrize("ia", [16, 32, 64])
@pytest.mark.parametrize("kind,dtype,limit", [("pedestal", np.uint16, False), ("pedestal", np.uint8, True),
                                              ("pedestal", np.float32, False), ("two_level", np.uint8, False),
                                              ("two_level", np.float32, True)])
def test_flagged_windows_against_oracle(orc, kind, dtype, limit, ia, mode):
    # an odd width (rows off any alignment) and a last odd window
    h, w = 3 * ia + 7, 4 * ia + 9
    a, b = frames(kind, dtype, h, w, 100 * ia + mode)
    plan = og.Plan(w, h, dtype, ia, ia // 2, ia // 4 + 1, mode=mode, limit_search=limit)
    vec, pk = plan.process(a, b)
    flagged = plan.exact_count()
    ref_vec, ref_pk, _ = orc.process_windows(a.astype(np.float64), b.astype(np.float64), plan.grid(), ia, mode, limit,
                                             THREADS)
    plan.close()
    code = np.where(ref_pk[:, 0] >= 0, ref_pk[:, 1] * ia + ref_pk[:, 0], -1)
    assert np.array_equal(np.where(pk >= 0, pk & og.PEAK_MASK, -1), code)
    exact = (pk >= 0) & ((pk & og.PEAK_EXACT) != 0)
    if mode == og.CORR_COMPLEX and kind == "pedestal" and not limit:
        assert flagged >= len(pk) // 4 and exact.any(), "the frames no longer flag windows"
    got, want = vec[exact].astype(np.float64), ref_vec[exact]
    assert np.array_equal(got[:, :2], want[:, :2])
    assert np.array_equal(np.isnan(got), np.isnan(want))
    d = np.abs(got - want)
    assert np.nanmax(d[:, 2:4], initial=0.0) <= 3e-6
    assert np.nanmax(d[:, 4] / np.maximum(np.abs(want[:, 4]), 1e-30), initial=0.0) <= 1e-6


@pytest.mark.parametrize("ia", [16, 32, 64])
def test_counters_between_passes(ia):
    """The second launch leaves the flag counters ready: passes over frames
    that flag many windows, few and many again on one plan, and the pipelined
    call over both, give what a fresh plan gives."""
    h, w = 3 * ia + 7, 4 * ia + 9
    many = frames("pedestal", np.uint16, h, w, 11)
    few = frames("two_level", np.uint16, h, w, 12)

    def fresh(pair):
        plan = og.Plan(w, h, np.uint16, ia, ia // 2, ia // 4 + 1)
        out = plan.process(*pair), plan.exact_count()
        plan.close()
        return out

    want = {id(p): fresh(p) for p in (many, few)}
    assert want[id(many)][1] != want[id(few)][1]
    plan = og.Plan(w, h, np.uint16, ia, ia // 2, ia // 4 + 1)
    order = (many, few, many, many, few)
    for pair in order:
        (vec, pk), n = plan.process(*pair), plan.exact_count()
        ref, count = want[id(pair)]
        assert n == count
        assert np.array_equal(vec, ref[0], equal_nan=True) and np.array_equal(pk, ref[1])
    for (vec, pk), pair in zip(plan.process_pairs(list(order)), order):
        ref = want[id(pair)][0]
        assert np.array_equal(vec, ref[0], equal_nan=True) and np.array_equal(pk, ref[1])
    plan.close()
