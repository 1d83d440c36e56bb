"""Passes that flag nearly every window: how a flagged window is decided must
not hang on its place in the flag list, which is the order in which warps
reached it.  A pass repeats bit for bit, the exact sums settle the same number
of windows each time, and the pipelined call, the allocation-free call and the
queue of a batch give the plan's results.
"""
import numpy as np
import pytest

import opiv_gb300 as og

pytestmark = pytest.mark.gpu
SPREAD = {16: 300, 32: 400, 64: 700}


def flat_frames(h, w, level, spread, seed):
    """Texture on a level far above it: the FP32 kernel can decide next to no
    window, and the exact sums some windows but not others."""
    rng = np.random.default_rng(seed)
    t = rng.normal(0.0, 1.0, (h + 8, w + 8))
    t = (t + np.roll(t, 1, 0) + np.roll(t, 1, 1) + np.roll(t, (1, 1), (0, 1))) / 2
    return [np.clip(np.rint(level + spread * f + spread * rng.normal(0.0, 0.25, (h, w))), 0, 65535).astype(np.uint16)
            for f in (t[3:3 + h, 5:5 + w], t[5:5 + h, 4:4 + w])]


@pytest.mark.parametrize("ia,step,h,w", [(16, 4, 768, 1024), (32, 8, 512, 640), (64, 16, 512, 640)])
def test_same_result_whatever_the_order(ia, step, h, w):
    torch = pytest.importorskip("torch")
    pair = flat_frames(h, w, 60000, SPREAD[ia], ia)
    plan = og.Plan(w, h, np.uint16, ia, step)
    vec, pk = plan.process(*pair)
    flagged, settled = plan.exact_count(), plan.settled_count()
    assert flagged >= plan.n // 2 and 0 < settled < flagged, "the frames no longer flag windows of both kinds"
    for _ in range(4):
        v, k = plan.process(*pair)
        assert (plan.exact_count(), plan.settled_count()) == (flagged, settled)
        assert np.array_equal(v, vec, equal_nan=True) and np.array_equal(k, pk)
    for again, (v, k) in enumerate(plan.process_pairs([pair] * 6)):
        assert np.array_equal(v, vec, equal_nan=True) and np.array_equal(k, pk), f"pass {again}"
    if ia <= 32:
        d = [torch.from_numpy(f.view(np.int16)).cuda() for f in pair]
        out = torch.zeros((plan.n, 5), dtype=torch.float32, device="cuda")
        codes = torch.zeros(plan.n, dtype=torch.int32, device="cuda")
        for _ in range(2):
            og.process_pair_device_noalloc(d[0].data_ptr(), d[1].data_ptr(), 2 * w, w, h, np.uint16, ia, step, step,
                                           og.CORR_COMPLEX, False, out.data_ptr(), codes.data_ptr())
            torch.cuda.synchronize()
            assert np.array_equal(codes.cpu().numpy(), pk)
            assert np.array_equal(out.cpu().numpy(), vec, equal_nan=True)
    plan.close()
    other = flat_frames(h // 2, w // 2, 60000, SPREAD[ia], ia + 1)
    batch = og.Batch([(w, h), (w // 2, h // 2)], np.uint16, [(ia, step)])
    for schedule in (og.BATCH_QUEUE, og.BATCH_STREAMS):
        batch.set_schedule(schedule)
        batch.upload(0, *pair)
        batch.upload(1, *other)
        for _ in range(2):
            batch.run(use_graph=False)
            v, k, _ = batch.results(0, 0)
            assert np.array_equal(v, vec, equal_nan=True) and np.array_equal(k, pk), schedule
    batch.close()


def test_more_flagged_windows_than_records():
    """The allocation-free call on a grid whose flag list leaves its fixed
    scratch fewer records than windows are flagged: the FP64 transforms decide
    all of them, as they do for a plan of that precision."""
    torch = pytest.importorskip("torch")
    ia, step, h, w = 16, 2, 1024, 1024
    pair = flat_frames(h, w, 60000, SPREAD[ia], 5)
    plan = og.Plan(w, h, np.uint16, ia, step)
    plan.process(*pair)
    # 4 MiB of scratch, 4 bytes of list a window, 40 bytes a record
    assert plan.exact_count() > ((4 << 20) - 4 * plan.n) // 40, "the frames no longer flag enough windows"
    plan.set_precision(og.PREC_FP64)
    vec, pk = plan.process(*pair)
    d = [torch.from_numpy(f.view(np.int16)).cuda() for f in pair]
    out = torch.zeros((plan.n, 5), dtype=torch.float32, device="cuda")
    codes = torch.zeros(plan.n, dtype=torch.int32, device="cuda")
    og.process_pair_device_noalloc(d[0].data_ptr(), d[1].data_ptr(), 2 * w, w, h, np.uint16, ia, step, step,
                                   og.CORR_COMPLEX, False, out.data_ptr(), codes.data_ptr())
    torch.cuda.synchronize()
    got, code = out.cpu().numpy(), codes.cpu().numpy()
    exact = (code >= 0) & ((code & og.PEAK_EXACT) != 0)
    assert exact.sum() > plan.n // 2
    assert np.array_equal(code[exact] & og.PEAK_MASK, pk[exact] & og.PEAK_MASK)
    assert np.array_equal(got[exact], vec[exact], equal_nan=True)
    plan.close()
