"""The adjoint over every layout of a window in the lanes and warps (16, 32
and 64 px, both modes), on frames of odd sizes with overlapping windows:
gradients and propagated standard deviations against an FP64 numpy gradient.

Tolerance: 2e-3 of the largest entry, as the 32 px tests: FP32 sums of up to
4096 products carry about 4e-6 of the plane value into the fit's second
difference, which for these images is a few percent of the value.
"""
import numpy as np
import pytest

import opiv_gb300 as og
from opiv_gb300 import synth

pytestmark = pytest.mark.gpu


def project(x):
    sign = 1.0 - 2.0 * (np.arange(x.shape[0]) % 2)[:, None]
    x = x - x.mean(1, keepdims=True)
    return x - x.mean(0) - sign * (x * sign).mean(0)


def window_gradients(a, b, code, real):
    """du/da, du/db, dv/da, dv/db of one window, or None per axis without a derivative."""
    w = a.shape[0]
    px, py = code % w, code // w
    if real:
        a, b = project(a), project(b)
    out = []
    for lo, hi in (((-1, 0), (1, 0)), ((0, -1), (0, 1))):
        lags = [(px - w // 2 + ex, py - w // 2 + ey) for ex, ey in ((0, 0), lo, hi)]
        c, l, r = (np.sum(a * np.roll(b, (-dy, -dx), (0, 1))) for dx, dy in lags)
        if min(c, l, r) <= 0:
            out.append(None)
            continue
        n, d = np.log(l) - np.log(r), 2 * (np.log(l) + np.log(r) - 2 * np.log(c))
        g = (-4 * n / (c * d * d), -(d - 2 * n) / (l * d * d), (d + 2 * n) / (r * d * d))
        out.append((sum(k * np.roll(b, (-dy, -dx), (0, 1)) for k, (dx, dy) in zip(g, lags)),
                    sum(k * np.roll(a, (dy, dx), (0, 1)) for k, (dx, dy) in zip(g, lags))))
    return out


@pytest.mark.parametrize("mode", [og.CORR_COMPLEX, og.CORR_REAL])
@pytest.mark.parametrize("ia", [16, 32, 64])
@pytest.mark.parametrize("dtype,outputs", [(np.float32, "both"), (np.uint8, "both"), (np.uint16, "vjp"),
                                           (np.uint16, "sigma")])
def test_layouts_against_fp64(ia, mode, dtype, outputs):
    torch = pytest.importorskip("torch")
    h, w = 2 * ia + 5, 3 * ia + 3
    i0, noise, full = {np.float32: ((0.6, 1.0), 0.02, 1.0), np.uint8: ((150, 255), 3.0, 255.0),
                       np.uint16: ((1500, 4000), 20.0, 4095.0)}[dtype]
    a, b = synth.particle_pair(h, w, ppp=0.05, i0_range=i0, noise=noise, full_scale=full, dtype=dtype, seed=50 + ia,
                               displacement=lambda x, y: (np.full_like(x, 1.4), np.full_like(y, -2.25)))
    plan = og.Plan(w, h, dtype, ia, ia // 2 + 1, ia // 2, mode=mode)
    da, db = (torch.from_numpy(f.view(np.int16) if dtype == np.uint16 else f).cuda() for f in (a, b))
    pitch = w * np.dtype(dtype).itemsize
    vec = torch.empty((plan.n, 5), dtype=torch.float32, device="cuda")
    pk = torch.empty(plan.n, dtype=torch.int32, device="cuda")
    cot = torch.from_numpy(np.random.default_rng(ia).normal(size=(plan.n, 2)).astype(np.float32)).cuda()
    ga, gb = (torch.zeros((h, w + 3), device="cuda") for _ in range(2))
    sigma = torch.full((plan.n, 2), -1.0, device="cuda")
    var = noise * noise
    plan.process_device(da.data_ptr(), db.data_ptr(), pitch, vec.data_ptr(), pk.data_ptr())
    plan.adjoint_device(da.data_ptr(), db.data_ptr(), pitch, pk.data_ptr(), cot.data_ptr() if outputs != "sigma" else 0,
                        ga.data_ptr(), gb.data_ptr(), 4 * (w + 3), var, var,
                        sigma.data_ptr() if outputs != "vjp" else 0)
    torch.cuda.synchronize()
    ga, gb, sigma, pk, cot = (t.cpu().numpy() for t in (ga, gb, sigma, pk, cot))
    ra, rb, rs = np.zeros((h, w)), np.zeros((h, w)), np.zeros((plan.n, 2))
    for k, (x, y) in enumerate(plan.grid()):
        if pk[k] < 0:
            continue
        at = (slice(y, y + ia), slice(x, x + ia))
        grads = window_gradients(a[at].astype(np.float64), b[at].astype(np.float64), int(pk[k]) & og.PEAK_MASK,
                                 mode == og.CORR_REAL)
        for axis, g in enumerate(grads):
            if g is None:
                rs[k, axis] = np.nan
                continue
            ra[at] += cot[k, axis] * g[0]
            rb[at] += cot[k, axis] * g[1]
            rs[k, axis] = np.sqrt(var * np.sum(g[0] ** 2) + var * np.sum(g[1] ** 2))
    plan.close()
    if outputs != "sigma":
        assert np.abs(ra).max() > 0
        for got, want in ((ga, ra), (gb, rb)):
            assert np.abs(got[:, :w] - want).max() <= 2e-3 * np.abs(want).max()
            assert not got[:, w:].any()
    else:
        assert not ga.any() and not gb.any()
    if outputs != "vjp":
        assert np.array_equal(np.isnan(sigma), np.isnan(rs))
        assert np.nanmax(np.abs(sigma - rs)) <= 2e-3 * np.nanmax(rs)
    else:
        assert (sigma == -1.0).all()
