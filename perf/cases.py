"""Timed cases of the PIV window path: what a program that uses the library
has it do, from one small frame pair to a batch of pairs.

A case is one of five kinds:
  device     one pass over a frame pair that is already on the GPU
             (Plan.process_device), in one of the plan's precisions;
  host       the same from numpy frames to numpy vectors (Plan.process);
  multipass  the 64 / 32 / 16 px chain over one pair, host frames in and
             vectors out (MultiPass.process);
  batch      several pairs of uneven sizes through that chain, pinned host
             frames in and vectors out (Batch.process_into);
  adjoint    forward pass, vector-Jacobian product into both frames'
             gradients and the propagated standard deviations, as a training
             or uncertainty loop runs them (Plan.process_device followed by
             Plan.adjoint_device).

Frames are seeded particle images with the statistics of
opiv_gb300/synth.py, rendered on the GPU (whole-number accumulation, so the
same seed gives the same frames).  Vectors come back by column group: x and y
are whole numbers of pixels up to the frame size, u and v a few pixels, sn a
ratio near one.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "openpiv-cxx_gb300"))
import opiv_gb300 as og  # noqa: E402

PRECISIONS = {"fp32": og.PREC_FP32, "fp64": og.PREC_FP64, "tc_split_bf16": og.PREC_TC_SPLIT_BF16,
              "tc_split_fp16": og.PREC_TC_SPLIT_FP16, "tc_bf16": og.PREC_TC_BF16}
MODES = {"complex": og.CORR_COMPLEX, "real": og.CORR_REAL}
SCHEDULE = ((64, 32), (32, 16), (16, 8))
# peak intensity range, noise, full scale and particles per pixel of a pixel type
LOOKS = {"u8": ((150.0, 255.0), 3.0, 255.0, 0.02), "u16": ((1500.0, 4000.0), 20.0, 4095.0, 0.03),
         "f32": ((0.6, 1.0), 0.02, 1.0, 0.02)}
DTYPES = {"u8": (np.uint8, torch.uint8, 1), "u16": (np.uint16, torch.uint16, 2), "f32": (np.float32, torch.float32, 4)}
SIGMA_F32 = 0.02


def field(kind, width, height, dtype, ia, dx, dy, mode="complex", limit=False, precision="fp32"):
    return {"kind": kind, "width": width, "height": height, "dtype": dtype, "ia": ia, "dx": dx, "dy": dy,
            "mode": mode, "limit": limit, "precision": precision}


def named(name, case):
    return dict(case, name=name)


def listed():
    return [
        # a small crop or a preview: launches and latency
        named("device_160x128_u16_w32s8", field("device", 160, 128, "u16", 32, 8, 8)),
        # the process example's own job: one 1024 x 1024 8-bit pair, 50 % overlap, host to host
        named("host_1024_u8_w32s16", field("host", 1024, 1024, "u8", 32, 16, 16)),
        # the benchmark's field: 4096 x 4096 at 75 % overlap, reference-exact peaks
        named("device_4096_u16_w32s8", field("device", 4096, 4096, "u16", 32, 8, 8)),
        # the last pass of a fine grid: small windows
        named("device_2048x1536_u16_w16s8", field("device", 2048, 1536, "u16", 16, 8, 8)),
        # large displacements: large windows at 75 % overlap
        named("device_2048_u16_w64s16", field("device", 2048, 2048, "u16", 64, 16, 16)),
        # a cropped camera frame, rows off any alignment, the real-input
        # correlator and the limited search, uneven steps
        named("device_1531x1117_u8_w32_real", field("device", 1531, 1117, "u8", 32, 12, 10, "real", True)),
        # the tensor-core precisions: the benchmark's field, then the larger windows
        named("tc_4096_u16_w32s8", field("device", 4096, 4096, "u16", 32, 8, 8, precision="tc_split_bf16")),
        named("tc_2048_u16_w48s12", field("device", 2048, 2048, "u16", 48, 12, 12, precision="tc_split_fp16")),
        named("tc_2048_u16_w64s16", field("device", 2048, 2048, "u16", 64, 16, 16, precision="tc_split_bf16")),
        # the multi-pass chain over one pair
        named("multipass_2048x1536_u16", {"kind": "multipass", "width": 2048, "height": 1536, "dtype": "u16"}),
        # a recorded sequence: pairs of uneven sizes in one call
        named("batch_8_pairs_u16", {"kind": "batch", "sizes": "1024x1024,2048x1536,3072x2048,1024x1024,"
                                                             "2048x1536,1531x1117,2048x2048,1024x1024", "dtype": "u16"}),
        # gradients and uncertainties of a float pair at 50 % overlap
        named("adjoint_2048_f32_w32s16", field("adjoint", 2048, 2048, "f32", 32, 16, 16)),
    ]


# rough time of a window in ns, by window size: keeps a drawn case within the listed ones' cost
WINDOW_NS = {16: 2.0, 32: 5.0, 48: 19.0, 64: 30.0}


def draw(rng):
    kind = rng.choice(["device", "device", "device", "tc", "tc", "host", "multipass", "batch", "adjoint"])
    if kind in ("multipass", "batch"):
        n = 1 if kind == "multipass" else rng.randint(2, 6)
        sizes = [tuple(int(round(math.exp(rng.uniform(math.log(200), math.log(2048))))) for _ in range(2)) for _ in range(n)]
        dtype = rng.choice(["u8", "u16", "u16"])
        if kind == "multipass":
            return {"kind": kind, "width": sizes[0][0], "height": sizes[0][1], "dtype": dtype}
        return {"kind": kind, "sizes": ",".join("%dx%d" % s for s in sizes), "dtype": dtype}
    ia = rng.choice([16, 32, 48, 64] if kind == "tc" else [16, 32, 64])
    top = 2048 if kind == "adjoint" else 4096
    w, h = (int(round(math.exp(rng.uniform(math.log(2 * ia), math.log(top))))) for _ in range(2))
    dx, dy = (max(2, int(round(ia * rng.uniform(0.25, 0.75)))) for _ in range(2))
    precision, dtype = "fp32", rng.choice(["u8", "u16", "f32"])
    if kind == "tc":   # u8 / u16 frames; 32 px windows start on multiples of 8 pixels
        dtype = rng.choice(["u8", "u16"])
        precision = rng.choice(["tc_split_bf16", "tc_split_fp16", "tc_bf16"])
        dx = max(4, dx // 4 * 4) if ia == 16 else max(8, dx // 8 * 8)
        w = ia + (w - ia) // dx * dx
        if ia == 16 and rng.random() < 0.5:
            dy = rng.randint(3, 6)
    elif kind == "adjoint":
        dtype = rng.choice(["u16", "f32", "f32"])
    else:
        precision = "fp64" if rng.random() < 0.1 else "fp32"

    def count():
        return (1 + (w - ia) // dx) * (1 + (h - ia) // dy)

    ns = WINDOW_NS[ia] * (4 if kind == "adjoint" else 400 if precision == "fp64" else 1)
    while count() * ns > 1.0e6 and h > 2 * ia:
        h = max(2 * ia, h * 2 // 3)
    while count() * ns > 1.0e6 and w > 2 * ia:
        w = ia + max(ia, (w - ia) * 2 // 3) // dx * dx
    mode = rng.choice(["complex", "complex", "real"])
    return field("device" if kind == "tc" else kind, w, h, dtype, ia, dx, dy, mode, kind != "adjoint" and rng.random() < 0.25,
                 precision)


# ---- frames ------------------------------------------------------------------
STAMP = 6          # half-width of a particle's spot in pixels
FIXED = 1 << 20    # spots are added up as whole numbers of 2^-20


def render(width, height, x, y, d, i0):
    acc = torch.zeros(height * width, dtype=torch.int64, device="cuda")
    offs = torch.arange(-STAMP, STAMP + 1, device="cuda")
    for s in range(0, x.numel(), 1 << 17):
        cx, cy, dd, ii = (v[s:s + (1 << 17)] for v in (x, y, d, i0))
        ix, iy = torch.floor(cx).long()[:, None] + offs, torch.floor(cy).long()[:, None] + offs
        gx = torch.exp(-8.0 * (ix + 0.5 - cx[:, None]) ** 2 / dd[:, None] ** 2)
        gy = torch.exp(-8.0 * (iy + 0.5 - cy[:, None]) ** 2 / dd[:, None] ** 2)
        gx = torch.where((ix >= 0) & (ix < width), gx, torch.zeros_like(gx))
        gy = torch.where((iy >= 0) & (iy < height), gy, torch.zeros_like(gy))
        value = torch.round((ii[:, None] * gy)[:, :, None] * gx[:, None, :] * FIXED).long()
        at = iy.clamp(0, height - 1)[:, :, None] * width + ix.clamp(0, width - 1)[:, None, :]
        acc.index_add_(0, at.reshape(-1), value.reshape(-1))
    return acc.reshape(height, width).double() / FIXED


def frames(width, height, dtype, seed):
    """A particle image pair on the GPU: a wavy field of a few pixels around a uniform shift."""
    (lo, hi), noise, full, ppp = LOOKS[dtype]
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    n = max(1, int(round(ppp * width * height)))

    def uniform(a, b, k=n):
        return a + (b - a) * torch.rand(k, dtype=torch.float64, device="cuda", generator=g)

    x, y = uniform(-4.0, width + 4.0), uniform(-4.0, height + 4.0)
    d = (2.5 + 0.5 * torch.randn(n, dtype=torch.float64, device="cuda", generator=g)).clamp(1.5, 4.0)
    i0, phase, shift = uniform(lo, hi), uniform(0.0, 2.0 * math.pi, 2), uniform(-1.0, 1.0, 2)
    if dtype == "f32":
        u, v = 0.40 + 0.1 * shift[0], 0.25 + 0.1 * shift[1]
    else:
        u = 3.0 * torch.sin(2 * math.pi * y / 1024.0 + phase[0]) + shift[0]
        v = 2.0 * torch.cos(2 * math.pi * x / 768.0 + phase[1]) + shift[1]
    pair = []
    for px, py in ((x, y), (x + u, y + v)):
        im = render(width, height, px, py, d, i0)
        im = im + noise * torch.randn(im.shape, dtype=torch.float64, device="cuda", generator=g)
        im = (torch.round(im) if dtype != "f32" else im).clamp(0.0, full)
        pair.append(im.to(torch.int32).to(DTYPES[dtype][1]) if dtype == "u16" else im.to(DTYPES[dtype][1]))
    return pair


def pitched(im, align):
    """The frame with rows on multiples of `align` bytes, and its pitch."""
    size = im.element_size()
    pitch = -(-im.shape[1] * size // align) * align
    store = torch.zeros((im.shape[0], pitch // size), dtype=im.dtype, device=im.device)
    store[:, :im.shape[1]].copy_(im)
    return store, pitch


def host_array(im):
    return im.cpu().numpy() if im.dtype != torch.uint16 else im.to(torch.int32).cpu().numpy().astype(np.uint16)


def sizes_of(case):
    if case["kind"] == "batch":
        return [tuple(int(v) for v in s.split("x")) for s in case["sizes"].split(",")]
    return [(case["width"], case["height"])]


def columns(vec):
    return [vec[:, 0:2], vec[:, 2:4], vec[:, 4]]


# ---- the timed calls -----------------------------------------------------------
def prepare(case, seed):
    kind, dtype = case["kind"], DTYPES[case["dtype"]]
    s = {"case": case}
    pairs = [frames(w, h, case["dtype"], 1000003 * seed + k) for k, (w, h) in enumerate(sizes_of(case))]
    if kind == "multipass":
        s["plan"] = og.MultiPass(case["width"], case["height"], dtype[0], SCHEDULE)
        s["a"], s["b"] = (host_array(f) for f in pairs[0])
        return s
    if kind == "batch":
        s["plan"] = og.Batch(sizes_of(case), dtype[0], SCHEDULE)
        s["frames"] = [[f.cpu().pin_memory() for f in p] for p in pairs]
        n = [s["plan"].window_count(k, len(SCHEDULE) - 1) for k in range(len(pairs))]
        s["vec"] = [torch.zeros((k, 5), dtype=torch.float32).pin_memory() for k in n]
        s["args"] = ([p[0].data_ptr() for p in s["frames"]], [p[1].data_ptr() for p in s["frames"]],
                     [w * dtype[2] for w, _ in sizes_of(case)], [v.data_ptr() for v in s["vec"]])
        s["out"] = [columns(v) for v in s["vec"]]
        return s
    tensor_core = case["precision"].startswith("tc_")
    plan = og.Plan(case["width"], case["height"], dtype[0], case["ia"], case["dx"], case["dy"], MODES[case["mode"]],
                   case["limit"], tensor_core=PRECISIONS[case["precision"]] if tensor_core else None)
    if case["precision"] == "fp64":
        plan.set_precision(og.PREC_FP64)
    s["plan"] = plan
    if kind == "host":
        s["a"], s["b"] = (host_array(f) for f in pairs[0])
        return s
    # tensor-core plans take 16-byte rows; other frames are packed as a program's arrays are
    (s["a"], s["pitch"]), (s["b"], _) = (pitched(f, 16 if tensor_core else 1) for f in pairs[0])
    s["vec"] = torch.zeros((plan.n, 5), dtype=torch.float32, device="cuda")
    s["out"] = columns(s["vec"])
    if kind == "adjoint":
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed) + 7)
        s["peak"] = torch.zeros(plan.n, dtype=torch.int32, device="cuda")
        s["cot"] = torch.randn((plan.n, 2), device="cuda", generator=g)
        s["grad_a"], s["grad_b"] = (torch.zeros((case["height"], case["width"]), device="cuda") for _ in range(2))
        s["sigma"] = torch.zeros((plan.n, 2), device="cuda")
        s["var"] = LOOKS[case["dtype"]][1] ** 2
        s["out"] = s["out"] + [s["grad_a"], s["grad_b"], s["sigma"]]
    return s


def run(s):
    kind, plan = s["case"]["kind"], s["plan"]
    if kind == "multipass":
        vec, _, disp = plan.process(s["a"], s["b"])
        return columns(vec) + [disp]
    if kind == "batch":
        plan.process_into(*s["args"])
        return s["out"]
    if kind == "host":
        return columns(plan.process(s["a"], s["b"], with_peaks=False)[0])
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "device":
        plan.process_device(s["a"].data_ptr(), s["b"].data_ptr(), s["pitch"], s["vec"].data_ptr(), None, stream)
        return s["out"]
    plan.process_device(s["a"].data_ptr(), s["b"].data_ptr(), s["pitch"], s["vec"].data_ptr(), s["peak"].data_ptr(), stream)
    s["grad_a"].zero_()
    s["grad_b"].zero_()
    plan.adjoint_device(s["a"].data_ptr(), s["b"].data_ptr(), s["pitch"], s["peak"].data_ptr(), s["cot"].data_ptr(),
                        s["grad_a"].data_ptr(), s["grad_b"].data_ptr(), s["grad_a"].stride(0) * 4, s["var"], s["var"],
                        s["sigma"].data_ptr(), stream)
    return s["out"]


# ---- what a pass cannot do without ------------------------------------------------
def grid(width, height, ia, dx, dy):
    nx, ny = 1 + (width - ia) // dx, 1 + (height - ia) // dy
    return (width - ia - dx * (nx - 1)) // 2, (height - ia - dy * (ny - 1)) // 2, nx, ny


def window_flops(ia):
    """Two complex 2-D transforms' worth (three share two windows' planes) and the product."""
    n = ia * ia
    return 2 * 5 * n * math.log2(n) + 8 * n


def work(case):
    size, total = DTYPES[case["dtype"]][2], {"bytes": 0.0, "flops": 0.0}
    steps = SCHEDULE if case["kind"] in ("multipass", "batch") else ((case["ia"], case["dx"]),)
    for w, h in sizes_of(case):
        total["bytes"] += 2.0 * w * h * size
        for k, (ia, dx) in enumerate(steps):
            _, _, nx, ny = grid(w, h, ia, dx, case.get("dy", dx))
            total["flops"] += nx * ny * window_flops(ia)
            if k == len(steps) - 1:
                total["bytes"] += nx * ny * (24.0 if case["kind"] == "multipass" else 20.0)
        if case["kind"] == "adjoint":   # gradients of both frames out; five taps of both frames, twice over
            total["bytes"] += 2.0 * w * h * 4 + nx * ny * 20.0
            total["flops"] += nx * ny * case["ia"] ** 2 * 50.0
    return total


# ---- the same in 64 bits ---------------------------------------------------------
def stacks(im, xs, ys, ia):
    """(n, ia, ia) windows of a double image at corners (xs, ys)."""
    r = torch.arange(ia, device="cuda")
    return im[(ys[:, None] + r)[:, :, None], (xs[:, None] + r)[:, None, :]]


def correlation(a, b, mode):
    z = torch.conj(torch.fft.fft2(a)) * torch.fft.fft2(b)
    if mode == "real":
        z[:, 0, :] = 0
        z[:, a.shape[1] // 2, :] = 0
        z[:, :, 0] = 0
    return torch.fft.fftshift(torch.fft.ifft2(z).real, dim=(1, 2))


def top_two(plane, limit):
    """First peak's row-major place (-1: fewer than two peaks) and the two highest values."""
    n, ia, _ = plane.shape
    d0, size = (ia // 4, ia // 2) if limit else (0, ia)
    best = torch.full_like(plane, -math.inf)
    ys, xs = slice(d0 + 1, d0 + size - 2), slice(d0 + 1, d0 + size - 1)
    c = plane[:, ys, xs]
    near = torch.stack([plane[:, d0:d0 + size - 3, xs], plane[:, d0 + 2:d0 + size - 1, xs],
                        plane[:, ys, d0:d0 + size - 2], plane[:, ys, d0 + 2:d0 + size]]).amax(0)
    best[:, ys, xs] = torch.where(near < c, c, torch.full_like(c, -math.inf))
    value, place = best.reshape(n, -1).topk(2, dim=1)
    return torch.where(torch.isfinite(value[:, 1]), place[:, 0], torch.full_like(place[:, 0], -1)), value


def offset_of(left, centre, right):
    den = 2.0 * (torch.log(left) + torch.log(right) - 2.0 * torch.log(centre))
    return torch.where(den == 0, torch.zeros_like(den), (torch.log(left) - torch.log(right)) / den)


def one_pass(fa, fb, ia, dx, dy, mode, limit, previous=None):
    """(vectors, integer displacements, first peaks) of a pass in 64 bits."""
    height, width = fa.shape
    gx, gy, nx, ny = grid(width, height, ia, dx, dy)
    k = torch.arange(nx * ny, device="cuda")
    bx, by = gx + k % nx * dx, gy + k // nx * dy
    ox, oy = torch.zeros_like(bx), torch.zeros_like(by)
    if previous is not None:
        (px0, py0, pnx, pny), pia, pdx, pdy, pdisp = previous

        def nearest(c, c0, step, n):
            return torch.where(c < c0, torch.zeros_like(c), (c - c0 + step // 2) // step).clamp(max=n - 1)

        at = nearest(by + ia // 2, py0 + pia // 2, pdy, pny) * pnx + nearest(bx + ia // 2, px0 + pia // 2, pdx, pnx)
        ox = torch.minimum(torch.maximum(pdisp[at, 0], -bx), width - ia - bx)
        oy = torch.minimum(torch.maximum(pdisp[at, 1], -by), height - ia - by)
    vec = torch.zeros((k.numel(), 5), dtype=torch.float64, device="cuda")
    disp, first = torch.stack([ox, oy], 1), torch.full_like(k, -1)
    some = max(1, (1 << 25) // (ia * ia))
    for s in range(0, k.numel(), some):
        e = slice(s, s + some)
        plane = correlation(stacks(fa, bx[e], by[e], ia), stacks(fb, bx[e] + ox[e], by[e] + oy[e], ia), mode)
        place, value = top_two(plane, limit)
        found = place >= 0
        flat, p = plane.reshape(plane.shape[0], -1), place.clamp(min=ia + 1)

        def at(o):
            return flat.gather(1, (p + o)[:, None])[:, 0]

        fx, fy = offset_of(at(-1), at(0), at(1)), offset_of(at(-ia), at(0), at(ia))
        x, y = p % ia, p // ia
        v = torch.stack([(bx[e] + ia // 2).double(), (height - by[e] - ia // 2).double(),
                         (ia // 2 - x - ox[e]).double() - fx, (ia // 2 - y - oy[e]).double() - fy,
                         torch.where(value[:, 1] > 0, value[:, 0] / value[:, 1], torch.zeros_like(fx))], 1)
        vec[e] = torch.where(found[:, None], v, torch.zeros_like(v))
        disp[e] += torch.where(found[:, None], torch.stack([x - ia // 2, y - ia // 2], 1), torch.zeros_like(disp[e]))
        first[e] = place
    return vec, disp, first


def adjoint(fa, fb, ia, dx, dy, mode, first, cot, var):
    """Gradients of both frames and the standard deviations, in 64 bits."""
    height, width = fa.shape
    gx, gy, nx, _ = grid(width, height, ia, dx, dy)
    grads, sigma = [torch.zeros(height * width, dtype=torch.float64, device="cuda") for _ in range(2)], []
    r = torch.arange(ia, device="cuda")
    some = max(1, (1 << 23) // (ia * ia))
    for s in range(0, first.numel(), some):
        k = torch.arange(s, min(s + some, first.numel()), device="cuda")
        bx, by, place = gx + k % nx * dx, gy + k // nx * dy, first[k]
        ok = place >= 0
        a, b = stacks(fa, bx, by, ia), stacks(fb, bx, by, ia)
        if mode == "real":
            sign = (1 - 2 * (r % 2)).double()[:, None]
            for w in (a, b):
                w -= w.mean(2, keepdim=True)
                w -= w.mean(1, keepdim=True) + sign * (w * sign).mean(1, keepdim=True)
        x, y = place.clamp(min=0) % ia - ia // 2, place.clamp(min=0) // ia - ia // 2

        def rolled(w, lx, ly):
            rows = ((r[None, :] + ly[:, None]) % ia)[:, :, None].expand(-1, -1, ia)
            cols = ((r[None, :] + lx[:, None]) % ia)[:, None, :].expand(-1, ia, -1)
            return w.gather(1, rows).gather(2, cols)

        lags = [(x, y), (x - 1, y), (x + 1, y), (x, y - 1), (x, y + 1)]
        c, left, right, up, down = ((a * rolled(b, lx, ly)).sum((1, 2)) for lx, ly in lags)
        coef = []
        for lo, hi in ((left, right), (up, down)):
            n, d = torch.log(lo) - torch.log(hi), 2.0 * (torch.log(lo) + torch.log(hi) - 2.0 * torch.log(c))
            good = ok & (lo > 0) & (hi > 0) & (c > 0) & (d != 0)
            part = torch.stack([-4.0 * n / (c * d * d), -(d - 2.0 * n) / (lo * d * d), (d + 2.0 * n) / (hi * d * d)])
            coef.append((torch.where(good, part, torch.zeros_like(part)), good))
        var_of = []
        da, db = torch.zeros_like(a), torch.zeros_like(a)
        for axis, (part, good) in enumerate(coef):
            taps = (0, 1, 2) if axis == 0 else (0, 3, 4)
            pa = sum(part[j][:, None, None] * rolled(b, *lags[t]) for j, t in enumerate(taps))
            pb = sum(part[j][:, None, None] * rolled(a, -lags[t][0], -lags[t][1]) for j, t in enumerate(taps))
            deviation = torch.sqrt(var * (pa * pa).sum((1, 2)) + var * (pb * pb).sum((1, 2)))
            var_of.append(torch.where(good, deviation, torch.full_like(deviation, math.nan)) * torch.where(ok, 1.0, 0.0))
            da += cot[k, axis][:, None, None] * pa
            db += cot[k, axis][:, None, None] * pb
        at = ((by[:, None] + r)[:, :, None] * width + (bx[:, None] + r)[:, None, :]).reshape(-1)
        grads[0].index_add_(0, at, da.reshape(-1))
        grads[1].index_add_(0, at, db.reshape(-1))
        sigma.append(torch.stack(var_of, 1))
    return [v.reshape(height, width) for v in grads] + [torch.cat(sigma)]


def chain(fa, fb):
    previous, vec, disp = None, None, None
    for ia, step in SCHEDULE:
        vec, disp, _ = one_pass(fa, fb, ia, step, step, "complex", False, previous)
        previous = (grid(fa.shape[1], fa.shape[0], ia, step, step), ia, step, step, disp)
    return vec, disp


def exact(case, seed):
    s = prepare(case, seed)
    width = case.get("width")

    def doubled(f):
        f = torch.as_tensor(f.astype(np.float64)) if isinstance(f, np.ndarray) else f.to(torch.float32).double()
        return f.cuda()

    if case["kind"] == "batch":
        return [columns(chain(*(doubled(f) for f in p))[0]) for p in s["frames"]]
    fa, fb = (doubled(s[k])[:, :width] for k in ("a", "b"))
    if case["kind"] == "multipass":
        vec, disp = chain(fa, fb)
        return columns(vec) + [disp]
    shape = (case["ia"], case["dx"], case["dy"])
    vec, _, first = one_pass(fa, fb, *shape, case["mode"], case["limit"])
    out = columns(vec)
    if case["kind"] == "adjoint":
        out += adjoint(fa, fb, *shape, case["mode"], first, s["cot"].double(), s["var"])
    return out
