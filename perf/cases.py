"""The scene-flow workloads whose speed counts, through the package's public calls.

A case is a dict of plain values; `prepare` makes a seeded state on the GPU
(or on the host, where a program hands over host frames), `run` does one pass,
`work` states what a pass cannot do without, `exact` gives its result in 64
bits from plain torch.  `listed` holds the reference set, `draw` more cases of
the same ranges.
"""
import math
import os
import sys

import numpy as np
import torch
import torch.nn.functional as F

sys.path.insert(0, os.path.abspath("pd-flow_gb300"))
import pdflow  # noqa: E402

ROWS = (15, 30, 60, 120, 240, 480)


def listed():
    return [
        # One 320x240 pair solved at 60x80 from host frames: the smallest call of a camera loop.
        dict(name="pair_qvga_r60", kind="pair", rows=60, width=320, input="u16", finest=100, objects=3),
        # The reference application's default: one 320x240 pair at full resolution, float staging buffers.
        dict(name="pair_qvga_r240", kind="pair", rows=240, width=320, input="float", finest=100, objects=3),
        # The live application: one 640x480 RGB-D camera pair at full resolution.
        dict(name="pair_vga_r480", kind="pair", rows=480, width=640, input="rgb", finest=100, objects=6),
        # A serving lane's batch: the new frames of six cameras, solved together, flows back to the host.
        dict(name="slots_qvga_r240_n6", kind="slots", rows=240, width=320, n=6, finest=100, objects=3),
        # An odd number of 320x240 pairs from device frames, with the energy of each solution.
        dict(name="batch_qvga_r240_n13", kind="batch", rows=240, width=320, n=13, finest=100, objects=3, energy=True),
        # A few 640x480 pairs of a device pipeline, with a schedule that leaves a remainder at every level.
        dict(name="batch_vga_r480_n5", kind="batch", rows=480, width=640, n=5, finest=97, objects=6, energy=False),
        # 640x480 frames solved at half resolution: the preview setting of a VGA camera rig.
        dict(name="batch_vga_r240_n16", kind="batch", rows=240, width=640, n=16, finest=100, objects=6, energy=False),
        # The throughput workload: 64 pairs of 640x480 frames at full resolution, frames and flows on the device.
        dict(name="batch_vga_r480_n64", kind="batch", rows=480, width=640, n=64, finest=100, objects=6, energy=False),
        # Pairs of four resolutions in one call, host frames and host flows.
        dict(name="mixed_n16", kind="mixed", n60=4, n120=4, n240=3, n480=5, objects=4),
        # The learned warm start of a batch (network, energies, decision, continuation).
        dict(name="learned_vga_r480_n16", kind="learned", rows=480, width=640, n=16, scale=0.75, objects=6),
        # One training step's loss and gradients of the warm-start network (forward and backward).
        dict(name="net_gradients_n64", kind="net", n=64, objects=3),
    ]


def draw(rng):
    kind = rng.choice(("pair", "pair", "slots", "batch", "batch", "mixed", "learned", "net"))
    objects = rng.randint(1, 8)
    spread = lambda hi: int(round(math.exp(rng.uniform(0.0, math.log(hi)))))  # noqa: E731
    finest = rng.choice((100, 100, rng.randint(40, 99)))
    if kind == "mixed":
        return dict(kind=kind, n60=rng.randint(0, 6), n120=rng.randint(0, 5), n240=rng.randint(1, 5),
                    n480=rng.randint(0, 5), objects=objects)
    if kind == "net":
        return dict(kind=kind, n=spread(64), objects=objects)
    if kind == "pair":
        width = rng.choice((320, 640))
        return dict(kind=kind, rows=rng.choice(ROWS if width == 640 else ROWS[:5]), width=width,
                    input=rng.choice(("u16", "float", "rgb")), finest=finest, objects=objects)
    rows = rng.choice((120, 240, 480) if kind == "learned" else (60, 120, 240, 480))
    width = 640 if rows == 480 else rng.choice((320, 640))
    if kind == "learned":
        return dict(kind=kind, rows=rows, width=width, n=1 + spread(23), scale=rng.choice((0.5, 0.6, 0.75, 0.9)),
                    objects=objects)
    if kind == "slots":
        return dict(kind=kind, rows=rows, width=width, n=spread(12), finest=finest, objects=objects)
    return dict(kind=kind, rows=rows, width=width, n=1 + spread(60), finest=finest, objects=objects,
                energy=rng.random() < 0.3)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _frames(n, width, objects, seed):
    """Two frames of n scenes on the GPU: intensity uint8 and depth in 1/5000 m
    (int16) [n, h, w].  A textured slanted plane at 2-4 m, spheres and slanted
    squares at 1-2.3 m that move by up to 5 cm, textures fixed to the surfaces,
    depth noise 1.5e-3 z^2 and 2 % holes."""
    h = width * 3 // 4
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + width * 131 + n)
    dev = dict(device="cuda", generator=g)
    uni = lambda lo, hi, *s: lo + (hi - lo) * torch.rand(*s, **dev)  # noqa: E731
    f = 525.0 * width / 640
    xn = ((torch.arange(width, device="cuda") - width / 2) / f).view(1, 1, -1).expand(n, h, width)
    yn = ((torch.arange(h, device="cuda") - h / 2) / f).view(1, -1, 1).expand(n, h, width)
    sample = lambda grid, x, y: F.grid_sample(grid, torch.stack((x, y), -1), mode="bicubic",  # noqa: E731
                                              padding_mode="reflection", align_corners=False)[:, 0]
    per = lambda lo, hi: uni(lo, hi, n, 1, 1)  # noqa: E731
    plane = per(2.6, 3.2) / (1.0 - per(-0.2, 0.2) * xn - per(-0.2, 0.2) * yn)
    px, py = 1.4 * xn, 1.4 * yn
    ground = 0.65 * sample(torch.rand(n, 1, 96, 96, **dev), px, py) + 0.35 * sample(
        torch.rand(n, 1, 192, 192, **dev), px, py)
    things = []
    for _ in range(objects):
        zc = per(1.0, 2.3)
        things.append((per(-0.4, 0.4) * zc, per(-0.3, 0.3) * zc, zc, per(0.08, 0.2), torch.rand(n, 1, 1, **dev) < 0.5,
                       [per(-0.03, 0.03) for _ in range(3)], per(0.6, 1.0), torch.rand(n, 1, 12, 12, **dev)))
    out = []
    for k in range(2):
        z, tex = plane, 0.15 + 0.8 * ground
        for cx, cy, zc, rad, ball, move, albedo, grid in things:
            pz = zc + k * move[2]
            dx, dy = xn * pz - (cx + k * move[0]), yn * pz - (cy + k * move[1])
            r2 = dx * dx + dy * dy
            depth = torch.where(ball, pz - (rad * rad - r2).clamp_min(0).sqrt(), pz - 0.3 * dx)
            hit = torch.where(ball, r2 < rad * rad, torch.maximum(dx.abs(), dy.abs()) < rad) & (depth < z)
            z = torch.where(hit, depth, z)
            tex = torch.where(hit, albedo * (0.1 + 0.9 * sample(grid, dx / rad, dy / rad)), tex)
        zn = z + torch.randn(z.shape, **dev) * (1.5e-3 * z * z)
        zn = torch.where(torch.rand(z.shape, **dev) < 0.02, torch.zeros_like(z), zn)
        out.append(((tex * 255).round().clamp(0, 255).to(torch.uint8), (zn * 5000).round().clamp(0, 32767).to(
            torch.int16)))
    return out


def _host(frame):
    """(uint8, uint16) host arrays of a device frame, as a camera driver or a PNG decoder returns them."""
    return frame[0].cpu().numpy(), frame[1].cpu().numpy().view(np.uint16)


def _rgb(frame):
    """RGB888 and millimetre depth of a device frame (one pair), as a live camera returns them."""
    i, z = frame[0][0].float(), frame[1][0].float()
    rgb = torch.stack((0.9 * i, i, 0.8 * i), -1).round().to(torch.uint8)
    return rgb.cpu().numpy(), (z / 5).round().to(torch.int16).cpu().numpy().view(np.uint16)


def _staging(frame):
    """The reference's float staging buffers of one frame: column-major intensity and metres."""
    i, z = _host((frame[0][0], frame[1][0]))
    return (np.ascontiguousarray(i.T).astype(np.float32).ravel(),
            (np.ascontiguousarray(z.T).astype(np.float32) * np.float32(1.0 / 5000.0)).ravel())


def _schedule(rows, finest):
    """Iterations per level, coarsest first: `finest` at the finest level, 15 fewer per coarser one."""
    levels = (rows // 15).bit_length()
    return [max(5, finest - 15 * (levels - 1 - i)) for i in range(levels)]


def _params(case):
    p = pdflow.default_params(case["rows"])
    for i, n in enumerate(_schedule(case["rows"], case["finest"])):
        p.num_max_iter[i] = n
    return p


def _mixed_rows(case):
    """The pairs' rows, resolutions interleaved as requests arrive."""
    left = {480: case["n480"], 240: case["n240"], 120: case["n120"], 60: case["n60"]}
    rows = []
    while any(left.values()):
        for r in left:
            if left[r]:
                rows.append(r)
                left[r] -= 1
    return rows


def _mixed_frames(case, seed):
    """Frames (intensity, depth) of every pair of a mixed batch: 640x480 for rows 480, 320x240 otherwise."""
    rows = _mixed_rows(case)
    big, small = sum(r == 480 for r in rows), sum(r != 480 for r in rows)
    sets = {True: _frames(big, 640, case["objects"], seed) if big else None,
            False: _frames(small, 320, case["objects"], seed) if small else None}
    at, pick = {True: 0, False: 0}, []
    for r in rows:
        pick.append((r == 480, at[r == 480]))
        at[r == 480] += 1
    return rows, [[(sets[b][k][0][q], sets[b][k][1][q]) for b, q in pick] for k in range(2)]


def _net_data(case, seed):
    """Network inputs [n, 4, 4800] (both frames' 60x80 intensity and depth) and labels [n, 3, 4800]."""
    n = case["n"]
    (i1, z1), (i2, z2) = _frames(n, 320, case["objects"], seed)
    small = lambda a: a[:, 2::4, 2::4].float().transpose(1, 2).reshape(n, 4800)  # noqa: E731
    x = torch.stack((small(i1), small(i2), small(z1) * 2e-4, small(z2) * 2e-4), 1).contiguous()
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 7)
    coarse = torch.randn(n, 3, 8, 6, generator=g, device="cuda")
    flow = F.interpolate(coarse, size=(80, 60), mode="bicubic", align_corners=False).reshape(n, 3, 4800)
    return x, (flow * torch.tensor([0.5, 0.5, 0.02], device="cuda").view(1, 3, 1)).contiguous()


# ---------------------------------------------------------------------------
# A pass
# ---------------------------------------------------------------------------
_stream = None


def _work_stream():
    """The one compute stream of the program, given to every handle it makes."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def _ok(status):
    if status != pdflow.OK:
        raise pdflow.PDFlowError(status, "a call of the C interface")


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind == "net":
        st["net"] = pdflow.Net(case["n"])
        st["net"].set_params(pdflow.load_weights())
        st["x"], st["label"] = _net_data(case, seed)
        return st
    if kind == "mixed":
        rows, frames = _mixed_frames(case, seed)
        st["rows"] = rows
        st["frames"] = [([_host(f)[0] for f in fs], [_host(f)[1] for f in fs]) for fs in frames]
        st["solver"] = pdflow.MixedBatch(len(rows))
        return st
    rows, width, height = case["rows"], case["width"], case["width"] * 3 // 4
    n = case.get("n", 1)
    frames = _frames(n, width, case["objects"], seed)
    if kind == "pair":
        form = {"u16": lambda f: tuple(a[0] for a in _host(f)), "float": _staging, "rgb": _rgb}[case["input"]]
        st["frames"] = [form(f) for f in frames]
        st["solver"] = pdflow.Solver(rows, width, height, _params(case)).initializeCUDA()
    elif kind == "slots":
        st["frames"] = [_host(f) for f in frames]
        st["solver"] = pdflow.BatchSolver(rows, width, height, n, _params(case))
    else:
        params = _params(case) if kind == "batch" else None
        st["frames"] = frames
        st["solver"] = pdflow.BatchSolver(rows, width, height, n, params)
        _ok(pdflow.load().pdflow_set_stream(st["solver"].handle, _work_stream().cuda_stream))
        st["out"] = [torch.empty(n, rows * (rows * 4 // 3), device="cuda") for _ in range(3)]
        if kind == "learned":
            st["net"] = pdflow.Net(n)
            st["net"].set_params(pdflow.load_weights())
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "net":
        loss, grads = st["net"].gradients(case["n"], st["x"].data_ptr(), st["label"].data_ptr())
        return dict(loss=loss, grads=grads)
    s, n = st["solver"], case.get("n", 1)
    if kind == "pair":
        push = {"u16": s.push_raw, "float": s.createImagePyramidGPU, "rgb": s.push_rgb}[case["input"]]
        for frame in st["frames"]:
            push(*frame)
        s.solveSceneFlowGPU()
        return dict(dx=s.dxp, dy=s.dyp, dz=s.dzp)
    if kind == "slots":
        slots = list(range(n))
        for intensity, depth in st["frames"]:
            s.push_slots(slots, intensity, depth)
        s.solve_slots(slots)
        return dict(zip(("dx", "dy", "dz"), s.read_flow_slots(slots)))
    if kind == "mixed":
        for intensity, depth in st["frames"]:
            s.push(st["rows"], intensity, depth)
        s.solve()
        flows = [s.flow(k) for k in range(len(st["rows"]))]
        return {a: np.concatenate([f[c] for f in flows]) for c, a in enumerate(("dx", "dy", "dz"))}
    work = _work_stream()
    work.wait_stream(torch.cuda.current_stream())
    for intensity, depth in st["frames"]:
        s.push_raw_device(n, intensity.data_ptr(), depth.data_ptr())
    if kind == "learned":
        s.solve_learned(n, st["net"], case["scale"], 0.01)
    else:
        s.solve(n)
    _ok(pdflow.load().pdflow_copy_flow_device(s.handle, n, *[o.data_ptr() for o in st["out"]]))
    out = dict(zip(("dx", "dy", "dz"), st["out"]))
    if case.get("energy"):
        out["energy"] = s.energy(n)
    torch.cuda.current_stream().wait_stream(work)
    return out


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
# Floating-point operations of one primal-dual iteration at one pixel
# (gradient 14, data term 5, dual update 14, projections 18, divergence 21,
# primal step 15, shrinkage 14, over-relaxation 6).
FLOPS_PER_PIXEL_ITERATION = 107
# Frames in (uint8 + uint16, two of them), three floats of flow out.
BYTES_PER_FRAME_PIXEL = 3
NET_MACS = 9 * (4800 * (8 * 16 + 16 * 16 + 48 * 16 + 16 * 16) + 1200 * (16 * 32 + 32 * 32 + 96 * 32) + 300 * (
    32 * 64 + 64 * 64 + 160 * 64) + 80 * (64 * 96 + 96 * 96))


def _pair_work(rows, width, schedule):
    iters = sum(n * (rows >> (len(schedule) - 1 - i)) ** 2 * 4 // 3 for i, n in enumerate(schedule))
    frames = 2 * width * (width * 3 // 4) * BYTES_PER_FRAME_PIXEL
    return frames + 12 * (rows * rows * 4 // 3), FLOPS_PER_PIXEL_ITERATION * iters


def work(case):
    kind = case["kind"]
    if kind == "net":
        return dict(bytes=case["n"] * 7 * 4800 * 4 + 2 * 4 * 338000, flops=3 * 2 * NET_MACS * case["n"])
    if kind == "mixed":
        each = [_pair_work(r, 640 if r == 480 else 320, _schedule(r, 100)) for r in _mixed_rows(case)]
        return dict(bytes=sum(b for b, _ in each), flops=sum(f for _, f in each))
    schedule = _schedule(case["rows"], case.get("finest", 100))
    if kind == "learned":
        schedule = [m + math.ceil(m * case["scale"]) if i == 2 else math.ceil(m * case["scale"]) if i > 2 else m
                    for i, m in enumerate(schedule)]
    b, f = _pair_work(case["rows"], case["width"], schedule)
    n = case.get("n", 1)
    return dict(bytes=n * b, flops=n * f)


# ---------------------------------------------------------------------------
# The same in 64 bits, from plain torch
# ---------------------------------------------------------------------------
LAMBDA_I, LAMBDA_D, MU, FOVH = 0.04, 0.35, 75.0, math.pi * 62.5 / 180.0
MASK = [m / 16.0 for m in (1, 4, 6, 4, 1)]


def _focal(cols):
    return 2.0 * math.tan(0.5 * FOVH) / cols


def _back(z):
    """Back-projected x and y of a depth image [n, cols, rows]."""
    C, R = z.shape[1:]
    u = (torch.arange(C, device=z.device, dtype=z.dtype) - 0.5 * (C - 1)).view(1, -1, 1)
    v = (torch.arange(R, device=z.device, dtype=z.dtype) - 0.5 * (R - 1)).view(1, 1, -1)
    return u * z * _focal(C), v * z * _focal(C)


def _down(col, dep):
    C, R = col.shape[1] // 2, col.shape[2] // 2
    pc, pd, on = (F.pad(a, (2, 2, 2, 2)) for a in (col, dep, torch.ones_like(col)))
    centre = dep[:, ::2, ::2]
    sc, wc, sd, wd = (torch.zeros_like(centre) for _ in range(4))
    for l in range(5):
        for k in range(5):
            cut = (slice(None), slice(l, l + 2 * C, 2), slice(k, k + 2 * R, 2))
            gm, d = MASK[l] * MASK[k], pd[cut]
            sc += gm * pc[cut]
            wc += gm * on[cut]
            away = (d - centre).abs()
            w = torch.where((d > 0) & (away < 0.1), gm * (0.1 - away), torch.zeros_like(d))
            wd += w
            sd += w * d
    return sc / wc, torch.where(sd > 0, sd / torch.where(wd > 0, wd, torch.ones_like(wd)), torch.zeros_like(sd))


def _up(coarse, scale):
    n, C, R = coarse.shape
    fine, on = torch.zeros(n, 2 * C, 2 * R, dtype=coarse.dtype, device=coarse.device), None
    fine[:, ::2, ::2] = coarse * scale
    kernel = torch.tensor(MASK, dtype=coarse.dtype, device=coarse.device)
    kernel = (kernel.view(-1, 1) * kernel.view(1, -1)).view(1, 1, 5, 5)
    on = F.conv2d(torch.ones_like(fine[:1]).unsqueeze(1), kernel, padding=2)
    return (F.conv2d(fine.unsqueeze(1), 4 * kernel, padding=2) / on).squeeze(1)


def _diff(a, dim):
    """Forward difference, zero at the far border."""
    d = torch.zeros_like(a)
    m = a.shape[dim] - 1
    d.narrow(dim, 0, m).copy_(a.narrow(dim, 1, m) - a.narrow(dim, 0, m))
    return d


def _back_diff(a, dim):
    """Adjoint of _diff, negated: a without its last entry, minus its neighbour."""
    m = a.shape[dim] - 1
    d = a.clone()
    d.narrow(dim, m, 1).zero_()
    d.narrow(dim, 1, m).sub_(a.narrow(dim, 0, m))
    return d


def _weights(xx, yy, z):
    out = []
    for a, dim in ((xx, 1), (yy, 2)):
        da, dz = _diff(a, dim), _diff(z, dim)
        norm = torch.hypot(da, dz)
        out.append(torch.where(norm > 0, 2.0 / torch.where(norm > 0, norm, torch.ones_like(norm)),
                               torch.ones_like(norm)))
    return out


def _gradient(a, r, dim, holes):
    """Connectivity-weighted central difference; plain at the borders; zero in depth holes."""
    m = a.shape[dim] - 1
    d = a.narrow(dim, 1, m) - a.narrow(dim, 0, m)
    w = r.narrow(dim, 0, m)
    out = torch.empty_like(a)
    mid = (w.narrow(dim, 1, m - 1) * d.narrow(dim, 1, m - 1) + w.narrow(dim, 0, m - 1) * d.narrow(dim, 0, m - 1)) / (
        w.narrow(dim, 1, m - 1) + w.narrow(dim, 0, m - 1))
    if holes:
        mid = torch.where(a.narrow(dim, 1, m - 1) > 0, mid, torch.zeros_like(mid))
    out.narrow(dim, 1, m - 1).copy_(mid)
    out.narrow(dim, 0, 1).copy_(d.narrow(dim, 0, 1))
    out.narrow(dim, m, 1).copy_(d.narrow(dim, m - 1, 1))
    return out


def _warp(o, new, ri2, rj2, du, dv):
    """Both frames at the flow (du, dv): the data terms and their weight."""
    col, dep = new
    n, C, R = col.shape
    grads = [_gradient(col, ri2, 1, False), _gradient(col, rj2, 2, False), _gradient(dep, ri2, 1, True),
             _gradient(dep, rj2, 2, True)]
    u = (torch.arange(C, device=col.device, dtype=col.dtype).view(1, -1, 1) + du).clamp(0, C - 1)
    v = (torch.arange(R, device=col.device, dtype=col.dtype).view(1, 1, -1) + dv).clamp(0, R - 1)
    fu, fv, su, sv = u.floor(), v.floor(), u.ceil(), v.ceil()
    wu, wv = u - fu, v - fv
    at = [(b + R * a).long().view(n, -1) for a in (fu, su) for b in (fv, sv)]
    take = lambda m, i: torch.gather(m.reshape(n, -1), 1, i).view(n, C, R)  # noqa: E731

    def blend(m):
        a, b, c, d = (take(m, i) for i in at)
        return (1 - wu) * ((1 - wv) * a + wv * b) + wu * ((1 - wv) * c + wv * d)

    dct = blend(col) - o[0]
    dcu, dcv, ddu, ddv = (blend(g) for g in grads)
    hole = torch.zeros_like(dep, dtype=torch.bool)
    for i in at:
        hole |= take(dep, i) == 0
    near = take(dep, (v.round() + R * u.round()).long().view(n, -1))
    wz = torch.where(hole, near, blend(dep))
    ddt = torch.where(wz > 0, wz - o[1], torch.zeros_like(wz))
    mu = MU / (1000.0 * (ddu * ddu + ddv * ddv + ddt * ddt) + 1.0)
    return dct, dcu, dcv, ddt, ddu, ddv, mu


def _median(z, ddt, planes):
    """Weighted 3x3 median of each plane (weights from depth and depth change; half of the first plane's
    total for all of them); pixels without depth stay as they are."""
    n, C, R = z.shape
    on = torch.ones_like(z)

    def taps(a):
        p = F.pad(a, (1, 1, 1, 1))
        return torch.stack([p[:, 1 + l:1 + l + C, 1 + k:1 + k + R] for k in (-1, 0, 1) for l in (-1, 0, 1)], -1)

    here = taps(on) > 0
    w = torch.where(here, 1.0 / (1.0 + 5.0 * (z.unsqueeze(-1) - taps(z)) ** 2 + 10.0 * taps(ddt) ** 2),
                    torch.zeros((), dtype=z.dtype, device=z.device))
    half, out = None, []
    for a in planes:
        s, order = torch.where(here, taps(a), torch.full((), math.inf, dtype=z.dtype, device=z.device)).sort(
            dim=-1, stable=True)
        cum = torch.gather(w, -1, order).cumsum(-1)
        half = 0.5 * cum[..., -1:] if half is None else half
        k = (half > cum).sum(-1, keepdim=True)
        hi, lo = k.clamp(max=8), (k - 1).clamp(min=0)
        cr, cl, fr, fl = cum.gather(-1, hi), cum.gather(-1, lo), s.gather(-1, hi), s.gather(-1, lo)
        mid = ((cr - half) * fl + (half - cl) * fr) / torch.where(cr > cl, cr - cl, torch.ones_like(cr))
        out.append(torch.where(z > 0, torch.where(k > 0, mid, s[..., :1]).squeeze(-1), a))
    return out


def _disc(a, b):
    m = torch.hypot(a, b).clamp_min(1.0)
    return a / m, b / m


def _solve(frames, rows, schedule, energy=False):
    """Flow (and energy) of decoded frames [(intensity, metres)] * 2, each [n, h, w] in 64 bits."""
    pyr = []
    for i, z in frames:
        levels = [(i.transpose(1, 2).contiguous(), z.transpose(1, 2).contiguous())]
        while levels[-1][0].shape[2] > 15:
            levels.append(_down(*levels[-1]))
        pyr.append(levels)
    top = int(math.log2(pyr[0][0][0].shape[2] // rows))
    sol = None
    for i, iters in enumerate(schedule):
        li = top + len(schedule) - 1 - i
        o, new = pyr[0][li], pyr[1][li]
        zero = torch.zeros_like(o[0])
        if sol is None:
            dup = dvp = zero
            dw, duals = zero, [zero] * 7
        else:
            dup, dvp = _up(sol[0], 2.0), _up(sol[1], 2.0)
            dw, duals = _up(sol[2], 1.0), [_up(p, 1.0) for p in sol[3]]
        xy_o, xy_n = _back(o[1]), _back(new[1])
        ri, rj = _weights(*xy_o, o[1])
        ri2, rj2 = _weights(*xy_n, new[1])
        dct, dcu, dcv, ddt, ddu, ddv, mu = _warp(o, new, ri2, rj2, dup, dvp)
        s_pd = 1.0 / (mu * (1.0 + ddu.abs() + ddv.abs()) + 1e-10)
        su, sv = (0.5 / (LAMBDA_I * r + 1e-10) * LAMBDA_I for r in (ri, rj))
        swu, swv = (0.5 / (LAMBDA_D * r + 1e-10) * LAMBDA_D for r in (ri, rj))
        acc = ri + rj
        acc[:, 1:] += ri[:, :-1]
        acc[:, :, 1:] += rj[:, :, :-1]
        tu, tv = (1.0 / (LAMBDA_I * acc + mu * d.abs() + 1e-10) for d in (ddu, ddv))
        tw = 1.0 / (LAMBDA_D * acc + mu + 1e-10)
        du = dv = ua = va = zero
        wa = dw
        pd, puu, puv, pvu, pvv, pwu, pwv = duals
        a1, b1 = tu * dcu, tv * dcv
        th = a1 * dcu + b1 * dcv
        for _ in range(iters):
            U, V = ua + dup, va + dvp
            pd = (pd + s_pd * mu * (ddt - wa + ddu * ua + ddv * va)).clamp(-1, 1)
            puu, puv = _disc(puu + su * ri * _diff(U, 1), puv + sv * rj * _diff(U, 2))
            pvu, pvv = _disc(pvu + su * ri * _diff(V, 1), pvv + sv * rj * _diff(V, 2))
            pwu, pwv = _disc(pwu + swu * ri * _diff(wa, 1), pwv + swv * rj * _diff(wa, 2))
            du0, dv0, dw0 = du, dv, dw
            du = du - tu * (mu * ddu * pd - LAMBDA_I * (_back_diff(ri * puu, 1) + _back_diff(rj * puv, 2)))
            dv = dv - tv * (mu * ddv * pd - LAMBDA_I * (_back_diff(ri * pvu, 1) + _back_diff(rj * pvv, 2)))
            dw = dw - tw * (-mu * pd - LAMBDA_D * (_back_diff(ri * pwu, 1) + _back_diff(rj * pwv, 2)))
            of = dct + dcu * du + dcv * dv
            step = torch.where(of < -th, -torch.ones_like(of), torch.where(of > th, torch.ones_like(of),
                                                                          of / (th + 1e-10)))
            du, dv = du - a1 * step, dv - b1 * step
            ua, va, wa = 2 * du - du0, 2 * dv - dv0, 2 * dw - dw0
        du, dv = du.clamp(-1, 1) + dup, dv.clamp(-1, 1) + dvp
        dw = torch.where(o[1] == 0, zero, dw)
        sol = _median(o[1], ddt, (du, dv, dw)) + [[pd, puu, puv, pvu, pvv, pwu, pwv]]
    du, dv, dw = sol[:3]
    z, n = o[1], o[1].shape[0]
    safe = torch.where(z > 0, z, torch.ones_like(z))
    flow = (dw, z * du * _focal(z.shape[1]) + dw * xy_o[0] / safe, z * dv * _focal(z.shape[1]) + dw * xy_o[1] / safe)
    out = {a: torch.where(z > 0, f, torch.zeros_like(f)).reshape(n, -1) for a, f in zip(("dx", "dy", "dz"), flow)}
    if energy:
        dct, _, _, ddt, _, _, mu = _warp(o, new, ri2, rj2, du, dv)
        tv_ = lambda a: torch.hypot(ri * _diff(a, 1), rj * _diff(a, 2))  # noqa: E731
        e = dct.abs() + mu * (ddt - dw).abs() + LAMBDA_I * (tv_(du) + tv_(dv)) + LAMBDA_D * tv_(dw)
        out["energy"] = e.sum((1, 2))
    return out


def _decoded(frame):
    return frame[0].double(), frame[1].double() / 5000.0


def _network(params, x):
    """The warm-start network's head [n, 3, 80, 60] from inputs [n, 4, 4800]."""
    z = x[:, 2:]
    x = torch.cat((x[:, :2] / 255 - 0.5, torch.where(z > 0, 0.5 * (z - 2.5), torch.full_like(z, -1.5))), 1)
    x = F.pad(x, (0, 0, 0, 4)).view(-1, 8, 80, 60)
    at = 0

    def conv(a, cout, relu=True):
        nonlocal at
        cin = a.shape[1]
        w = params[at:at + cout * 9 * cin].view(cout, 3, 3, cin).permute(0, 3, 1, 2)
        at += cout * 9 * cin
        b = params[at:at + cout]
        at += cout
        y = F.conv2d(a, w, b, padding=1)
        return y.relu() if relu else y

    pool = lambda a: F.avg_pool2d(a, 2, ceil_mode=True)  # noqa: E731
    join = lambda a, b: torch.cat((F.interpolate(a, scale_factor=2.0)[..., :b.shape[2], :b.shape[3]], b), 1)  # noqa: E731
    e1 = conv(conv(x, 16), 16)
    e2 = conv(conv(pool(e1), 32), 32)
    e3 = conv(conv(pool(e2), 64), 64)
    e4 = conv(conv(pool(e3), 96), 96)
    d3 = conv(join(e4, e3), 64)
    d2 = conv(join(d3, e2), 32)
    d1 = conv(join(d2, e1), 16)
    return conv(d1, 3, relu=False)


def _exact_net(case, seed):
    x, label = (a.double() for a in _net_data(case, seed))
    with np.load(os.path.join("pd-flow_gb300", "pdflow", "weights", "warmstart.npz")) as f:
        params = torch.from_numpy(f["params"]).double().cuda().requires_grad_(True)
    head = _network(params, x).reshape(-1, 3, 4800)
    target = label * torch.tensor([1.0, 1.0, 20.0], dtype=torch.float64, device="cuda").view(1, 3, 1)
    valid = (x[:, 2] > 0).unsqueeze(1)
    loss = (((head - target) * valid) ** 2).sum() / (3 * valid.sum())
    loss.backward()
    return dict(loss=float(loss), grads=params.grad)


def exact(case, seed):
    kind = case["kind"]
    if kind == "net":
        return _exact_net(case, seed)
    if kind == "learned":   # its accept / fall back decision per pair hangs on a bf16 network's energies
        return None
    if kind == "mixed":
        rows, frames = _mixed_frames(case, seed)
        got = {}
        for r in sorted(set(rows)):
            ks = [k for k, x in enumerate(rows) if x == r]
            stack = [_decoded([torch.stack([fs[k][c] for k in ks]) for c in range(2)]) for fs in frames]
            flows = _solve(stack, r, _schedule(r, 100))
            for q, k in enumerate(ks):
                got[k] = {a: flows[a][q] for a in flows}
        return {a: torch.cat([got[k][a] for k in range(len(rows))]) for a in ("dx", "dy", "dz")}
    n = case.get("n", 1)
    frames = _frames(n, case["width"], case["objects"], seed)
    if case.get("input") == "rgb":
        rgb = [_rgb(f) for f in frames]
        luma = torch.tensor([0.299, 0.587, 0.114], dtype=torch.float64, device="cuda")
        frames = [(torch.from_numpy(c).cuda().double() @ luma, torch.from_numpy(z.view(np.int16)).cuda().double() * 1e-3)
                  for c, z in rgb]
        frames = [(i.unsqueeze(0), z.unsqueeze(0)) for i, z in frames]
    else:
        frames = [_decoded(f) for f in frames]
    schedule = _schedule(case["rows"], case["finest"])
    parts = [_solve([(i[k:k + 8], z[k:k + 8]) for i, z in frames], case["rows"], schedule, case.get("energy", False))
             for k in range(0, n, 8)]
    out = {a: torch.cat([p[a] for p in parts]) for a in parts[0]}
    return {a: x.reshape(-1) for a, x in out.items()} if kind == "pair" else out
