"""The fused pyramid passes on both sides of the rule that splits them (few or
many pixels a push), for each kind of frame: every level's bits against the
FP32 oracle's images of a single frame's push, pair by pair."""
import numpy as np
import pytest

from pdflow import BatchSolver, Solver, scenes

pytestmark = pytest.mark.gpu


def _levels(width):
    return 6 if width == 640 else 5


@pytest.mark.parametrize("width,n", [(320, 9), (640, 3)])
def test_batched_pushes_equal_single_ones(built_lib, width, n):
    """n frames are above the rule's line (two levels in the first pass), one
    frame below it (three): same bits at every level, through the flow of the
    smallest solve, which reads them all."""
    h = width * 3 // 4
    frames = [scenes.make_pair(90 + k, vga=width == 640) for k in range(n)]
    b = BatchSolver(15, width, h, n)
    for f in (0, 1):
        b.push_raw(np.stack([p[2 * f] for p in frames]), np.stack([p[2 * f + 1] for p in frames]))
    b.solve(n)
    flows = np.stack(b.read_flow(n))
    b.close()
    for k in range(n):
        s = Solver(15, width, h).initializeCUDA()
        s.loadRGBDFrames(*frames[k])
        s.solveSceneFlowGPU()
        one = np.stack([s.dxp, s.dyp, s.dzp])
        assert np.array_equal(one.view(np.uint32), flows[:, k].view(np.uint32)), k
        s.freeGPUMemory()


@pytest.mark.parametrize("width", [320, 640])
def test_frame_kinds_give_the_same_pyramid(built_lib, width):
    """uint16 frames and the float staging buffers of the same images: bit-equal
    levels; and level l + 1 against a plain numpy 5x5 average of level l's
    intensity away from the borders (weights exact in binary; the kernel's
    serial FP32 sum of 25 products is off by at most 25 ulp of 255)."""
    h = width * 3 // 4
    i1, z1, _, _ = scenes.make_pair(5, vga=width == 640)
    a, b = Solver(15, width, h).initializeCUDA(), Solver(15, width, h).initializeCUDA()
    a.push_raw(i1, z1)
    b.createImagePyramidGPU(*scenes.decode(i1, z1))
    m = np.array([1, 4, 6, 4, 1], np.float64) / 16
    prev = None
    for level in range(_levels(width)):
        x, y = a.level_images(level, 1), b.level_images(level, 1)
        for k in x:
            assert np.array_equal(x[k].view(np.uint32), y[k].view(np.uint32)), (level, k)
        c = x["colour"].reshape(width >> level, h >> level).astype(np.float64)
        if prev is not None:
            C, R = c.shape
            p = sum(m[i] * m[j] * prev[i:i + 2 * (C - 2):2, j:j + 2 * (R - 2):2] for i in range(5) for j in range(5))
            assert np.abs(c[1:C - 1, 1:R - 1] - p).max() <= 25 * 255 * 2.0 ** -24
        prev = c
    a.freeGPUMemory()
    b.freeGPUMemory()


def _images(handle, width, level):
    from pdflow._lib import check, load
    out = [np.zeros((width >> level) * (width * 3 // 4 >> level), np.float32) for _ in range(4)]
    check(load().pdflow_read_level_images(handle, level, 1, *[a.ctypes.data for a in out]), "level images")
    return out


@pytest.mark.parametrize("width,n", [(320, 1), (320, 9), (640, 1), (640, 3)])
def test_every_level_against_the_oracle(built_lib, width, n):
    """Each level's four planes (of pair 0, on either side of the rule) against the
    FP32 oracle's step from the level above as the GPU left it.  The oracle rounds a
    product where the kernel fuses it: a 25-term sum of intensities up to 255 differs
    by at most 2 * 25 * 255 * 2^-24, a depth (same weights, a fused numerator, one
    division) by 2 * 27 * 2^-24 of itself, its back-projections by 10 * 2^-24 more
    (four products, a tangent and a division)."""
    from oracle import oracle
    h = width * 3 // 4
    frames = [scenes.make_pair(70 + k, vga=width == 640)[:2] for k in range(n)]
    b = BatchSolver(15, width, h, n)
    b.push_raw(np.stack([f[0] for f in frames]), np.stack([f[1] for f in frames]))
    mask = np.array([1, 4, 6, 4, 1], np.float32)
    g = np.ascontiguousarray(np.outer(mask, mask) / np.float32(256), np.float32).ravel()
    above = [np.ascontiguousarray(a, np.float32).ravel() for a in scenes.decode(*frames[0])]
    for level in range(_levels(width)):
        C, R = width >> level, h >> level
        want = [np.zeros(R * C, np.float32) for _ in range(4)]
        src = (*above, None, None) if level == 0 else (None, None, *above)
        oracle.stage_call("pyramid_level", "f32", R, C, level == 0, *src, g, float(np.float32(np.pi * 62.5 / 180)), *want)
        got = _images(b.handle, width, level)
        eps = 2.0 ** -24
        assert np.abs(got[0].astype(np.float64) - want[0]).max() <= 2 * 25 * 255 * eps, level
        for k, ulps in ((1, 54), (2, 64), (3, 64)):
            away = np.abs(got[k].astype(np.float64) - want[k])
            assert np.all(away <= ulps * eps * np.abs(want[k])), (level, k)
        above = [got[0], got[1]]
    b.close()


@pytest.mark.parametrize("width,rows,n", [(320, 240, 9), (640, 480, 3)])
def test_batched_pushes_solved_at_full_resolution(built_lib, width, rows, n):
    """A solve at the image's resolution reads all four planes of every level of both
    frames: each pair of the batch (two levels in the first pass) has the bits of a
    single pair's solve (three)."""
    h = width * 3 // 4
    frames = [scenes.make_pair(190 + k, vga=width == 640) for k in range(n)]
    b = BatchSolver(rows, width, h, n)
    for f in (0, 1):
        b.push_raw(np.stack([p[2 * f] for p in frames]), np.stack([p[2 * f + 1] for p in frames]))
    b.solve(n)
    flows = np.stack(b.read_flow(n))
    b.close()
    for k in range(n):
        s = Solver(rows, width, h).initializeCUDA()
        s.loadRGBDFrames(*frames[k])
        s.solveSceneFlowGPU()
        one = np.stack([s.dxp, s.dyp, s.dzp])
        assert np.array_equal(one.view(np.uint32), flows[:, k].view(np.uint32)), k
        s.freeGPUMemory()
