"""The surface classify kernel's bins and launch shapes, against the CPU oracle's GPU-arithmetic mode.

Each mesh is made of triangles whose grid boxes sit on both sides of a bin's edge (voxels per row,
rows per triangle, extents), in numbers on both sides of the rules on the number of tiles, and in
groups that are ragged or not 16-byte aligned.  The tables must be equal, bit for bit.
"""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
from cuda_voxelizer_gb300 import api as cv  # noqa: E402
from oracle import build as oracle_build  # noqa: E402

pytestmark = pytest.mark.gpu

GUARD = 64


@pytest.fixture(scope="module")
def rsqrt():
    """The device's own rsqrtf, which the oracle needs for the normals."""
    L = ctypes.CDLL(oracle_build.build_gpu_runner())
    L.refgpu_rsqrt.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_void_p]

    def f(x):
        a = torch.from_numpy(x).cuda()
        b = torch.empty_like(a)
        assert L.refgpu_rsqrt(a.data_ptr(), b.data_ptr(), a.numel(), torch.cuda.current_stream().cuda_stream) == 0
        return np.ascontiguousarray(b.cpu().numpy())

    return f


def _triangles(seed, n, ext, g):
    """n random triangles, each spanning about ext[k] voxels along axis k of a unit grid of g voxels."""
    rng = np.random.default_rng(seed)
    ext = np.minimum(np.asarray(ext, dtype=np.float64), g - 1.0)
    t = rng.random((n, 3, 3))
    t = (t - t.min(1, keepdims=True)) / (t.max(1, keepdims=True) - t.min(1, keepdims=True))
    lo = rng.uniform(0.3, g - ext - 0.3, (n, 3))
    return (lo[:, None, :] + t * ext).reshape(n, 9).astype(np.float32)


def _check(rsqrt, tris, g, morton, offset=0):
    info = cv.make_info((0, 0, 0), (float(g),) * 3, g, len(tris))
    buf = torch.zeros(tris.size + 4, dtype=torch.float32, device="cuda")
    d = buf[offset:offset + tris.size]
    d.copy_(torch.from_numpy(tris.reshape(-1)))
    table = torch.zeros(cv.table_words(info) + GUARD, dtype=torch.int32, device="cuda")
    cv.voxelize(info, d, table, morton)
    cv.device_status()
    inv = rsqrt(oracle.len2(bytes(info), tris, oracle.gpu_mode(morton)))
    want = oracle.voxelize(bytes(info), tris, morton, mode=oracle.gpu_mode(morton, inv_len=inv))
    got = table.cpu().numpy().view(np.uint32)
    assert not got[len(want):].any()
    bad = np.nonzero(got[:len(want)] != want)[0]
    assert bad.size == 0, f"{bad.size} words differ, first {bad[:5]}"


@pytest.mark.parametrize("morton", [False, True])
@pytest.mark.parametrize("ext", [
    (0.4, 0.4, 0.4), (2.5, 2.5, 2.5), (15, 3, 3), (16, 3, 3), (17, 3, 3),   # rows of up to and above 16 voxels
    (40, 0.3, 0.3), (63, 0.2, 0.2),                                          # few voxels, all in one or two rows
    (3, 14, 14), (3, 16, 16), (3, 20, 20),                                   # rows around 256
    (2, 254, 0.3), (2, 256, 0.3), (2, 0.3, 256), (255, 2, 2), (257, 2, 2),   # extents around 256
    (60, 60, 31), (60, 60, 33),                                              # around one queue item per triangle
])
def test_bins(rsqrt, ext, morton):
    _check(rsqrt, _triangles(7, 301, ext, 512), 512, morton)


@pytest.mark.parametrize("n", [1, 3, 4, 5, 31, 33, 127, 129, 8500, 17100, 34100, 68200, 136300])
def test_launch_shapes(rsqrt, n):
    """Ragged groups, and triangles per warp of 4, 8, 16 and 32 (the last from about 900 tiles of 128 on)."""
    _check(rsqrt, _triangles(n, n, (4, 4, 4), 128), 128, False)


@pytest.mark.parametrize("n", [130, 140_001])
@pytest.mark.parametrize("offset", [1, 2])  # floats past a 16-byte boundary: no bulk copy
def test_unaligned_triangles(rsqrt, n, offset):
    _check(rsqrt, _triangles(n, n, (3, 3, 3), 128), 128, True, offset)


@pytest.mark.parametrize("n", [200, 140_000])
def test_mixed_sizes(rsqrt, n):
    """Warps that hold a few large triangles among small ones, and more rows than a small launch keeps."""
    t = _triangles(1, n, (2, 2, 2), 256)
    t[::37] = _triangles(2, len(t[::37]), (9, 15, 15), 256)
    t[::411] = _triangles(3, len(t[::411]), (90, 90, 90), 256)
    _check(rsqrt, t, 256, False)


@pytest.mark.parametrize("ext,morton", [((3, 2.4, 2.4), False), ((3, 2.6, 2.6), True), ((14, 7, 7), False), ((2, 61, 0.3), True)])
def test_collected_rows(rsqrt, ext, morton):
    """Warps of 32 triangles with about 384 rows, where rows that pass are collected, and with up to 64 rows each."""
    t = _triangles(13, 120_003, ext, 256)
    t[40_000:80_000] = _triangles(14, 40_000, (2, 1.2, 1.2), 256)  # warps with few rows
    _check(rsqrt, t, 256, morton)


@pytest.mark.parametrize("n_large,g", [(1, 640), (31, 640), (3_000, 640), (60_000, 640), (60_000, 200), (61_000, 448)])
def test_queued_items_in_a_large_launch(rsqrt, n_large, g):
    """Queues from less than one item per warp to several per claim, of triangles with one item and with more, on
    both sides of the rule on the grid's faces."""
    t = _triangles(21, 70_001, (1, 1, 1), g)
    t[:n_large] = _triangles(22, n_large, (12, 9, 9), g)
    t[:n_large:7] = _triangles(23, len(t[:n_large:7]), (5, 4, 70), g)
    _check(rsqrt, t, g, False)


@pytest.mark.parametrize("n", [400, 60_000])
def test_large_queued_items_in_a_large_launch(rsqrt, n):
    """The same with more items of large triangles than of others."""
    t = _triangles(24, 60_001, (1, 1, 1), 512)
    t[:n] = _triangles(25, n, (4, 9, 140), 512)
    _check(rsqrt, t, 512, True)


def test_grid_aligned_triangles(rsqrt):
    """Vertices on voxel corners: plane offsets that are exactly zero, and degenerate triangles."""
    rng = np.random.default_rng(11)
    lo = rng.integers(1, 50, (4000, 1, 3))
    t = (lo + rng.integers(0, 6, (4000, 3, 3))).astype(np.float32)
    t[::3, :, 0] = t[::3, :1, 0]  # in a plane of constant x, y or z
    t[1::3, :, 1] = t[1::3, :1, 1]
    t[2::3, :, 2] = t[2::3, :1, 2]
    _check(rsqrt, t.reshape(-1, 9), 64, False)


@pytest.mark.parametrize("morton", [False, True])
@pytest.mark.parametrize("ext", [
    (100, 120, 31), (100, 120, 33), (100, 129, 70), (20, 300, 40), (1, 200, 200),  # windows of 128 y, items of 32 z
    (300, 200, 1), (300, 1, 200), (400, 0.5, 0.5), (0.2, 300, 300),                # one row of y or z, thin in x
])
def test_large_triangles(rsqrt, ext, morton):
    _check(rsqrt, _triangles(5, 60, ext, 512), 512, morton)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("tilt", [0.0, 1e-6, 1e-4, 1e-2])
def test_large_triangles_nearly_parallel_to_an_axis(rsqrt, axis, tilt):
    """Edges and planes whose tests hardly depend on a coordinate: estimates that are not good enough."""
    rng = np.random.default_rng(axis)
    t = _triangles(9, 80, (200, 200, 200), 256).reshape(-1, 3, 3)
    t[:40, :, axis] = t[:40, :1, axis] + tilt * rng.uniform(-1, 1, (40, 3))        # the plane
    t[40:, 1, axis] = t[40:, 0, axis] + tilt * rng.uniform(-1, 1, 40)              # one edge
    _check(rsqrt, t.reshape(-1, 9).astype(np.float32), 256, False)


@pytest.mark.parametrize("morton", [False, True])
@pytest.mark.parametrize("g", [2, 8, 32])
@pytest.mark.parametrize("extra", [0, 1, 5000])
def test_many_triangles_per_word(rsqrt, g, morton, extra):
    """Around three triangles per voxel of the grid, where rows are tested against the table before the atomic."""
    n = 3 * g ** 3 + extra
    t = _triangles(g, n, (0.6, 0.6, 0.6) if extra < 5000 else (1.5, 1.5, 1.5), g)
    if g == 32:
        t = t[np.lexsort(np.floor(t[:, :3]).T)]  # neighbours in space next to each other
    _check(rsqrt, t, g, morton)


def test_dense_and_sparse_jobs_in_one_plan():
    """A plan with jobs on both sides of the rule writes the tables of its jobs one by one."""
    rng = np.random.default_rng(4)
    metas = [(16, 13_000, False), (64, 900, False), (33, 120_000, False), (16, 12_000, True), (32, 100_000, True)]
    jobs, alone = [], []
    for g, n, morton in metas:
        tris = _triangles(rng.integers(1 << 30), n, (1, 1, 1), g)
        info = cv.make_info((0, 0, 0), (float(g),) * 3, g, n)
        d = torch.from_numpy(tris.reshape(-1)).cuda()
        one, many = (torch.zeros(cv.table_words(info), dtype=torch.int32, device="cuda") for _ in range(2))
        cv.voxelize(info, d, one, morton)
        alone.append(one)
        jobs.append(cv.Job(info, d, many, morton))
    plan = cv.Plan(jobs, clear_tables=True)
    for _ in range(2):
        plan.launch()
    torch.cuda.synchronize()
    for one, job in zip(alone, jobs):
        assert torch.equal(one, job.table)


def _check_info(rsqrt, tris, info, morton=False):
    d = torch.from_numpy(np.ascontiguousarray(tris).reshape(-1)).cuda()
    table = torch.zeros(cv.table_words(info) + GUARD, dtype=torch.int32, device="cuda")
    cv.voxelize(info, d, table, morton)
    cv.device_status()
    inv = rsqrt(oracle.len2(bytes(info), tris, oracle.gpu_mode(morton)))
    want = oracle.voxelize(bytes(info), tris, morton, mode=oracle.gpu_mode(morton, inv_len=inv))
    got = table.cpu().numpy().view(np.uint32)
    assert not got[len(want):].any()
    bad = np.nonzero(got[:len(want)] != want)[0]
    assert bad.size == 0, f"{bad.size} words differ, first {bad[:5]}"


def _floor(seed, n, ext, g, height, tilt=0.0):
    """n random triangles of about ext voxels along x and y in the plane z = height + tilt * x."""
    t = _triangles(seed, n, (ext, ext, 0.0 if ext < 1 else 1.0), g).reshape(n, 3, 3).astype(np.float64)
    t[:, :, 2] = height + tilt * t[:, :, 0]
    return t.reshape(n, 9).astype(np.float32)


@pytest.mark.parametrize("height", [0.0, 1e-16])
@pytest.mark.parametrize("n", [300, 70_001])
def test_floor_of_a_wide_flat_grid(rsqrt, n, height):
    """Offsets of the plane test that are zero or tiny, where 32 bits hold a row's place but not that of 16 slices on."""
    t = _floor(n, n, 2.5, 16384, height)
    t[:150] = _floor(1, 150, 24, 16384, height)   # fewer rows than an item of 32 slices may have in a small launch
    t[150:300] = _floor(2, 150, 120, 16384, height)
    _check_info(rsqrt, t, cv.make_info((0, 0, 0), (16384.0, 16384.0, 4.0), (16384, 16384, 4), n))


@pytest.mark.parametrize("unit", [1.0, 2.0 ** -10, 2.0 ** -40])
@pytest.mark.parametrize("height,tilt", [(0, 0), (1, 0), (1e-16, 0), (1e-39, 0), (0, 1e-17), (0, -1e-17), (0, -1e-30),
                                         (0, -1e-36), (0, -1e-39)])
def test_products_of_the_plane_test_that_underflow(rsqrt, unit, height, tilt):
    """Planes through, or next to, the corner of the box's first voxels: the product of the plane test's two sums
    underflows where they do not cancel."""
    n, g = 900, 64
    t = np.concatenate([_floor(3, 300, 40, g, height, tilt), _floor(4, 600, 3, g, height, tilt)]).reshape(n, 3, 3)
    t = (t.astype(np.float64) * unit).astype(np.float32)
    for axis in range(3):
        a = np.roll(t, axis, 2)
        a[::2] = a[::2, ::-1]  # both orientations
        _check_info(rsqrt, a.reshape(n, 9), cv.make_info((0, 0, 0), (g * unit,) * 3, g, n), axis == 1)


@pytest.mark.parametrize("unit", [2.0 ** -128, 2.0 ** -129, 1e-37 / 64, 2.0 ** -140])
def test_unit_whose_reciprocal_overflows(rsqrt, unit):
    """Boxes so small that 1 / unit is not finite: the grid boxes come from the divisions."""
    g, n = 64, 400
    t = np.concatenate([_triangles(31, 300, (3, 3, 3), g), _triangles(32, 100, (20, 20, 20), g)])
    t = (t.astype(np.float64) * unit).astype(np.float32)
    _check_info(rsqrt, t, cv.make_info((0, 0, 0), (g * unit,) * 3, g, n))


def _time(info, d, reps=20):
    table = torch.zeros(cv.table_words(info), dtype=torch.int32, device="cuda")
    best = float("inf")
    for _ in range(4):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        for _ in range(reps):
            cv.voxelize(info, d, table)
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) / reps)
    return best


@pytest.mark.parametrize("height,tilt", [(0, 0), (1, 0), (0, 6e-17)])
def test_small_triangles_of_the_first_planes_stay_in_the_classify_kernel(height, tilt):
    """A fine floor in the box's first planes (also one with the rounding noise of a rotation) takes about as long as
    one further up: 1.4 times at most where it was measured, 38 times when its triangles were queued one by one."""
    g = n = 512
    i, j = (a.reshape(-1, 1) for a in np.meshgrid(np.arange(n), np.arange(n), indexing="ij"))
    quad = np.array([[0, 0], [1, 0], [1, 1], [0, 0], [1, 1], [0, 1]])
    t = np.zeros((n * n, 6, 3))
    t[:, :, 0], t[:, :, 1] = i + quad[:, 0], j + quad[:, 1]
    info = cv.make_info((0, 0, 0), (float(g),) * 3, g, 2 * n * n)
    ms = []
    for h, s in ((height, tilt), (3, 0)):
        t[:, :, 2] = h + s * t[:, :, 0]
        ms.append(_time(info, torch.from_numpy(t.astype(np.float32).reshape(-1)).cuda()))
    assert ms[0] < 4 * ms[1], ms


@pytest.mark.parametrize("morton", [False, True])
@pytest.mark.parametrize("ext,n", [
    ((16, 3, 3), 700), ((15.4, 3, 3), 9_000), ((17, 7, 3.5), 9_000), ((17, 8, 3.5), 9_000),  # 16 voxels; around 32 rows
    ((60, 7, 7), 9_000), ((40, 6.2, 5.2), 9_000), ((200, 63, 0.2), 3_000),                   # around as many rows as voxels, 64 rows
    ((500, 2, 2), 2_000), ((509, 1, 1), 2_000),                                              # around 512 voxels
    ((30, 2, 2), 1), ((30, 2, 2), 33), ((30, 2, 2), 130_001),                                # triangles per warp
])
def test_triangles_of_few_long_rows(rsqrt, ext, n, morton):
    _check(rsqrt, _triangles(41, n, ext, 512), 512, morton)


def test_long_rows_beside_all_other_kinds(rsqrt):
    """Queues of all three kinds in one launch, and in a plan of several meshes with different grids."""
    jobs, alone = [], []
    for seed, g, morton in ((1, 640, False), (2, 256, True), (3, 400, False)):
        t = _triangles(seed, 20_011, (1.5, 1.5, 1.5), g)
        t[::7] = _triangles(seed, len(t[::7]), (40, 2, 2), g)
        t[::53] = _triangles(seed, len(t[::53]), (30, 20, 4), g)
        t[::97] = _triangles(seed, len(t[::97]), (20, 30, 90), g)
        _check(rsqrt, t, g, morton)
        info = cv.make_info((0, 0, 0), (float(g),) * 3, g, len(t))
        d = torch.from_numpy(t.reshape(-1)).cuda()
        one, many = (torch.zeros(cv.table_words(info), dtype=torch.int32, device="cuda") for _ in range(2))
        cv.voxelize(info, d, one, morton)
        alone.append(one)
        jobs.append(cv.Job(info, d, many, morton))
    plan = cv.Plan(jobs, clear_tables=True)
    for _ in range(2):
        plan.launch()
    torch.cuda.synchronize()
    for one, job in zip(alone, jobs):
        assert torch.equal(one, job.table)


def test_long_rows_on_a_wide_grid(rsqrt):
    """A grid with an axis much longer than the others, whose voxels are 64 times shorter along it."""
    t = _triangles(51, 9_000, (0.6, 1.2, 1.2), 64)
    _check_info(rsqrt, t, cv.make_info((0, 0, 0), (64.0,) * 3, (4096, 64, 64), len(t)))


def test_rows_of_17_voxels_cost_about_as_much_as_rows_of_15():
    """Many triangles of few rows on both sides of the rule on a row's voxels: as much on both sides where it was
    measured, 4.4 times as much when those of longer rows were items of their own."""
    n, g = 200_000, 512
    info = cv.make_info((0, 0, 0), (float(g),) * 3, g, n)
    ms = [_time(info, torch.from_numpy(_triangles(10, n, (ext, 2, 2), g).reshape(-1)).cuda()) for ext in (14, 17)]
    assert ms[1] < 2.5 * ms[0], ms
