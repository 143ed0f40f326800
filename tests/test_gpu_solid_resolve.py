"""The resolve passes of solid voxelization against numpy, on meshes whose result is known exactly.

The mesh is a set of axis-aligned boxes with faces a quarter voxel past integer coordinates on a
unit grid, so that no column centre and no x crossing is near a decision boundary: box
(x0, y0, z0) .. (x1, y1, z1) flips exactly the voxels x0 <= x < x1, y0 <= y < y1, z0 <= z < z1.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from cuda_voxelizer_gb300 import api as cv  # noqa: E402

pytestmark = pytest.mark.gpu

GUARD = 64


def _boxes(grid, seed, n=12):
    rng = np.random.default_rng(seed)
    g = np.asarray(grid)
    out = []
    for _ in range(n):
        a, b = rng.integers(0, g, 3), rng.integers(0, g, 3)
        out.append((np.minimum(a, b), np.maximum(a, b) + 1))
    out.append((np.zeros(3, int), g.copy()))         # the whole grid: rows that stay set to their end
    out.append((np.array([g[0] // 2, 0, 0]), g.copy()))
    return [(lo, np.minimum(hi, g)) for lo, hi in out]


def _mesh(boxes, grid):
    """Two x faces per box (the other faces hold no column's x crossing), two triangles each."""
    tris = []
    for lo, hi in boxes:
        y0, z0, y1, z1 = lo[1] + 0.25, lo[2] + 0.25, hi[1] + 0.25, hi[2] + 0.25
        for x in (lo[0], hi[0]):
            if x == 0:
                continue  # no voxel below it
            p = [(x + 0.25, y, z) for y, z in ((y0, z0), (y1, z0), (y1, z1), (y0, z1))]
            tris += [p[0] + p[1] + p[2], p[0] + p[2] + p[3]]
    return np.array(tris, dtype=np.float32)


def _want(boxes, grid, morton):
    v = np.zeros((grid[2], grid[1], grid[0]), dtype=np.uint8)
    for lo, hi in boxes:
        v[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]] ^= 1
    bits = v.reshape(-1)
    if morton:
        c = np.arange(grid[0], dtype=np.int64)
        s = sum(((c >> i) & 1) << (3 * i) for i in range(11))
        code = (s[None, None, :] | s[None, :, None] << 1 | s[:, None, None] << 2).reshape(-1)
        out = np.empty_like(bits)
        out[code] = bits
        bits = out
    return np.packbits(np.concatenate([bits, np.zeros(-len(bits) % 32, np.uint8)])).view(np.uint32).byteswap()


def _run(grid, morton, offset, plan, seed):
    boxes = _boxes(grid, seed)
    tris = _mesh(boxes, grid)
    info = cv.make_info((0, 0, 0), [float(x) for x in grid], grid, len(tris))
    words = cv.table_words(info)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    buf = torch.randint(-2 ** 31, 2 ** 31 - 1, (words + GUARD,), dtype=torch.int32, device="cuda", generator=gen)
    before = buf.cpu().numpy().view(np.uint32)
    table = buf[offset:offset + words]
    d = torch.from_numpy(tris.reshape(-1)).cuda()
    want = _want(boxes, grid, morton)
    if plan:  # the engine owns the table: every word is stored
        p = cv.Plan([cv.Job(info, d, table, morton, True)], clear_tables=True)
        p.launch()
        p.launch()
        torch.cuda.synchronize()
        p.close()
    else:     # XORed into what the caller left there
        cv.voxelize_solid(info, d, table, morton)
        want = want ^ before[offset:offset + words]
    cv.device_status()
    after = buf.cpu().numpy().view(np.uint32)
    assert np.array_equal(after[offset:offset + words], want)
    assert np.array_equal(after[:offset], before[:offset])
    assert np.array_equal(after[offset + words:], before[offset + words:])


@pytest.mark.parametrize("plan", [False, True])
@pytest.mark.parametrize("offset", [0, 1])  # 1: a table that is not 16-byte aligned
@pytest.mark.parametrize("g", [4, 16, 32, 64, 128, 256, 512])
def test_morton(g, offset, plan):
    _run((g, g, g), True, offset, plan, g + offset)


def test_morton_2048_beyond_one_kilovoxel_axis():
    """More than 32 words per row; checked against the linear table of the same boxes."""
    g = 2048
    boxes = _boxes((g, g, g), 5, n=4)
    tris = _mesh(boxes, (g, g, g))
    info = cv.make_info((0, 0, 0), (float(g),) * 3, g, len(tris))
    d = torch.from_numpy(tris.reshape(-1)).cuda()
    lin = torch.zeros(cv.table_words(info), dtype=torch.int32, device="cuda")
    mor = torch.zeros_like(lin)
    cv.voxelize_solid(info, d, lin, False)
    cv.voxelize_solid(info, d, mor, True)
    assert torch.equal(cv.transcode(mor, g, False), lin)
    for (lo, hi) in boxes[:2]:  # spot checks of the linear table: the parity of the boxes over a voxel
        for p in ((lo + hi) // 2, lo, hi - 1):
            bit = int(p[0] + g * (p[1] + g * p[2]))
            word = int(lin[bit >> 5].item()) & 0xFFFFFFFF
            inside = sum(bool(np.all(p >= a) and np.all(p < b)) for a, b in boxes)
            assert (word >> (31 - (bit & 31))) & 1 == inside & 1


@pytest.mark.parametrize("plan", [False, True])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("grid", [
    (1, 40, 30), (3, 33, 65), (7, 50, 41), (31, 64, 64),        # several rows per word
    (32, 40, 24), (64, 96, 80), (96, 20, 50), (160, 33, 9),     # rows on word boundaries
    (33, 64, 64), (100, 100, 100), (250, 31, 77), (500, 40, 41),  # rows that begin inside words
    (4096, 9, 7), (5000, 5, 6), (4100, 7, 5),                   # rows longer than a warp's words
    (500, 300, 240),                                            # a table with long units
])
def test_linear(grid, offset, plan):
    _run(grid, False, offset, plan, sum(grid) + offset)


@pytest.mark.parametrize("plan", [False, True])
@pytest.mark.parametrize("offset", [0, 1])  # 1: not 16-byte aligned, so not by lane
@pytest.mark.parametrize("grid", [(128, 7, 5), (128, 32, 32), (256, 31, 33), (384, 13, 5), (512, 64, 40), (640, 11, 3),
                                  (768, 11, 3), (128, 1, 1), (640, 32, 1)])
def test_linear_rows_by_lane(grid, offset, plan):
    """Rows of 16-byte groups, up to the longest one that a lane walks by itself and beyond it."""
    _run(grid, False, offset, plan, sum(grid) + offset)


@pytest.mark.parametrize("n_boxes", [1, 40, 700])  # x faces: a partial warp, a few tiles, a grid that fills the chip
@pytest.mark.parametrize("extent", [1, 4, 5, 11, 12, 16, 17])  # columns: 1, 16 | 25, 121 | 144, 256 | 289
def test_columns_per_triangle(n_boxes, extent):
    """Column counts around each bin's edge (16 and 128 columns in the classify kernel, 256 per queued
    item), in launches on both sides of the rule on the number of tiles."""
    g = 96
    rng = np.random.default_rng(extent)
    n = n_boxes * (32 if n_boxes == 700 else 1)
    lo = rng.integers(0, g - extent + 1, (n, 3))
    size = np.stack([rng.integers(1, g, n), np.full(n, extent), np.full(n, extent)], 1)
    boxes = [(a, np.minimum(a + s, g)) for a, s in zip(lo, size)]
    tris = _mesh(boxes, (g, g, g))
    info = cv.make_info((0, 0, 0), (float(g),) * 3, g, len(tris))
    table = torch.zeros(cv.table_words(info), dtype=torch.int32, device="cuda")
    cv.voxelize_solid(info, torch.from_numpy(tris.reshape(-1)).cuda(), table, False)
    cv.device_status()
    assert np.array_equal(table.cpu().numpy().view(np.uint32), _want(boxes, (g, g, g), False))


def test_more_than_2_to_the_27_resolve_units():
    """A table of 64 GiB in units of 128 words: the first and the last rows, and nothing else, hold their solids."""
    g = (128, 1 << 21, (1 << 11) + 4)
    words = g[0] // 32 * g[1] * g[2]
    if torch.cuda.mem_get_info()[0] < 2 * 4 * words + (8 << 30):
        pytest.skip("needs 140 GiB of device memory")
    tris, rows = [], []
    for z in (1, g[2] - 3):  # a quad in the plane x = 64 over 10 x 2 columns
        a, b, c, d = ([64.25, y, w] for y, w in ((10, z), (20, z), (20, z + 2), (10, z + 2)))
        tris += [a + b + c, a + c + d]
        rows += [y + (z + k) * g[1] for k in range(2) for y in range(10, 20)]
    info = cv.make_info((0, 0, 0), [float(n) for n in g], g, len(tris))
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        table = torch.zeros(words, dtype=torch.int32, device="cuda")
        cv.voxelize_solid(info, torch.tensor(tris, dtype=torch.float32, device="cuda").reshape(-1), table)
        cv.device_status(stream)
        got = torch.stack([table[4 * r:4 * r + 4] for r in rows]).cpu().numpy().view(np.uint32)
        n = sum(int(torch.count_nonzero(part)) for part in table.split(1 << 28))
    del table
    cv.stream_release(stream)
    torch.cuda.empty_cache()
    assert (got == np.array([0xFFFFFFFF, 0xFFFFFFFF, 0, 0], dtype=np.uint32)).all()
    assert n == 2 * len(rows)
