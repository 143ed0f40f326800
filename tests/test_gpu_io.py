"""GPU ingest, layout and output kernels against the reference's writers and the oracle:

* cvx_encode_binvox == the reference's write_binvox payload (golden files from src/util_io.cpp);
* cvx_encode_voxel_list == the restated write_vox voxel loop;
* cvx_transcode: Morton <-> linear, pinned by the engine's own (reference-exact) Morton and linear
  tables of the same mesh, and by round trips of random tables;
* cvx_mesh_bbox_device / cvx_voxinfo_from_device == the host setup; cvx_gather_soup == indexing.
"""
import os

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
from cuda_voxelizer_gb300 import api as cv  # noqa: E402
from cuda_voxelizer_gb300 import meshgen  # noqa: E402
from cuda_voxelizer_gb300._lib import CvxVoxinfo  # noqa: E402

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "golden_io.npz")


def _cases():
    g = np.load(GOLDEN)
    return sorted({k.rsplit("__", 1)[0] for k in g.files})


@pytest.fixture(scope="module")
def golden():
    return np.load(GOLDEN)


def _dev(table):
    return torch.from_numpy(np.ascontiguousarray(table).view(np.int32)).cuda()


@pytest.mark.parametrize("name", _cases())
def test_binvox_payload_equals_reference_writer(golden, name):
    info = CvxVoxinfo.from_buffer_copy(golden[f"{name}__info"].tobytes())
    got = cv.encode_binvox(info, _dev(golden[f"{name}__table"]))
    assert got == golden[f"{name}__payload"].tobytes()


def test_binvox_of_engine_table_equals_reference_writer_restatement():
    tris = meshgen.icosphere(4, level=6)
    info = cv.make_voxinfo(tris, 256)
    tab = torch.zeros(cv.table_words(info), dtype=torch.int32, device="cuda")
    cv.voxelize_solid(info, torch.from_numpy(tris.reshape(-1)).cuda(), tab)
    host = tab.cpu().numpy().view(np.uint32)
    assert cv.encode_binvox(info, tab) == oracle.binvox_payload(bytes(info), host)


@pytest.mark.parametrize("name", ["torus_g64__linear__surface", "ico5_g128__linear__solid", "random_g32",
                                  "sparse_g128", "full_g64", "empty_g64", "ico3_g8__linear__surface"])
def test_voxel_list_equals_restated_writer(golden, name):
    info_b = golden[f"{name}__info"].tobytes()
    info = CvxVoxinfo.from_buffer_copy(info_b)
    table = golden[f"{name}__table"]
    got = cv.encode_voxel_list(info, _dev(table)).cpu().numpy()
    want = oracle.vox_list(info_b, table)
    assert got.shape == want.shape and np.array_equal(got, want)


def test_voxel_list_rejects_grids_with_y_unequal_z(golden):
    info = CvxVoxinfo.from_buffer_copy(golden["random_40x24x36__info"].tobytes())
    with pytest.raises(cv.CvxError) as e:
        cv.encode_voxel_list(info, _dev(golden["random_40x24x36__table"]))
    assert e.value.status == 2


@pytest.mark.parametrize("g", [8, 16, 64, 128, 512])
@pytest.mark.parametrize("solid", [False, True])
def test_transcode_matches_engine_morton_tables(g, solid):
    tris = meshgen.icosphere(5, level=6 if g >= 128 else 4)
    info = cv.make_voxinfo(tris, g)
    d = torch.from_numpy(tris.reshape(-1)).cuda()
    lin = torch.zeros(cv.table_words(info), dtype=torch.int32, device="cuda")
    mor = torch.zeros_like(lin)
    f = cv.voxelize_solid if solid else cv.voxelize
    f(info, d, lin, False)
    f(info, d, mor, True)
    assert torch.equal(cv.transcode(lin, g, True), mor)
    assert torch.equal(cv.transcode(mor, g, False), lin)


@pytest.mark.parametrize("g", [4, 32, 256])
def test_transcode_round_trip_random(g):
    gen = torch.Generator(device="cuda").manual_seed(g)
    t = torch.randint(-2 ** 31, 2 ** 31 - 1, (g ** 3 // 32,), dtype=torch.int32, device="cuda", generator=gen)
    m = cv.transcode(t, g, True)
    assert torch.equal(cv.transcode(m, g, False), t)
    # spot-check single bits against the oracle's Morton encoder
    host = t.cpu().numpy().view(np.uint32)
    mh = m.cpu().numpy().view(np.uint32)
    rng = np.random.default_rng(g)
    for _ in range(200):
        x, y, z = (int(v) for v in rng.integers(0, g, 3))
        li = x + g * (y + g * z)
        mi = oracle.morton_encode(x, y, z)
        assert ((host[li >> 5] >> (31 - (li & 31))) & 1) == ((mh[mi >> 5] >> (31 - (mi & 31))) & 1)


@pytest.mark.parametrize("g", [4, 16, 32, 64, 128, 256, 512])
@pytest.mark.parametrize("offset", [0, 1])
def test_transcode_every_bit_against_numpy(g, offset):
    """Each grid's column layout (words per row 1 .. 16) and both store widths: a table that begins
    4 bytes after a 16-byte boundary takes the scalar one."""
    n = g ** 3 // 32
    gen = torch.Generator(device="cuda").manual_seed(g + offset)
    t = torch.randint(-2 ** 31, 2 ** 31 - 1, (n + offset,), dtype=torch.int32, device="cuda", generator=gen)[offset:]
    c = np.arange(g, dtype=np.int64)
    s = sum(((c >> i) & 1) << (3 * i) for i in range(10))  # the coordinate's bits, three apart
    code = s[None, None, :] | s[None, :, None] << 1 | s[:, None, None] << 2
    bits = np.unpackbits(t.cpu().numpy().view(np.uint32).byteswap().view(np.uint8))
    want = np.empty_like(bits)
    want[code.reshape(-1)] = bits
    want = np.packbits(want).view(np.uint32).byteswap()
    m = cv.transcode(t, g, True)
    assert np.array_equal(m.cpu().numpy().view(np.uint32), want)
    back = torch.empty(n + offset, dtype=torch.int32, device="cuda")[offset:]
    back.copy_(m)
    assert torch.equal(cv.transcode(back, g, False), t)


@pytest.mark.parametrize("mesh", ["torus", "ico", "soup"])
def test_device_bbox_and_voxinfo_equal_host_setup(mesh):
    tris = {"torus": lambda: meshgen.torus(3), "ico": lambda: meshgen.icosphere(1, level=7),
            "soup": lambda: meshgen.soup(2, n=300_000)}[mesh]()
    d = torch.from_numpy(tris.reshape(-1)).cuda()
    lo, hi = cv.mesh_bbox_device(d)
    hlo, hhi = cv.mesh_bbox(tris)
    assert np.array_equal(lo, hlo) and np.array_equal(hi, hhi)
    assert bytes(cv.voxinfo_from_device(d, 256)) == bytes(cv.make_voxinfo(tris, 256))


def test_gather_soup_matches_indexing_and_flags_bad_faces():
    rng = np.random.default_rng(9)
    verts = rng.normal(size=(5000, 3)).astype(np.float32)
    faces = rng.integers(0, 5000, size=(20000, 3)).astype(np.int32)
    soup, bad = cv.gather_soup(torch.from_numpy(verts).cuda(), torch.from_numpy(faces).cuda())
    assert bad == 0
    assert np.array_equal(soup.cpu().numpy().reshape(-1, 3, 3), verts[faces])
    faces[[3, 77], 1] = 5000
    soup, bad = cv.gather_soup(torch.from_numpy(verts).cuda(), torch.from_numpy(faces).cuda())
    s = soup.cpu().numpy().reshape(-1, 9)
    assert bad == 2 and np.isnan(s[[3, 77]]).all() and not np.isnan(np.delete(s, [3, 77], axis=0)).any()


def _pattern(grid, kind, seed):
    """A linear-order table: bits of the given density, or boxes, whose runs are long."""
    rng = np.random.default_rng(seed)
    v = np.zeros((grid[2], grid[1], grid[0]), dtype=np.uint8)
    if kind == "boxes":
        for _ in range(4):
            a, b = (np.sort(rng.integers(0, np.array(grid) + 1, (2, 3)), axis=0))
            v[a[2]:b[2], a[1]:b[1], a[0]:b[0]] ^= 1
    elif kind == "full":
        v[:] = 1
    elif kind != "empty":
        v[:] = rng.random(v.shape) < float(kind)
    bits = np.concatenate([v.reshape(-1), np.zeros(-v.size % 32, np.uint8)])
    return np.packbits(bits).view(np.uint32).byteswap()


ENCODE_GRIDS = [(1, 1, 1), (2, 3, 5), (5, 16, 16), (40, 17, 17), (33, 31, 31), (32, 32, 32), (31, 33, 33), (64, 64, 64),
                (100, 100, 100), (7, 255, 255), (9, 256, 256), (130, 96, 96), (300, 65, 65), (3, 500, 500),
                (40, 1, 700), (40, 16, 300), (64, 64, 20), (50, 290, 31)]


@pytest.mark.parametrize("kind", ["empty", "full", "boxes", "0.5", "0.01"])
@pytest.mark.parametrize("grid", ENCODE_GRIDS)
def test_encoders_on_any_grid(grid, kind):
    """Stream rows that end inside, on and before words, dense streams (gy <= 16), one tile and many."""
    table = _pattern(grid, kind, sum(grid))
    info = cv.make_info((0, 0, 0), [float(g) for g in grid], grid, 0)
    d = _dev(table)
    assert cv.encode_binvox(info, d) == oracle.binvox_payload(bytes(info), table)
    if grid[1] == grid[2]:
        got = cv.encode_voxel_list(info, d).cpu().numpy()
        assert np.array_equal(got, oracle.vox_list(bytes(info), table)[:got.shape[0]])
        assert got.shape[0] == int(np.unpackbits(table.view(np.uint8)).sum())


def test_encoders_refuse_small_buffers_and_write_nothing():
    import ctypes
    grid = (40, 33, 33)
    table = _pattern(grid, "0.5", 1)
    info = cv.make_info((0, 0, 0), [float(g) for g in grid], grid, 0)
    d = _dev(table)
    payload = oracle.binvox_payload(bytes(info), table)
    n_vox = int(np.unpackbits(table.view(np.uint8)).sum())
    s = torch.cuda.current_stream().cuda_stream
    n = ctypes.c_uint64()
    for f, size, dtype, unit in ((cv.lib.cvx_encode_binvox, len(payload), torch.uint8, 1),
                                 (cv.lib.cvx_encode_voxel_list, n_vox, torch.int32, 3)):
        out = torch.full((size * unit + 8,), 77, dtype=dtype, device="cuda")
        assert f(ctypes.byref(info), d.data_ptr(), out.data_ptr(), size - 1, ctypes.byref(n), s) == 1
        assert n.value == size and bool((out == 77).all())
        assert f(ctypes.byref(info), d.data_ptr(), out.data_ptr(), size, ctypes.byref(n), s) == 0
        assert n.value == size and bool((out[size * unit:] == 77).all())
        ws = torch.empty(256, dtype=torch.uint8, device="cuda")
        g = cv.lib.cvx_encode_binvox_ws if unit == 1 else cv.lib.cvx_encode_voxel_list_ws
        assert g(ctypes.byref(info), d.data_ptr(), ws.data_ptr(), 256, out.data_ptr(), size, ctypes.byref(n), s) == 1


@pytest.mark.parametrize("offset", [0, 1])  # 1: a soup that is not 16-byte aligned
@pytest.mark.parametrize("n", [1, 2, 3, 255, 256, 257, 70_001])
def test_bbox_and_gather_at_odd_sizes(n, offset):
    rng = np.random.default_rng(n)
    verts = rng.normal(size=(n + 2, 3)).astype(np.float32)
    verts[rng.integers(0, n + 2)] *= 100  # an extreme corner anywhere, the ragged end included
    faces = rng.integers(0, n + 2, size=(n, 3)).astype(np.int32)
    faces[-1] = [n + 1, 0, n]
    buf = torch.zeros(9 * n + 8, dtype=torch.float32, device="cuda")
    soup = buf[offset:offset + 9 * n]
    bad = torch.zeros(1, dtype=torch.int64, device="cuda")
    v, f = torch.from_numpy(verts).cuda(), torch.from_numpy(faces).cuda()
    s = torch.cuda.current_stream().cuda_stream
    assert cv.lib.cvx_gather_soup(v.data_ptr(), n + 2, f.data_ptr(), n, soup.data_ptr(), bad.data_ptr(), s) == 0
    host = buf.cpu().numpy()
    want = verts[faces].reshape(-1)
    assert int(bad.item()) == 0 and np.array_equal(host[offset:offset + 9 * n], want)
    assert not host[:offset].any() and not host[offset + 9 * n:].any()
    lo, hi = cv.mesh_bbox_device(soup)
    assert np.array_equal(lo, want.reshape(-1, 3).min(0)) and np.array_equal(hi, want.reshape(-1, 3).max(0))


class _HasHandle:
    """A stream of another library: an object with its handle."""

    def __init__(self, stream):
        self.cuda_stream = stream.cuda_stream


def _io_calls(stream):
    tris = meshgen.torus(1)
    d = torch.from_numpy(tris.reshape(-1)).cuda()
    info = cv.make_voxinfo(tris, 64)
    table = torch.zeros(cv.table_words(info), dtype=torch.int32, device="cuda")
    cv.voxelize(info, d, table)
    torch.cuda.synchronize()
    lo, hi = cv.mesh_bbox_device(d, stream=stream)
    return (lo.tobytes(), hi.tobytes(), bytes(cv.voxinfo_from_device(d, 64, stream=stream)),
            cv.encode_binvox(info, table, stream=stream), cv.encode_voxel_list(info, table, stream=stream).cpu().numpy().tobytes())


@pytest.mark.parametrize("kind", ["torch", "handle", "object", "default", "legacy handle"])
def test_stream_arguments(kind):
    """Every form of a stream argument; the calls' scratch belongs to that stream, and to no other."""
    want = _io_calls(None)
    side = torch.cuda.Stream()
    stream = {"torch": side, "handle": side.cuda_stream, "object": _HasHandle(side), "default": 0, "legacy handle": 1}[kind]
    owners = lambda: {seg["stream"] for seg in torch.cuda.memory_snapshot()}  # noqa: E731
    before = owners()
    assert _io_calls(stream) == want
    assert owners() - before <= {side.cuda_stream}


def test_results_of_calls_on_another_stream():
    """Memory that the current stream still writes when a call on another stream takes it over: the result is not
    touched by that write, nor the write's value read."""
    tris = meshgen.torus(1)
    info = cv.make_voxinfo(tris, 128)
    table = torch.zeros(cv.table_words(info), dtype=torch.int32, device="cuda")
    cv.voxelize(info, torch.from_numpy(tris.reshape(-1)).cuda(), table)
    rng = np.random.default_rng(2)
    v = torch.from_numpy(rng.normal(size=(5000, 3)).astype(np.float32)).cuda()
    f = torch.from_numpy(rng.integers(0, 5002, size=(200_000, 3)).astype(np.int32)).cuda()
    calls = [lambda s: cv.transcode(table, 128, True, stream=s), lambda s: cv.encode_voxel_list(info, table, stream=s),
             lambda s: cv.gather_soup(v, f, stream=s)]
    side = torch.cuda.Stream()
    for call in calls:
        torch.cuda.synchronize()
        want = call(None)
        n_bad = None
        if isinstance(want, tuple):
            want, n_bad = want
        torch.cuda.synchronize()
        for stream in (side, side.cuda_stream):
            torch.cuda._sleep(20_000_000)  # 10 ms on the current stream
            late = torch.full_like(want, 7)
            del late
            got = call(stream)
            if n_bad is not None:
                got, k = got
                assert k == n_bad
            torch.cuda.synchronize()
            assert torch.equal(got.view(torch.int32), want.view(torch.int32))
            del got


def test_binvox_on_another_stream():
    tris = meshgen.icosphere(3, level=4)
    info = cv.make_voxinfo(tris, 200)
    table = torch.zeros(cv.table_words(info), dtype=torch.int32, device="cuda")
    cv.voxelize_solid(info, torch.from_numpy(tris.reshape(-1)).cuda(), table)
    want = cv.encode_binvox(info, table)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    torch.cuda._sleep(20_000_000)
    late = torch.full((4 * cv.table_words(info),), 7, dtype=torch.uint8, device="cuda")
    del late
    assert cv.encode_binvox(info, table, stream=side) == want
