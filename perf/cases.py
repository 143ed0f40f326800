"""The work a user of this package has it do, as cases to be timed through its public entry points.

Kinds of case (the field ``kind``):

* ``call``       one voxelization into a zeroed table: ``voxelize`` / ``voxelize_solid``
* ``plan``       one launch of a ``Plan`` over a mix of meshes, grids, modes and layouts
* ``host``       one round trip of a ``HostPlan``: triangles up, four tables down
* ``transcode``  one table from linear to Morton order or back
* ``binvox``     the run-length payload of a table, put into a host buffer
* ``voxels``     the list of a table's set voxels, on the device
* ``ingest``     an indexed mesh to a triangle soup, and the voxinfo of that soup

Meshes come from ``meshgen`` (tori, displaced icospheres, soups of triangles of very different
sizes), all made from the seed.
"""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import torch

import cuda_voxelizer_gb300 as cv
from cuda_voxelizer_gb300 import meshgen


def listed():
    return [
        # a small object at a small grid, as a tool calls once per object: launches and host time count
        {"name": "torus_64_surface", "kind": "call", "mesh": "torus", "size": 48, "grid": 64, "solid": False,
         "morton": False},
        # a medium mesh filled at a grid that is no multiple of a word: rows begin inside words
        {"name": "ico6_500_solid", "kind": "call", "mesh": "icosphere", "size": 6, "grid": 500, "solid": True,
         "morton": False},
        # the benchmark's mesh (1.3 M triangles of a few voxels) as a surface, and filled in Morton order
        {"name": "ico8_512_surface", "kind": "call", "mesh": "icosphere", "size": 8, "grid": 512, "solid": False,
         "morton": False},
        {"name": "ico8_512_solid_morton", "kind": "call", "mesh": "icosphere", "size": 8, "grid": 512, "solid": True,
         "morton": True},
        # two million triangles from a quarter voxel to half the grid: the size stress
        {"name": "soup_1024_surface", "kind": "call", "mesh": "soup", "size": 2_000_000, "grid": 1024, "solid": False,
         "morton": False},
        # many meshes of 1 k to 500 k triangles at 64^3 to 512^3, surface and solid, both orders, as one graph
        {"name": "plan_mix_48", "kind": "plan", "meshes": 48},
        # host buffers in and out, all four modes: what the reference's program does around its kernels
        {"name": "host_ico8_512", "kind": "host", "mesh": "icosphere", "size": 8, "grid": 512},
        # a large table reordered for a Morton reader, and a medium one brought back
        {"name": "transcode_1024_to_morton", "kind": "transcode", "mesh": "icosphere", "size": 7, "grid": 1024,
         "solid": True, "to_morton": True},
        {"name": "transcode_512_to_linear", "kind": "transcode", "mesh": "icosphere", "size": 7, "grid": 512,
         "solid": True, "to_morton": False},
        # the two exports of a filled mesh
        {"name": "binvox_512", "kind": "binvox", "mesh": "icosphere", "size": 7, "grid": 512, "solid": True},
        {"name": "voxels_512", "kind": "voxels", "mesh": "icosphere", "size": 7, "grid": 512, "solid": True},
        # a mesh as a loader hands it over (vertices and faces) to what the voxelizer reads
        {"name": "ingest_1m", "kind": "ingest", "nu": 1024, "nv": 512},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _mesh_fields(rng, most_level=8):
    if rng.random() < 0.5:
        return {"mesh": "torus", "size": _log_int(rng, 16, 500)}  # 1 k to 1 M triangles
    return {"mesh": "icosphere", "size": rng.randint(3, most_level)}


def draw(rng):
    kind = rng.choices(["call", "plan", "host", "transcode", "binvox", "voxels", "ingest"], [12, 2, 1, 3, 2, 2, 2])[0]
    if kind == "call":
        if rng.random() < 0.2:
            return {"kind": kind, "mesh": "soup", "size": _log_int(rng, 1_000, 1_000_000), "grid": _log_int(rng, 64, 1024),
                    "solid": False, "morton": False}
        morton = rng.random() < 0.4
        grid = 2 ** rng.randint(5, 10) if morton else _log_int(rng, 32, 1024)
        return {"kind": kind, **_mesh_fields(rng), "grid": grid, "solid": rng.random() < 0.4, "morton": morton}
    if kind == "plan":
        return {"kind": kind, "meshes": _log_int(rng, 4, 48)}
    if kind == "host":
        return {"kind": kind, **_mesh_fields(rng), "grid": 2 ** rng.randint(6, 9)}
    if kind == "transcode":
        return {"kind": kind, **_mesh_fields(rng, 7), "grid": 2 ** rng.randint(5, 10), "solid": rng.random() < 0.5,
                "to_morton": rng.random() < 0.5}
    if kind == "ingest":
        nv = _log_int(rng, 16, 700)
        return {"kind": kind, "nu": _log_int(rng, nv, 2 * nv + 1), "nv": nv}
    return {"kind": kind, **_mesh_fields(rng, 7), "grid": _log_int(rng, 32, 512), "solid": rng.random() < 0.5}


# ---- sizes ---------------------------------------------------------------------------------------

def _n_triangles(case):
    s = case["size"]
    return {"torus": 4 * s * s, "icosphere": 20 * 4 ** s, "soup": s}[case["mesh"]]


def _table_bytes(grid):
    return (grid ** 3 + 31) // 32 * 4


def _mix(case):
    return meshgen.batch_mix(0, case["meshes"])


def work(case):
    """Each input read once, each output written once."""
    kind = case["kind"]
    if kind == "plan":
        return {"bytes": sum(36 * s.n_triangles + _table_bytes(s.gridsize) for s in _mix(case)), "flops": 0}
    if kind == "ingest":
        quads = case["nu"] * case["nv"]
        return {"bytes": 12 * quads + 2 * quads * (12 + 36), "flops": 0}
    table = _table_bytes(case["grid"])
    if kind == "call":
        return {"bytes": 36 * _n_triangles(case) + table, "flops": 0}
    if kind == "host":
        return {"bytes": 36 * _n_triangles(case) + 4 * table, "flops": 0}
    if kind == "transcode":
        return {"bytes": 2 * table, "flops": 0}
    # The outputs of the two exports depend on the mesh; what a ball in the cube around it gives:
    # about a sixth of the voxels when filled, else a shell of about 2 g^2 of them.
    g = case["grid"]
    voxels = g ** 3 // 6 if case["solid"] else 2 * g * g
    if kind == "voxels":
        return {"bytes": table + 12 * voxels, "flops": 0}
    return {"bytes": table + 2 * (g ** 3 // 255 + 4 * g * g), "flops": 0}


# ---- inputs --------------------------------------------------------------------------------------

def _mesh(case, seed):
    if case["mesh"] == "torus":
        return meshgen.torus(seed, nu=2 * case["size"], nv=case["size"])
    if case["mesh"] == "icosphere":
        return meshgen.icosphere(seed, level=case["size"])
    return meshgen.soup(seed, n=case["size"])


def _device(tris):
    return torch.from_numpy(np.ascontiguousarray(tris, dtype=np.float32).reshape(-1)).cuda()


def _table(info):
    return torch.zeros(cv.table_words(info), dtype=torch.int32, device="cuda")


def _indexed(case, seed):
    """A torus as vertices and faces (host arrays), slightly jittered."""
    nu, nv = case["nu"], case["nv"]
    rng = np.random.default_rng(seed)
    u, v = np.meshgrid(2 * np.pi * np.arange(nu) / nu, 2 * np.pi * np.arange(nv) / nv, indexing="ij")
    verts = np.stack([(1 + 0.35 * np.cos(v)) * np.cos(u), (1 + 0.35 * np.cos(v)) * np.sin(u), 0.35 * np.sin(v)], -1)
    verts = (verts.reshape(-1, 3) + rng.normal(0.0, 1e-3, (nu * nv, 3))).astype(np.float32)
    i, j = np.meshgrid(np.arange(nu), np.arange(nv), indexing="ij")
    a, b = i * nv + j, (i + 1) % nu * nv + j
    c, d = (i + 1) % nu * nv + (j + 1) % nv, i * nv + (j + 1) % nv
    faces = np.stack([np.stack([a, b, c], -1), np.stack([a, c, d], -1)], -2).reshape(-1, 3).astype(np.int32)
    return verts, faces


def _most_pairs(grid):
    """Room for a closed mesh's binvox pairs: a run is cut at 255 voxels, and a line along y crosses
    the surface a few times."""
    return grid ** 3 // 255 + 16 * grid * grid + 256


def _moved(table, grid, seed):
    """A linear table with its voxels moved around cyclically, by whole voxels of the seed's choice."""
    place = torch.arange(31, -1, -1, device=table.device)
    bits = ((table.view(-1, 1) >> place) & 1).to(torch.uint8).view(-1)
    box = bits[:grid ** 3].view(grid, grid, grid)
    rng = np.random.default_rng(seed)
    bits[:grid ** 3] = torch.roll(box, [int(k) for k in rng.integers(0, grid, 3)], (0, 1, 2)).reshape(-1)
    return (bits.view(-1, 32).to(torch.int64) << place).sum(1).to(torch.int32)


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "call":
        tris = _mesh(case, seed)
        state["info"] = cv.make_voxinfo(tris, case["grid"])
        state["tris"] = _device(tris)
        state["table"] = _table(state["info"])
    elif kind == "plan":
        jobs = []
        for i, spec in enumerate(_mix(case)):  # the sizes and modes of one mix, meshes of the seed
            tris = replace(spec, seed=1000 * seed + i).build()
            info = cv.make_voxinfo(tris, spec.gridsize)
            jobs.append(cv.Job(info, _device(tris), _table(info), spec.morton, spec.solid))
        state["tables"] = [j.table for j in jobs]
        state["plan"] = cv.Plan(jobs, clear_tables=True)
    elif kind == "host":
        tris = _mesh(case, seed)
        info = cv.make_voxinfo(tris, case["grid"])
        h_tris = torch.from_numpy(np.ascontiguousarray(tris).reshape(-1)).pin_memory()
        d_tris = torch.empty(h_tris.numel(), dtype=torch.float32, device="cuda")
        jobs = []
        for solid in (False, True):
            for morton in (False, True):
                h_table = torch.empty(cv.table_words(info), dtype=torch.int32, pin_memory=True)
                jobs.append(cv.HostJob(info, h_tris, d_tris, h_table, _table(info), morton, solid))
        state["tables"] = [j.h_table for j in jobs]
        state["plan"] = cv.HostPlan(jobs)
    elif kind == "ingest":
        verts, faces = _indexed(case, seed)
        state["verts"], state["faces"] = torch.from_numpy(verts).cuda(), torch.from_numpy(faces).cuda()
    else:
        # one mesh at places of the seed for the voxel list, so that every seed's has the same length
        tris = _mesh(case, 0 if kind == "voxels" else seed)
        state["info"] = cv.make_voxinfo(tris, case["grid"])
        state["table"] = _table(state["info"])
        from_morton = kind == "transcode" and not case["to_morton"]
        voxelize = cv.voxelize_solid if case["solid"] else cv.voxelize
        voxelize(state["info"], _device(tris), state["table"], morton_code=from_morton)
        if kind == "binvox":
            state["file"] = np.zeros(2 * _most_pairs(case["grid"]), dtype=np.uint8)
        elif kind == "voxels":
            state["table"] = _moved(state["table"], case["grid"], seed)
    torch.cuda.synchronize()
    return state


# ---- one pass ------------------------------------------------------------------------------------

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "call":
        state["table"].zero_()
        voxelize = cv.voxelize_solid if case["solid"] else cv.voxelize
        voxelize(state["info"], state["tris"], state["table"], morton_code=case["morton"])
        return state["table"]
    if kind == "plan":
        state["plan"].launch()
        return state["tables"]
    if kind == "host":
        state["plan"].launch()
        torch.cuda.current_stream().synchronize()  # the tables are read on the host
        return state["tables"]
    if kind == "transcode":
        return cv.transcode(state["table"], case["grid"], case["to_morton"])
    if kind == "binvox":
        payload = np.frombuffer(cv.encode_binvox(state["info"], state["table"]), dtype=np.uint8)
        state["file"][:payload.size] = payload  # the image of the file; what follows it stays zero
        return state["file"]
    if kind == "voxels":
        return cv.encode_voxel_list(state["info"], state["table"])
    soup, bad = cv.gather_soup(state["verts"], state["faces"])
    info = cv.voxinfo_from_device(soup, 256)
    return {"soup": soup, "bad": bad, "min": list(info.bbox_min), "max": list(info.bbox_max), "unit": list(info.unit)}


def exact(case, seed):
    """Only the ingest computes numbers; the others' outputs are bits and integers."""
    if case["kind"] != "ingest":
        return None
    verts, faces = _indexed(case, seed)
    soup = verts.astype(np.float64)[faces].reshape(-1, 3)
    lo, hi = soup.min(0), soup.max(0)
    ext = hi - lo
    pad = (ext.max() - ext) / 2  # the bounding cube, then a margin of 1/10001 of it on every side
    lo, hi = lo - pad, hi + pad
    eps = (hi - lo) / 10001
    lo, hi = lo - eps, hi + eps
    return {"soup": soup.reshape(-1), "bad": None, "min": list(lo), "max": list(hi), "unit": list((hi - lo) / 256)}
