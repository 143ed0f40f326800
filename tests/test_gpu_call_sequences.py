"""Calls in any order on one stream: each finds its counters cleared, whoever cleared them.

The meshes have triangles of every size, so that every call queues work: a counter left over from an
earlier call would show as missing or repeated rows.
"""
import random

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from cuda_voxelizer_gb300 import api as cv  # noqa: E402
from cuda_voxelizer_gb300 import meshgen  # noqa: E402

pytestmark = pytest.mark.gpu


class _Work:
    def __init__(self):
        self.items = []
        for tris, g in ((meshgen.soup(1, n=3000), 200), (meshgen.icosphere(2, level=3), 256), (meshgen.torus(3), 64)):
            info = cv.make_voxinfo(tris, g)
            d = torch.from_numpy(np.ascontiguousarray(tris).reshape(-1)).cuda()
            for solid in ((False,) if g == 200 else (False, True)):
                ws = torch.empty(cv.workspace_size(info, solid), dtype=torch.uint8, device="cuda")
                want = self.table(info)
                cv.voxelize_ws(info, d, want, ws, solid=solid)  # its own counters, cleared by the host
                self.items.append((info, d, solid, want))

    @staticmethod
    def table(info):
        return torch.zeros(cv.table_words(info), dtype=torch.int32, device="cuda")

    def call(self, k, table):
        info, d, solid, _ = self.items[k]
        (cv.voxelize_solid if solid else cv.voxelize)(info, d, table)


@pytest.mark.parametrize("seed", range(4))
def test_direct_batched_and_captured_calls_interleaved(seed):
    rng = random.Random(seed)
    work = _Work()
    stream = torch.cuda.Stream()
    graphs = []
    with torch.cuda.stream(stream):
        # the scratch has to exist before a capture, in the size of the largest call that will be made
        cv.voxelize_batch([cv.Job(info, d, work.table(info), False, solid) for info, d, solid, _ in work.items])
        torch.cuda.synchronize()
        for k in rng.sample(range(len(work.items)), 3):
            table = work.table(work.items[k][0])
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=stream):
                table.zero_()
                work.call(k, table)
            graphs.append((g, k, table))
        done = []
        for _ in range(40):
            what = rng.randrange(3)
            if what == 0:
                k = rng.randrange(len(work.items))
                table = work.table(work.items[k][0])
                work.call(k, table)
                done.append((k, table))
            elif what == 1:  # surface and solid jobs: two launch sequences in one call
                ks = rng.sample(range(len(work.items)), rng.randint(2, len(work.items)))
                tables = [work.table(work.items[k][0]) for k in ks]
                cv.voxelize_batch([cv.Job(work.items[k][0], work.items[k][1], t, False, work.items[k][2])
                                   for k, t in zip(ks, tables)])
                done += list(zip(ks, tables))
            else:
                g, k, table = rng.choice(graphs)
                g.replay()
                done.append((k, table.clone()))
        cv.device_status(stream)
    torch.cuda.synchronize()
    for k, table in done:
        assert torch.equal(table, work.items[k][3])


def test_calls_on_several_streams():
    work = _Work()
    streams = [torch.cuda.Stream() for _ in range(3)]
    done = []
    for r in range(5):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                k = (r + i) % len(work.items)
                table = work.table(work.items[k][0])
                work.call(k, table)
                done.append((k, table))
    torch.cuda.synchronize()
    for s in streams:
        cv.device_status(s)
        cv.stream_release(s)
    for k, table in done:
        assert torch.equal(table, work.items[k][3])



def test_calls_from_several_threads():
    """Threads with a stream each: their calls share nothing."""
    import threading
    work = _Work()
    torch.cuda.synchronize()
    bad, streams = [], [torch.cuda.Stream() for _ in range(4)]

    def run(i):
        try:
            with torch.cuda.stream(streams[i]):
                done = []
                for r in range(25):
                    k = (r + i) % len(work.items)
                    table = work.table(work.items[k][0])
                    work.call(k, table)
                    done.append((k, table))
                cv.device_status(streams[i])
                bad.extend(k for k, table in done if not torch.equal(table, work.items[k][3]))
        except Exception as e:
            bad.append(e)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(streams))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    for s in streams:
        cv.stream_release(s)


@pytest.mark.parametrize("morton,g", [(False, 100), (False, 128), (False, 72), (True, 16), (True, 64), (True, 128)])
@pytest.mark.parametrize("n", [2, 3])
def test_solid_jobs_of_a_plan_that_share_a_table(morton, g, n):
    """Each job's bits are XORed into the table, as by one call after another: jobs that flip the same words, jobs
    in parts of the table of their own, a table that overlaps another one in part, and one of its own."""
    infos, tris = [], []
    for k in range(n):
        t = meshgen.icosphere(k, level=4)
        infos.append(cv.make_voxinfo(t, g))
        tris.append(torch.from_numpy(np.ascontiguousarray(t).reshape(-1)).cuda())
    low = cv.make_info((-1, -1, -1), (3, 3, 3), g, infos[0].n_triangles)  # one corner of the box
    high = cv.make_info((-3, -3, -3), (1, 1, 1), g, infos[0].n_triangles)
    unit = tris[0] / tris[0].abs().max()
    W = cv.table_words(infos[0])
    jobs = [(i, t, 0) for i, t in zip(infos, tris)]
    jobs += [(low, unit, 2 * W), (high, unit, 2 * W), (infos[0], tris[0], 3 * W - 5), (infos[0], tris[0], 5 * W)]
    want, got = (torch.zeros(6 * W, dtype=torch.int32, device="cuda") for _ in range(2))
    for info, t, at in jobs:
        cv.voxelize_solid(info, t, want[at:at + W], morton)
    plan = cv.Plan([cv.Job(info, t, got[at:at + W], morton, True) for info, t, at in jobs], clear_tables=True)
    for _ in range(20):
        got.fill_(-1)
        plan.launch()
        for at in (0, 2 * W, 5 * W):
            end = at + W if at != 2 * W else 4 * W - 5
            assert torch.equal(got[at:end], want[at:end]), at
    plan.close()
