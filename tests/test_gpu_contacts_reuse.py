"""Contacts, rays and mean origins of steps that follow one another in one
context without a wait between them, their maps of other sizes in the same
places of the same buffers: each step's results are its own, bit for bit and in
order against the oracle
(src/CollisionDetection/CreateUncollideRays.cpp:60-201). Each step has maps of
1,024 triangles and more beside small ones, which the order stage's two
launches work on side by side."""
import numpy as np
import pytest

from inmyroom_vulkan_gb300 import capi
from test_gpu_contacts import check_grouped, check_query
from test_gpu_contacts_edge import QUAD
from test_gpu_map_sizes import spikes

pytestmark = pytest.mark.gpu

SIZES = [[1500, 40, 700, 3, 1100, 129, 64, 500], [40, 1500, 2, 700, 130, 1100, 500, 33], [300, 10, 40, 1024, 1, 2000, 90, 128]]


def test_steps_after_one_another(port):
    torch = pytest.importorskip("torch")
    eye = np.eye(4, dtype=np.float32).reshape(16)
    with capi.Context() as ctx:
        steps, mids, ids = [], [], {}
        quad = port.tree_build(QUAD.points, QUAD.indices, QUAD.normals)
        qid = ctx.upload_flat(quad.export())
        trees = {n: port.tree_build(m.points, m.indices, m.normals) for n in sorted({n for s in SIZES for n in s})
                 for m in [spikes(n)]}
        ids = {n: ctx.upload_flat(t.export()) for n, t in trees.items()}
        oracle = {n: port.mid_phase(quad, t, eye, eye) for n, t in trees.items()}
        for sizes in SIZES:
            rel = np.stack([capi.relative_matrix(eye, eye)] * len(sizes))
            q = capi.make_queries([qid] * len(sizes), [ids[n] for n in sizes], rel)
            steps.append((torch.from_numpy(q.view(np.uint8).copy()).cuda(), len(sizes)))
            mids.append([oracle[n] for n in sizes])
        torch.cuda.synchronize()
        for order in ([0, 1], [1, 2, 0, 1, 2], [2, 1, 0], [0, 1, 2, 0, 1, 2, 0, 1, 2], [1, 0, 1, 0]):
            for k in order:
                ctx.collide_async(steps[k][0].data_ptr(), steps[k][1], capi.CG_CONTACTS)
            assert ctx.sync_stats()["status"] == 0
            contacts, rays, averages = ctx.contacts(), ctx.rays(), ctx.ray_averages()
            check_grouped(contacts, rays)
            assert len(contacts) == sum(len(m.contacts(s)[0]) for m in mids[order[-1]] for s in (0, 1))
            for i, m in enumerate(mids[order[-1]]):
                check_query(port, m, i, contacts, rays, averages)
