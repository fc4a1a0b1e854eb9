"""Steps that follow one another on a stream without a wait between them, each
after a copy that puts other queries into the same device buffer: every step
packs the queries that were there when it ran; its colliding pairs are the
oracle's (src/CollisionDetection/CreateUncollideRays.cpp:60-112)."""
import numpy as np
import pytest

from inmyroom_vulkan_gb300 import capi, scenes

pytestmark = pytest.mark.gpu


def test_queries_replaced_between_steps(port):
    torch = pytest.importorskip("torch")
    rng = np.random.Generator(np.random.PCG64(3))
    meshes = [scenes.octa_sphere(k, 1.0, 0.01, rng) for k in (4, 5)]
    trees = [port.tree_build(m.points, m.indices, m.normals) for m in meshes]
    at = lambda dx: scenes.pose(np.eye(3), [dx, 0.0, 0.0])  # noqa: E731
    sets = [[(0, 1, x) for x in (0.2, 9.0, 0.9)], [(1, 0, x) for x in (1.9, 0.1, 0.4)], [(0, 0, x) for x in (1.0, 1.5, 9.0)]]
    with capi.Context() as ctx:
        ids = [ctx.upload_flat(t.export()) for t in trees]
        queries, want = [], []
        for s in sets:
            rel = np.stack([capi.relative_matrix(at(0.0), at(x)) for _, _, x in s])
            q = capi.make_queries([ids[i] for i, _, _ in s], [ids[j] for _, j, _ in s], rel)
            queries.append(torch.from_numpy(q.view(np.uint8).copy()).cuda())
            got = []
            for k, (i, j, x) in enumerate(s):
                p, _, _, _ = port.mid_phase(trees[i], trees[j], at(0.0), at(x)).narrow()
                got += [(k, int(a), int(b)) for a, b in p[:, :2]]
            want.append(sorted(got))
        assert len({tuple(w) for w in want}) == len(sets) and all(want)
        stream = torch.cuda.Stream()
        buf = queries[0].clone()
        torch.cuda.synchronize()
        for order in ([0, 1], [1, 2, 0], [2, 1, 0, 2, 1, 0, 2], [0, 2, 1]):
            with torch.cuda.stream(stream):
                for k in order:
                    buf.copy_(queries[k], non_blocking=True)
                    ctx.collide_async(buf.data_ptr(), len(sets[k]), 0, stream.cuda_stream)
            assert ctx.sync_stats()["status"] == 0
            p = ctx.tri_pairs()
            got = sorted(zip(p["query"].tolist(), p["tri_a"].tolist(), p["tri_b"].tolist()))
            assert got == want[order[-1]], order
