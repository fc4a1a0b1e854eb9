"""Ordered candidate leaf pairs (CG_DFS_ORDER, csrc/cg_leaf_order.cu) against
the oracle's recursion, around the sizes where the sort's shape changes: no
leaf pairs, one, about a tile of 1,024, a few tiles, and more than 32 tiles
(two merges); alone and mixed in one launch, as cg_collide and as a captured
graph."""
import numpy as np
import pytest

from inmyroom_vulkan_gb300 import capi, scenes

pytestmark = pytest.mark.gpu
FLAGS = capi.CG_KEEP_LEAF_PAIRS | capi.CG_DFS_ORDER | capi.CG_MID_ONLY


@pytest.fixture(scope="module")
def setup(port):
    rng = np.random.Generator(np.random.PCG64(11))
    meshes = [scenes.octa_sphere(k, 1.0, 0.01, rng) for k in (6, 6, 4, 4, 0)]
    return meshes, [port.tree_build(m.points, m.indices, m.normals) for m in meshes]


def place(dx):
    return scenes.pose(np.eye(3), [dx, 0.0, 0.0])


# per case: (first mesh, second mesh, offset) of each query
CASES = {
    "none": [(2, 3, 9.0)],
    "one tiny": [(4, 4, 0.1)],
    "a tile or so": [(2, 3, 1.9), (2, 3, 1.0), (2, 3, 0.5), (2, 3, 0.1)],
    "many tiles": [(0, 1, 0.0)],
    "mixed": [(2, 3, 9.0), (0, 1, 0.3), (4, 4, 0.1), (2, 3, 0.0), (2, 3, 9.0), (0, 1, 0.0), (4, 2, 0.9), (2, 3, 9.0)],
}


@pytest.mark.parametrize("case", CASES)
def test_ordered_leaf_pairs(port, setup, case):
    torch = pytest.importorskip("torch")
    meshes, trees = setup
    with capi.Context() as ctx:
        ids = ctx.build_trees(meshes)
        a, b, dx = zip(*CASES[case])
        ma, mb = [place(0.0)] * len(a), [place(x) for x in dx]
        rel = np.stack([capi.relative_matrix(x, y) for x, y in zip(ma, mb)])
        q = capi.make_queries(ids[list(a)], ids[list(b)], rel)
        want = [port.mid_phase(trees[i], trees[j], x, y).leaf_pairs() for i, j, x, y in zip(a, b, ma, mb)]
        d_q = torch.from_numpy(q.view(np.uint8).copy()).cuda()
        torch.cuda.synchronize()
        for how in ("call", "again", "graph"):
            if how == "graph":
                ctx.graph_capture(d_q.data_ptr(), len(q), FLAGS)
                ctx.graph_launch()
                st = ctx.sync_stats()
            else:
                st = ctx.collide(q, FLAGS)
            lp = ctx.leaf_pairs()
            assert st["leaf_pairs"] == len(lp) == sum(len(w) for w in want)
            at = 0
            for k, w in enumerate(want):
                g = lp[at:at + len(w)]
                at += len(w)
                got = np.stack([g["offset_a"], g["count_a"], g["offset_b"], g["count_b"]], 1).astype(np.uint32)
                assert np.all(g["query"] == k) and np.array_equal(got, w.astype(np.uint32).reshape(-1, 4)), (how, k)
    if case == "many tiles":
        assert len(want[0]) > 32 * 1024
