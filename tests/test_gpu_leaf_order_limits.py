"""Ordered candidate leaf pairs (CG_DFS_ORDER, csrc/cg_leaf_order.cu) at the
limits of the list: more leaf pairs than max_leaf_pairs (the ones that were
stored come grouped and ordered), a query of more than 2^20 (three merges), and
the device memory that the first ordered step takes."""
import ctypes as C

import numpy as np
import pytest

from inmyroom_vulkan_gb300 import capi, scenes

pytestmark = pytest.mark.gpu
FLAGS = capi.CG_KEEP_LEAF_PAIRS | capi.CG_DFS_ORDER | capi.CG_MID_ONLY
EYE = np.eye(4, dtype=np.float32).reshape(16)


def spheres(port, subdiv, jitter):
    rng = np.random.Generator(np.random.PCG64(11))
    trees = [port.tree_build(m.points, m.indices, m.normals)
             for m in (scenes.octa_sphere(subdiv, 1.0, jitter, rng) for _ in range(2))]
    return trees, port.mid_phase(trees[0], trees[1], EYE, EYE).leaf_pairs().astype(np.uint32).reshape(-1, 4)


def rows(lp):
    return np.stack([lp["offset_a"], lp["count_a"], lp["offset_b"], lp["count_b"]], 1).astype(np.uint32)


def test_more_than_two_merges(port):
    trees, want = spheres(port, 6, 0.1)
    assert len(want) > 1 << 20
    with capi.Context() as ctx:
        a, b = (ctx.upload_flat(t.export()) for t in trees)
        q = capi.make_queries([a, a], [b, b], np.stack([capi.relative_matrix(EYE, EYE)] * 2))
        assert ctx.collide(q[:1], FLAGS)["leaf_pairs"] == len(want)
        assert np.array_equal(rows(ctx.leaf_pairs()), want)


@pytest.mark.parametrize("cap", [1, 2, 31, 700, 1023, 1024, 1025, 5000, 60000])
def test_overflowed_list_is_grouped_and_ordered(port, cap):
    trees, want = spheres(port, 5, 0.01)
    place = {tuple(r): i for i, r in enumerate(want.tolist())}
    n = 3
    assert n * len(want) > cap
    with capi.Context(max_leaf_pairs=cap) as ctx:
        a, b = (ctx.upload_flat(t.export()) for t in trees)
        q = capi.make_queries([a] * n, [b] * n, np.stack([capi.relative_matrix(EYE, EYE)] * n))
        for _ in range(2):
            st = ctx.collide(q, FLAGS, check=False)
            assert st["rc"] == st["status"] == capi.CG_ERR_OUTPUT_OVERFLOW and st["leaf_pairs"] == n * len(want)
            got, count = np.zeros(cap, capi.LEAF_PAIR_DTYPE), C.c_uint64()
            assert ctx.lib.cg_read_leaf_pairs(ctx.h, got.ctypes.data, cap, C.byref(count)) == capi.CG_ERR_OUTPUT_OVERFLOW
            assert count.value == n * len(want)
            at = [(int(k), place[tuple(r)]) for k, r in zip(got["query"], rows(got).tolist())]
            assert all(x < y for x, y in zip(at, at[1:])) and at[-1][0] < n  # each once, in the reference's order


def test_memory_of_the_first_ordered_step(port):
    torch = pytest.importorskip("torch")
    cap = 1 << 24
    with capi.Context(max_leaf_pairs=cap) as ctx:
        tree = ctx.build_trees([scenes.octa_sphere(3, 1.0, 0.01, np.random.Generator(np.random.PCG64(2)))])
        q = capi.make_queries(tree, tree, capi.relative_matrix(EYE, EYE)[None])
        ctx.collide(q, FLAGS & ~capi.CG_DFS_ORDER)
        free = torch.cuda.mem_get_info()[0]
        ctx.collide(q, FLAGS)
        assert free - torch.cuda.mem_get_info()[0] <= 24 * cap + (16 << 20)


def test_order_belongs_to_the_step_that_ran(port):
    """A capture between a step and its reads changes neither's leaf pairs, and a second read returns the first's."""
    torch = pytest.importorskip("torch")
    trees, want = spheres(port, 4, 0.01)
    with capi.Context() as ctx:
        a, b = (ctx.upload_flat(t.export()) for t in trees)
        q = capi.make_queries([a, b, a], [b, a, b], np.stack([capi.relative_matrix(EYE, EYE)] * 3))
        d_q = torch.from_numpy(q.view(np.uint8).copy()).cuda()
        torch.cuda.synchronize()
        plain = capi.CG_KEEP_LEAF_PAIRS | capi.CG_MID_ONLY
        ctx.collide(q[:1], FLAGS)
        ctx.graph_capture(d_q.data_ptr(), 3, plain)
        for _ in range(2):
            assert np.array_equal(rows(ctx.leaf_pairs()), want)
        ctx.graph_launch()  # unordered, of three queries
        lp = ctx.leaf_pairs()
        assert len(lp) > 2 * len(want) and sorted(map(tuple, rows(lp[lp["query"] == 2]).tolist())) == sorted(map(tuple, want.tolist()))
        ctx.graph_capture(d_q.data_ptr(), 1, FLAGS)
        again = ctx.leaf_pairs()
        assert np.array_equal(again, lp)
        for _ in range(2):
            ctx.graph_launch()
            assert np.array_equal(rows(ctx.leaf_pairs()), want)
