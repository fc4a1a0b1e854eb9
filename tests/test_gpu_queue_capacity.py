"""The work queue that a launch needs (queue_capacity): launches whose warps'
stacks hold their own work fit a queue of the smallest size, and with small
stacks a modest one, whatever blocks the traversal forms of its warps. Their
candidate leaf pairs are the defaults' in number, which the other tests compare
with the oracle."""
import numpy as np
import pytest

from inmyroom_vulkan_gb300 import capi, scenes

pytestmark = pytest.mark.gpu

# per case: settings beside the defaults (stack_entries 512, donate_min 32)
CASES = {"one heavy pair": dict(queue_capacity=8192, stack_entries=256), "scene": dict(queue_capacity=2048, stack_entries=256),
         "20 pairs": dict(queue_capacity=2048), "uneven queries": dict(queue_capacity=2048),
         "uneven queries, late donations": dict(queue_capacity=2048, donate_min=449)}


def queries(ctx, case):
    if case == "scene":
        sc = scenes.scene()
        ids = ctx.build_trees(sc.meshes)
        qa, qb, ma, mb = sc.pairs[:, 0], sc.pairs[:, 1], sc.mats[sc.pairs[:, 0]], sc.mats[sc.pairs[:, 1]]
    elif case.startswith("uneven"):
        sw = scenes.batch_sweep(n_queries=2000, pool=24)
        ids = ctx.build_trees(sw.meshes)
        qa, qb, ma, mb = sw.qa, sw.qb, sw.mats_a, sw.mats_b
    else:
        rng = np.random.Generator(np.random.PCG64(5))
        n = 1 if case == "one heavy pair" else 20
        ids = ctx.build_trees([scenes.octa_sphere(6, 1.0, 0.01, rng) if n == 1 else scenes.uv_sphere(20000, 1.0, 0.01, rng)
                               for _ in range(2)])
        qa, qb = np.zeros(n, int), np.ones(n, int)
        ma = [scenes.pose(np.eye(3), [0.0, 0.0, 0.0])] * n
        mb = [scenes.pose(scenes.random_rotation(rng) if n > 1 else np.eye(3), [0.1 * (k % 9), 0.0, 0.0]) for k in range(n)]
    return capi.make_queries(ids[qa], ids[qb], np.stack([capi.relative_matrix(a, b) for a, b in zip(ma, mb)]))


@pytest.mark.parametrize("case", CASES)
def test_queue_capacity_that_suffices(case):
    with capi.Context(max_leaf_pairs=1 << 24) as ctx:
        q = queries(ctx, case)
        want = ctx.collide(q, flags=capi.CG_MID_ONLY)["leaf_pairs"]
        assert want > 1000
        ctx.reconfigure(**CASES[case])
        for _ in range(3):
            assert ctx.collide(q, flags=capi.CG_MID_ONLY)["leaf_pairs"] == want
