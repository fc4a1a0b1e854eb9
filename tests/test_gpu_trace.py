"""The utilisation timeline (CG_TRACE): its columns add up to the step's own
counts (an item is a split whose two box pairs are tested; the root pairs are
the pack kernel's), with warps as the unit of a step, at every width of the
traversal's worker blocks."""
import numpy as np
import pytest

from inmyroom_vulkan_gb300 import capi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("settings", [dict(), dict(stack_entries=256)], ids=["default", "small stacks"])
@pytest.mark.parametrize("n", [1, 100, 600])
def test_timeline_adds_up(n, settings):
    rp = scenes.rigid_pair(n_poses=n)
    with capi.Context(**settings) as ctx:
        a, b = ctx.build_trees([rp.mesh_a, rp.mesh_b])
        q = capi.make_queries([a] * n, [b] * n, np.stack([capi.relative_matrix(x, y) for x, y in zip(rp.mats_a, rp.mats_b)]))
        ctx.set_trace_bucket(20000)
        st = ctx.collide(q, flags=capi.CG_TRACE)
        t = ctx.trace().sum(0, dtype=np.uint64)
        assert 2 * t[0] + n == st["node_pairs"] and t[0] > 100 and t[1] == st["warp_steps"]
        assert t[0] <= 32 * t[1] and t[2] == st["tri_tests"] and t[2] <= 32 * t[3]
