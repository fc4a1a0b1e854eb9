"""Trees of meshes at the sizes where the builder changes kernels (a thread, a
warp or a block per node; chains or segments for the covariances), alone, side
by side in one batch, and in a batch wide enough that its kernels follow one
another without overlap: bit for bit the oracle's
(src/Geometry/OBBtree.cpp:321-358)."""
import numpy as np
import pytest

from test_gpu_build import M, same

pytestmark = pytest.mark.gpu

EDGES = [4, 5, 16, 17, 33, 128, 129, 256, 257, 513, 682, 683, 1024, 1025, 2730, 2731, 5462]


def mesh(n, seed):
    rng = np.random.default_rng(seed)
    pts = rng.normal(size=(max(8, n // 2 + 2), 3)).astype(np.float32) * np.float32([3.0, 1.0, 0.3])
    return M(pts, rng.integers(0, len(pts), (n, 3)))


@pytest.mark.parametrize("sizes", [[n] for n in EDGES] + [EDGES, EDGES * 3], ids=lambda s: f"{len(s)}x{s[0]}")
def test_sizes(gpu_ctx, port, sizes):
    meshes = [mesh(n, 100 + n) for n in sizes]
    ids = gpu_ctx.build_trees(meshes)
    for m, tid in zip(meshes, ids):
        same(gpu_ctx.export_tree(int(tid)), port.tree_build(m.points, m.indices, None).export(), normals=False)
    for tid in ids:
        gpu_ctx.free_tree(int(tid))


@pytest.mark.parametrize("n", [152, 153, 609, 4864, 4865])
def test_level_widths(gpu_ctx, port, n):
    """Levels of n nodes, where the eigensystems' group of lanes changes."""
    kinds = [mesh(k, 31 + k) for k in (1, 5, 7, 12)]
    ids = gpu_ctx.build_trees([kinds[i % 4] for i in range(n)])
    for i in list(range(8)) + list(range(n - 8, n)):
        m = kinds[i % 4]
        same(gpu_ctx.export_tree(int(ids[i])), port.tree_build(m.points, m.indices, None).export(), normals=False)
    for tid in ids:
        gpu_ctx.free_tree(int(tid))


def test_wide_level(gpu_ctx, port):
    """20,000 small meshes beside large ones: every per-node grid is above a block an SM."""
    small = [mesh(n, 7 + n) for n in (1, 5, 6, 9, 17, 20)]
    large = [mesh(n, 100 + n) for n in (257, 1025, 2731)]
    meshes = [small[i % len(small)] for i in range(20000)]
    for k, m in enumerate(large):
        meshes[5000 * (k + 1)] = m
    ids = gpu_ctx.build_trees(meshes)
    for i in list(range(12)) + [5000, 10000, 15000] + list(range(19994, 20000)):
        m = meshes[i]
        same(gpu_ctx.export_tree(int(ids[i])), port.tree_build(m.points, m.indices, None).export(), normals=False)
    for tid in ids:
        gpu_ctx.free_tree(int(tid))
