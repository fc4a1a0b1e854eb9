"""Contacts, rays and mean origins of maps at the sizes where the order stage
changes its blocks (half a block below 128 triangles, a block of 1,024 threads
from 1,024 on), its sort and its vertex set, alone and many together, bit for
bit and in order against the oracle
(src/CollisionDetection/CreateUncollideRays.cpp:60-201)."""
import numpy as np
import pytest

from inmyroom_vulkan_gb300 import scenes
from test_gpu_contacts_edge import QUAD, run

pytestmark = pytest.mark.gpu


def spikes(n):
    """n small triangles of shared and own vertices that cross z = 0 inside the quad."""
    rng = np.random.default_rng(n)
    at = rng.uniform(-0.9, 0.9, (n, 2)).astype(np.float32)
    pts = np.zeros((n, 3, 3), np.float32)
    pts[:, :, :2] = at[:, None] + rng.uniform(-0.01, 0.01, (n, 3, 2))
    pts[:, :, 2] = rng.uniform(0.01, 0.03, (n, 3)) * np.float32([1, -1, 1])
    idx = np.arange(3 * n).reshape(n, 3)
    some = np.arange(1, n, 3)
    idx[some, 0] = idx[some - 1, 0]  # a third start at their predecessor's first vertex
    return scenes.Mesh(pts.reshape(-1, 3), None, idx.reshape(-1).astype(np.uint32))


SIZES = [1, 31, 32, 33, 64, 127, 128, 129, 255, 257, 511, 513, 1023, 1024, 1025, 2047, 2049, 3600]


@pytest.mark.parametrize("sizes", [[n] for n in SIZES] + [SIZES, [127] * 700 + [128, 40, 1024]],
                         ids=lambda s: f"{len(s)}x{s[0]}")
def test_map_sizes(port, sizes):
    contacts, mids = run(port, [(QUAD, spikes(n)) for n in sizes])
    for n, m in zip(sizes, mids):
        assert len(m.contacts(1)[0]) == n
    assert len(contacts) == sum(len(m.contacts(s)[0]) for m in mids for s in (0, 1))
