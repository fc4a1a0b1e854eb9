"""The narrow phase's quick plane tests (planes_miss in csrc/cg_device.cuh),
compiled for the host: a triangle pair that they reject must be a miss of the
whole test in every mode, with no plane distance that the recheck recomputes.
Pairs: near contact at several scales, sharing corners, almost coplanar,
corners within the 1e-6 band, slivers, points, far from the origin, the golden
near-epsilon pairs, non-finite values."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from test_sat_filter import CSRC, SOURCE

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")

MISS_SOURCE = "#include <algorithm>\nusing std::max; using std::min;\n" + SOURCE[:SOURCE.index("static Box box(")] + r"""
template <int kMode>
static int one(const float3 v[6], bool& rejected) {
    float3 s, t;
    Recheck rc;
    const int r = tri_tri_mode<kMode>(v[0], v[1], v[2], v[3], v[4], v[5], s, t, rc);
    rejected = planes_miss<kMode>(v[0], v[1], v[2], tri_plane(v[0], v[1], v[2]), v[3], v[4], v[5],
                                  tri_plane(v[3], v[4], v[5]));
    return rejected && (r != TT_MISS || rc.checked) ? 1 : 0;
}
// per pair: bad (bit per mode), rejected (by mode 0), the reference's verdict is a hit
extern "C" void check(const float* p, int n, int* bad, int* rejected, int* hit) {
    for (int i = 0; i < n; ++i) {
        float3 v[6];
        for (int k = 0; k < 6; ++k) v[k] = make_float3(p[18 * i + 3 * k], p[18 * i + 3 * k + 1], p[18 * i + 3 * k + 2]);
        bool r0, r1, r2;
        bad[i] = one<0>(v, r0) | one<1>(v, r1) << 1 | one<2>(v, r2) << 2;
        rejected[i] = r0;
        float3 s, t;
        hit[i] = tri_tri(v[0], v[1], v[2], v[3], v[4], v[5], s, t) == TT_HIT;
    }
}
"""


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    d = tmp_path_factory.mktemp("planes")
    src, so = d / "planes.cpp", d / "planes.so"
    src.write_text(MISS_SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC, str(src), "-o", str(so)],
                   check=True)
    lib = C.CDLL(str(so))

    def run(pairs):
        pairs = np.ascontiguousarray(pairs, np.float32).reshape(-1, 18)
        out = [np.zeros(len(pairs), np.int32) for _ in range(3)]
        lib.check(C.c_void_p(pairs.ctypes.data), len(pairs), *[C.c_void_p(x.ctypes.data) for x in out])
        return out

    return run


@pytest.mark.parametrize("kind", ["near", "small", "large", "shared", "coplanar", "band", "sliver", "point", "far", "golden",
                                  "nonfinite"])
def test_rejected_pairs_are_misses(check, kind):
    rng = np.random.Generator(np.random.PCG64(41))
    n = 150000
    size = {"small": 1e-2, "large": 50.0}.get(kind, 0.3)
    p = rng.normal(size=(n, 6, 3)) * size
    p[:, :3] += rng.normal(size=(n, 1, 3)) * size * 0.7
    if kind == "shared":
        p[:, 3] = p[:, 0]
        p[: n // 2, 4] = p[: n // 2, 1]
    if kind in ("coplanar", "band"):  # the second's corners in the first's plane, and off it by about the band
        e1, e2 = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
        uv = rng.uniform(-1, 2, size=(n, 3, 2))
        p[:, 3:] = p[:, :1] + uv[..., :1] * e1[:, None] + uv[..., 1:] * e2[:, None]
        nrm = np.cross(e1, e2)
        off = 10.0 ** rng.uniform(-9, -4, size=(n, 3, 1)) * rng.choice([-1, 1], size=(n, 3, 1))
        if kind == "band":
            p[:, 3:] += off * nrm[:, None] / (nrm * nrm).sum(1)[:, None, None]
    if kind == "sliver":
        p[:, 2] = p[:, 0] + (p[:, 1] - p[:, 0]) * rng.uniform(size=(n, 1)) + rng.normal(size=(n, 3)) * 1e-6
    if kind == "point":
        p[:, 1:3] = p[:, :1]
        p[: n // 3, 4:] = p[: n // 3, 3:4]
    if kind == "far":
        p += rng.normal(size=(n, 1, 3)) * 1000.0
    if kind == "golden":
        p = np.concatenate([np.concatenate([np.load(os.path.join(GOLDEN, f))[k].reshape(-1, 9) for k in ("a", "b")], 1)
                            for f in ("tritri.npz", "tritri_near.npz")])
    if kind == "nonfinite":
        at = rng.random(p.shape) < 0.02
        p[at] = rng.choice([np.nan, np.inf, -np.inf, 1e30, 3e38, -3e38], size=int(at.sum()))
    with np.errstate(over="ignore"):
        bad, rejected, hit = check(p)
    assert not bad.any(), (kind, np.bincount(bad), np.nonzero(bad)[0][:5])
    if kind == "near":  # and they reject nearly every miss that the plane tests decide
        assert hit.mean() > 0.02 and rejected.mean() > 0.4
