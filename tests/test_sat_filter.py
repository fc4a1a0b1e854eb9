"""The traversal's box-test filter (csrc/cg_sat.cuh), compiled for the host and
compared with the reference's 15-axis expressions on the CPU: an axis that it
decides must be what overlap_on says of it, in both argument orders, and the
axes that it leaves open decide the rest; its surface must be within its stated error.
Boxes: random pairs at every gap, parallel and identical ones, flat, needle
and point boxes, sheared ones, far from the origin, tiny and huge scales, and
non-finite values."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "inmyroom_vulkan_gb300", "csrc")

SOURCE = r"""
#include <cmath>
#include <cstdint>
using std::fabs;
#define __device__
#define __forceinline__ inline
#define __noinline__
struct float3 { float x, y, z; };
struct float4 { float x, y, z, w; };
static inline float3 make_float3(float x, float y, float z) { return {x, y, z}; }
static inline float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }
#include "cg_sat.cuh"
using namespace cg;
static Box box(const float* p) {
    return Box{{p[0], p[1], p[2]}, {p[3], p[4], p[5]}, {p[6], p[7], p[8]}, {p[9], p[10], p[11]}};
}
// per pair: 0 fine, 1 a wrong separation, 2 a wrong overlap, 3 a wrong verdict, 4 the surface's error; open counts the
// undecided axes of the pairs without a certain separation
extern "C" void check(const float* a, const float* b, int n, int* bad, int* open) {
    for (int i = 0; i < n; ++i) {
        const Box A = box(a + 12 * i), B = box(b + 12 * i);
        bad[i] = open[i] = 0;
        for (int order = 0; order < 2; ++order) {
            const Box& X = order ? B : A;
            const Box& Y = order ? A : B;
            const SatBox sx = sat_box(X), sy = sat_box(Y);
            unsigned m = 0;
            const bool sep = sat_filter(sx, sy, m), want = sat(A, B);
            if (sep && want) bad[i] = 1;
            if (!sep) {
                bool ok = true;
                for (unsigned k = 0; k < 15; ++k) {
                    if (!(m >> k & 1u) && !sat_axis(X, Y, k)) bad[i] = 2;
                    if ((m >> k & 1u) && !sat_axis(X, Y, k)) ok = false;
                    open[i] += m >> k & 1u;
                }
                if (ok != want) bad[i] = 3;
            }
            float err;
            const float s = sat_surface(sx, err), exact = surface(X);
            if (fabsf(s - exact) > err) bad[i] = 4;
        }
    }
}
"""


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    d = tmp_path_factory.mktemp("sat")
    src, so = d / "sat.cpp", d / "sat.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC, str(src), "-o", str(so)],
                   check=True)
    lib = C.CDLL(str(so))

    def run(a, b):
        a, b = (np.ascontiguousarray(x, np.float32) for x in (a, b))
        bad, opened = np.zeros(len(a), np.int32), np.zeros(len(a), np.int32)
        p = lambda x: C.c_void_p(x.ctypes.data)  # noqa: E731
        lib.check(p(a), p(b), len(a), p(bad), p(opened))
        return bad, opened

    return run


def rotations(n, rng):
    q = rng.normal(size=(n, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w), 2 * (x * y + z * w),
                     1 - 2 * (x * x + z * z), 2 * (y * z - x * w), 2 * (x * z - y * w), 2 * (y * z + x * w),
                     1 - 2 * (x * x + y * y)], 1).reshape(n, 3, 3)


def boxes(n, rng, half, centre, rot=None):
    r = rotations(n, rng) if rot is None else rot
    return np.concatenate([centre, (r * half[:, :, None]).reshape(n, 9)], 1)


@pytest.mark.parametrize("kind", ["random", "parallel", "flat", "needle", "sheared", "far", "tiny", "huge", "same",
                                  "point", "underflow", "nonfinite"])
def test_filter_agrees_with_the_reference_expressions(check, kind):
    rng = np.random.Generator(np.random.PCG64(17))
    n = 60000
    ha, hb = (10.0 ** rng.uniform(-2, 0, size=(n, 3)) for _ in range(2))
    d = rng.normal(size=(n, 3))
    gap = (ha.max(1) + hb.max(1)) * rng.uniform(0, 1.6, size=n)
    ca = rng.normal(size=(n, 3))
    cb = ca + d / np.linalg.norm(d, axis=1, keepdims=True) * gap[:, None]
    ra = rotations(n, rng)
    rb = rotations(n, rng)
    if kind == "parallel":  # common axes, and turned by a rounding error
        rb = ra + rng.normal(size=ra.shape) * 10.0 ** rng.uniform(-9, -5, size=(n, 1, 1)) * (rng.random((n, 1, 1)) < 0.5)
    if kind == "flat":
        ha[:, 2] = 2.0 ** -23
        hb[:, 1] *= 1e-6
    if kind == "needle":
        ha[:, 1:] = 2.0 ** -23
        hb[:, :2] *= 1e-6
    a, b = boxes(n, rng, ha, ca, ra), boxes(n, rng, hb, cb, rb)
    if kind == "sheared":
        a[:, 3:] += rng.normal(size=(n, 9)) * 0.3
        b[:, 3:] *= rng.uniform(0.1, 3, size=(n, 9))
    if kind == "far":
        a[:, :3] += 4096.0
        b[:, :3] += 4096.0
    if kind == "tiny":
        a, b = a * 1e-8, b * 1e-8
    if kind == "huge":
        a, b = a * 1e9, b * 1e9
    if kind == "same":
        b = a.copy()
        b[n // 2:, 3:] = -b[n // 2:, 3:]
    if kind == "point":
        a[:, 3:] = 0.0
        b[: n // 2, 3:] = 0.0
        b[: n // 4, :3] = a[: n // 4, :3]
    if kind == "underflow":
        s = 10.0 ** rng.uniform(-40, -10, size=(n, 1))
        a, b = a * s, b * s
    if kind == "nonfinite":
        for x in (a, b):
            at = rng.random(x.shape) < 0.05
            x[at] = rng.choice([np.nan, np.inf, -np.inf, 3e38, -3e38], size=int(at.sum()))
    with np.errstate(over="ignore"):
        bad, opened = check(a, b)
    assert not bad.any(), (kind, np.bincount(bad), np.nonzero(bad)[0][:5])
    if kind == "random":  # and it decides nearly all of them
        assert (opened > 0).mean() < 5e-3
