"""The surface that the box-test filter gives (csrc/cg_sat.cuh), compiled for the
host: within its stated error of the reference's at the scales where squares of
the face normals underflow or overflow, or in error without limit. The descent
computes the reference's own wherever that error leaves the larger box open."""
import numpy as np
import pytest
from test_sat_filter import boxes, check  # noqa: F401

# log10 of the edges: a decade at a time where the squares are subnormal, zero
# or near the largest float
SCALES = [(-16, -13), (-13, -12), (-12, -11), (-11.5, -10.5), (-10.5, -10), (-10, -9.5), (-9.5, -9), (-9, -8), (-8, -6),
          (3, 6), (6, 9), (9, 9.5), (9.5, 10.5), (10.5, 12)]


@pytest.mark.parametrize("scale", SCALES, ids=lambda s: f"{s[0]}..{s[1]}")
@pytest.mark.parametrize("flat", [False, True])
def test_surface_is_within_its_error(check, scale, flat):  # noqa: F811
    rng = np.random.Generator(np.random.PCG64(29))
    n = 60000
    half = 10.0 ** rng.uniform(*scale, size=(n, 3))
    if flat:
        half[:, 2] *= 10.0 ** rng.uniform(-4, 0, size=n)
    a = boxes(n, rng, half, rng.normal(size=(n, 3)) * half.max(1)[:, None])
    with np.errstate(over="ignore"):
        bad, _ = check(a, a)
    assert not bad.any(), (scale, np.bincount(bad), np.nonzero(bad)[0][:5])


def test_surface_at_the_edge_of_the_largest_float(check):  # noqa: F811
    # cubes whose normals' squares are within some roundings of the largest
    # float: the reference's sum of them can be finite where the filter's, in
    # another order, is not, and the other way round
    rng = np.random.Generator(np.random.PCG64(31))
    n = 400000
    edge = np.sqrt(np.sqrt(float(np.finfo(np.float32).max))) * (1.0 + rng.uniform(-3e-7, 3e-7, size=(n, 1)))
    a = boxes(n, rng, np.repeat(edge, 3, 1), np.zeros((n, 3)))
    with np.errstate(over="ignore"):
        bad, _ = check(a, a)
    assert not bad.any(), (np.bincount(bad), np.nonzero(bad)[0][:5])
