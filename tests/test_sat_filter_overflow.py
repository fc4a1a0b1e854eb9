"""The traversal's box-test filter (csrc/cg_sat.cuh) on boxes so large or so far
out that projections overflow FP32, compiled for the host: where the
reference's expressions meet infinities the filter may decide no axis."""
import numpy as np
import pytest
from test_sat_filter import boxes, check  # noqa: F401

# log10 of the edges, log10 of the centres' distance from the origin
RANGES = {"below": ((10, 11.5), (9, 12)), "edges 1e12": ((11.5, 12.5), (10, 13)), "edges 1e13": ((12.5, 13.5), (10, 13)),
          "edges 1e14": ((13.5, 14.5), (10, 15)), "far 1e15": ((11.5, 12.2), (14.5, 15.5)),
          "far 1e30": ((3, 6), (29, 31)), "all": ((5, 20), (5, 25))}


@pytest.mark.parametrize("kind", RANGES)
@pytest.mark.parametrize("near", [True, False])
def test_no_axis_is_decided_by_an_overflow(check, kind, near):  # noqa: F811
    rng = np.random.Generator(np.random.PCG64(23))
    n = 60000
    (e0, e1), (c0, c1) = RANGES[kind]
    edge = 10.0 ** rng.uniform(e0, e1, size=(n, 1))
    ha, hb = (edge * 10.0 ** rng.uniform(-1, 0, size=(n, 3)) for _ in range(2))
    unit = lambda: (lambda d: d / np.linalg.norm(d, axis=1, keepdims=True))(rng.normal(size=(n, 3)))  # noqa: E731
    ca = unit() * 10.0 ** rng.uniform(c0, c1, size=(n, 1))
    # beside it, at a gap of the boxes' size, or anywhere at that distance
    gap = edge * rng.uniform(0, 2.5, size=(n, 1)) if near else 10.0 ** rng.uniform(c0, c1, size=(n, 1))
    with np.errstate(over="ignore"):
        bad, _ = check(boxes(n, rng, ha, ca), boxes(n, rng, hb, ca + unit() * gap))
    assert not bad.any(), (kind, np.bincount(bad), np.nonzero(bad)[0][:5])
